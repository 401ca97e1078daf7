"""The work whose speed is tracked: training steps, forward passes and the blocks a rank of a larger job runs.

Every case goes through the calls a user makes: ``train.Trainer.train_step`` on a pinned host batch, the model's forward,
the parallel blocks of ``parallel/`` and the attention primitives of ``ops.functional``.  Sizes are those of the presets in
``config.py``, of ``bench.py``, ``benchmarks/`` and the tests.  Models keep the width of their preset; the number of layers
is two, so that weights, optimizer state and activations of several runs fit one GPU (a rank of an 8-GPU job holds an
eighth of them).

Kinds:

* ``step``: one optimizer step; returns the loss, the gradients, the updated weights and the optimizer state.
* ``logits``: forward without labels under ``no_grad``: evaluation of a prompt; returns the logits.
* ``mlp``: forward and backward of the Odysseus MLP block, weight gradients written where the optimizer reads them.
* ``attention``: forward and backward of the packed causal attention core of one rank: few heads, the whole sequence.
* ``ring_block``: forward and backward of one off-diagonal block of zigzag ring attention: no mask, ``Tq != Tk``.
"""
import math

import torch

from odysseus_transformer_b200.config import get_model_config
from odysseus_transformer_b200.mesh import ParallelContext, set_context
from odysseus_transformer_b200.ops import functional as F
from odysseus_transformer_b200.ops import native
from odysseus_transformer_b200.optim.adamw import ShardedAdamW
from odysseus_transformer_b200.parallel.apply import build_model, prepare_attn_inputs
from odysseus_transformer_b200.parallel.attention import packed_rope_attention
from odysseus_transformer_b200.parallel.linear import Zero3Schedule
from odysseus_transformer_b200.parallel.odysseus import OdysseusMLP
from odysseus_transformer_b200.train import Trainer
from odysseus_transformer_b200.utils.buffers import set_global_memory_buffer


def _step(name, model, layers, tokens, mode="odysseus", checkpoint=False):
    return {"name": name, "kind": "step", "model": model, "layers": layers, "tokens": tokens, "mode": mode,
            "checkpoint": checkpoint}


def listed():
    return [
        # the smallest run of the GPU tests and of the smoke check, at a short sequence: host time and launches count
        _step("step_small_512", "small", 2, 512),
        # grouped-query variant at a length that is no multiple of any tile
        _step("step_small_gqa_1531", "small-gqa", 2, 1531, mode="ulysses"),
        # Llama-2-7B width on a short sequence: optimizer and small GEMMs weigh as much as the tokens
        _step("step_7b_2k", "llama2-7b", 2, 2048, mode="tpsp"),
        # the weak-scaling benchmark's shape per GPU: 8K tokens of Llama-2-7B
        _step("step_7b_8k", "llama2-7b", 2, 8192),
        # Llama-3-8B width (vocabulary 128256): logits past 2 GiB, so lm_head and loss run in chunks
        _step("step_8b_12k", "llama3-8b", 2, 12288, mode="ring"),
        # long sequence with activation checkpointing: the sweep's 32K point, attention as heavy as the GEMMs
        _step("step_3b_gqa_32k_ckpt", "llama2-3b-gqa", 2, 32768, checkpoint=True),
        # evaluation of a short prompt: the smallest call, nothing but launches
        {"name": "logits_small_128", "kind": "logits", "model": "small", "layers": 2, "tokens": 128},
        # evaluation of a long document, ragged length
        {"name": "logits_7b_4001", "kind": "logits", "model": "llama2-7b", "layers": 2, "tokens": 4001},
        # the MLP block benchmark at 8K tokens per rank
        {"name": "mlp_7b_8k", "kind": "mlp", "model": "llama2-7b", "tokens": 8192},
        # what one of 8 ranks computes of Llama-2-7B attention at 32K tokens: 4 heads, whole sequence
        {"name": "attention_32k_4h", "kind": "attention", "tokens": 32768, "heads": 4, "kv_heads": 4},
        # one of 8 ranks of a grouped-query model: 4 query heads on 1 kv head, ragged length
        {"name": "attention_10007_gqa", "kind": "attention", "tokens": 10007, "heads": 4, "kv_heads": 1},
        # one step of a 4-rank zigzag ring at 32K tokens: the late half of a rank's rows against another rank's whole block
        {"name": "ring_block_8k", "kind": "ring_block", "tokens": 4096, "keys": 8192, "heads": 32, "kv_heads": 8},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _round(rng, n):
    """Half of the lengths are multiples of 128, the others whatever was drawn."""
    return max(128, n // 128 * 128) if rng.random() < 0.5 else n


def draw(rng):
    kind = rng.choice(["step", "step", "step", "logits", "mlp", "attention", "attention", "ring_block"])
    if kind in ("step", "logits"):
        model = rng.choice(["small", "small-gqa", "llama2-7b", "llama2-3b-gqa", "llama3-8b", "mistral-7b"])
        small = model.startswith("small")
        layers = rng.randint(1, 4 if small else 2)
        c = {"kind": kind, "model": model, "layers": layers, "tokens": _round(rng, _log(rng, 128, 4096 if small else 16384))}
        if kind == "step":
            c["mode"] = rng.choice(["odysseus", "tpsp", "ulysses", "ring", "dp"])
            c["checkpoint"] = rng.random() < 0.25
        return c
    if kind == "mlp":
        return {"kind": kind, "model": rng.choice(["small", "llama2-7b", "llama3-8b"]), "tokens": _round(rng, _log(rng, 256, 16384))}
    kv = rng.choice([1, 2, 4, 8])
    heads = kv * rng.choice([1, 4])
    if kind == "attention":
        return {"kind": kind, "tokens": _round(rng, _log(rng, 256, 32768 if heads <= 8 else 12288)), "heads": heads, "kv_heads": kv}
    return {"kind": kind, "tokens": _round(rng, _log(rng, 256, 8192)), "keys": _round(rng, _log(rng, 256, 8192)),
            "heads": heads, "kv_heads": kv}


def _context():
    native.set_backend("fused")
    dev = torch.device("cuda", torch.cuda.current_device())
    ctx = ParallelContext(device=dev, backend="fused")
    set_context(ctx)
    return ctx


def _config(case):
    cfg = get_model_config(case["model"])
    return cfg.replace(num_hidden_layers=case["layers"]) if "layers" in case else cfg


def prepare(case, seed):
    ctx = _context()
    dev = ctx.device
    kind, T = case["kind"], case["tokens"]
    g = torch.Generator(device=dev).manual_seed(seed)
    hg = torch.Generator().manual_seed(seed)

    def normal(*shape, scale):
        return (torch.randn(*shape, generator=g, device=dev) * scale).to(torch.bfloat16)

    if kind == "step":
        cfg = _config(case)
        trainer = Trainer(cfg, case["mode"], ctx, T, lr=1e-5, dtype=torch.bfloat16, seed=seed,
                          grad_checkpoint=case["checkpoint"])
        batch = torch.randint(cfg.vocab_size, (1, T + 1), generator=hg).pin_memory()
        return {"kind": kind, "trainer": trainer, "batch": batch}
    if kind == "logits":
        cfg = _config(case)
        model = build_model(cfg, "odysseus", ctx, dtype=torch.bfloat16, device=dev, seed=seed)
        ids = torch.randint(cfg.vocab_size, (1, T), generator=hg)
        s = prepare_attn_inputs("odysseus", ids, torch.arange(T).unsqueeze(0), None, 0, 1, dev)
        return {"kind": kind, "model": model, "ids": s["local_input_ids"], "pos": s["local_position_ids"]}
    if kind == "mlp":
        cfg = get_model_config(case["model"])
        set_global_memory_buffer(dev)
        mlp = OdysseusMLP(cfg, ctx, Zero3Schedule(), dtype=torch.bfloat16, device=dev)
        with torch.no_grad():
            for p in mlp.parameters():
                p.copy_(normal(*p.shape, scale=cfg.initializer_range))
        opt = ShardedAdamW(mlp.parameters(), lr=1e-5)
        x = normal(T, cfg.hidden_size, scale=1.0).requires_grad_(True)
        return {"kind": kind, "mlp": mlp, "opt": opt, "x": x, "dy": normal(T, cfg.hidden_size, scale=0.1)}
    hq, hkv = case["heads"], case["kv_heads"]
    if kind == "attention":
        cos, sin = F.rope_tables(torch.arange(T, device=dev), 128, 10000.0)
        qkv = normal(T, (hq + 2 * hkv) * 128, scale=0.5).requires_grad_(True)
        return {"kind": kind, "qkv": qkv, "do": normal(T, hq * 128, scale=0.1), "cos": cos, "sin": sin, "hq": hq, "hkv": hkv}
    k, v = normal(case["keys"], hkv, 128, scale=0.5), normal(case["keys"], hkv, 128, scale=0.5)
    return {"kind": kind, "q": normal(T, hq, 128, scale=0.5), "k": k, "v": v, "do": normal(T, hq, 128, scale=0.1)}


def run(state):
    kind = state["kind"]
    if kind == "step":
        tr = state["trainer"]
        loss = tr.train_step(state["batch"])
        o = tr.optimizer
        return {"loss": loss, "grad": o.flat_grad, "param": o.flat_param, "master": o.master, "exp_avg": o.exp_avg,
                "exp_avg_sq": o.exp_avg_sq}
    if kind == "logits":
        with torch.no_grad():
            return state["model"](state["ids"], state["pos"])
    if kind == "mlp":
        x, mlp = state["x"], state["mlp"]
        x.grad = None
        y = mlp(x)
        y.backward(state["dy"])
        state["opt"].zero_grad()
        return {"y": y.detach(), "dx": x.grad, "dw": [p.main_grad for p in mlp.parameters()]}
    if kind == "attention":
        qkv = state["qkv"]
        qkv.grad = None
        # the projection's epilogue rotates q and k, as in the model blocks
        o = packed_rope_attention(qkv, state["cos"], state["sin"], state["hq"], state["hkv"], pre_rotated=True)
        o.backward(state["do"])
        return {"o": o.detach(), "dqkv": qkv.grad}
    q, k, v = state["q"], state["k"], state["v"]
    o, lse = F.attn_block_fwd(q, k, v, False)
    dq, dk, dv = F.attn_block_bwd(state["do"], q, k, v, o, lse, False)
    return {"o": o, "lse": lse, "dq": dq, "dk": dk, "dv": dv}


def _f64(t):
    return t.detach().to(torch.float64)


def _rotate(x, cos, sin, sign=1.0):
    """Rotary embedding (half split) of x [T, heads, 128] by sign times the angles."""
    c, s = cos.unsqueeze(1), sign * sin.unsqueeze(1)
    a, b = x[..., :64], x[..., 64:]
    return torch.cat([a * c - b * s, b * c + a * s], dim=-1)


def _attention(q, k, v, causal, do=None):
    """Softmax attention of q [Tq, H, 128] on k, v [Tk, Hkv, 128], a head and some rows at a time; with ``do`` also the
    gradients of q, k and v."""
    Tq, H, hd = q.shape
    G, rows = H // k.shape[1], max(128, (1 << 27) // k.shape[0])
    o, lse = torch.empty_like(q), torch.empty(H, Tq, dtype=q.dtype, device=q.device)
    dq, dk, dv = (torch.zeros_like(t) for t in (q, k, v))
    for h in range(H):
        kh, vh = k[:, h // G], v[:, h // G]
        for r in range(0, Tq, rows):
            sl = slice(r, min(Tq, r + rows))
            n = sl.stop if causal else k.shape[0]
            s = (q[sl, h] @ kh[:n].t()) / math.sqrt(hd)
            if causal:
                s[:, r:] += torch.full((n - r, n - r), float("-inf"), dtype=s.dtype, device=s.device).triu_(1)
            lse[h, sl] = torch.logsumexp(s, 1)
            p = s.sub_(lse[h, sl].unsqueeze(1)).exp_()
            o[sl, h] = p @ vh[:n]
            if do is not None:
                dv[:n, h // G] += p.t() @ do[sl, h]
                delta = (do[sl, h] * o[sl, h]).sum(1, keepdim=True)
                ds = (do[sl, h] @ vh[:n].t()).sub_(delta).mul_(p).mul_(1.0 / math.sqrt(hd))
                dq[sl, h] = ds @ kh[:n]
                dk[:n, h // G] += ds.t() @ q[sl, h]
    return o, lse, dq, dk, dv


def _rms(x, w, eps):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w


def exact(case, seed):
    """What ``run`` returns for these inputs, in 64 bits.  A step has no such value here: after the optimizer's first
    update of +-lr the sign of a gradient that is nearly zero decides, and its products are those of the other kinds."""
    kind = case["kind"]
    if kind == "step":
        return None
    state = prepare(case, seed)
    if kind == "logits":
        cfg, m = _config(case), state["model"]
        if case["tokens"] > 8192:
            return None
        w = {k: _f64(t) for k, t in m.export_hf_state_dict().items()}
        T, hd = case["tokens"], 128
        ang = torch.arange(T, dtype=torch.float64, device=state["ids"].device).unsqueeze(1) / cfg.rope_theta ** (
            torch.arange(0, hd, 2, dtype=torch.float64, device=state["ids"].device) / hd)
        cos, sin = ang.cos(), ang.sin()
        x = w["model.embed_tokens.weight"][state["ids"].reshape(-1)]
        for i in range(cfg.num_hidden_layers):
            p = "model.layers.%d." % i
            h = _rms(x, w[p + "input_layernorm.weight"], cfg.rms_norm_eps)
            q, k, v = ((h @ w[p + "self_attn.%s_proj.weight" % n].t()).view(T, -1, hd) for n in "qkv")
            o = _attention(_rotate(q, cos, sin), _rotate(k, cos, sin), v, True)[0]
            x = x + o.reshape(T, -1) @ w[p + "self_attn.o_proj.weight"].t()
            h = _rms(x, w[p + "post_attention_layernorm.weight"], cfg.rms_norm_eps)
            g, u = (h @ w[p + "mlp.%s_proj.weight" % n].t() for n in ("gate", "up"))
            x = x + (g * torch.sigmoid(g) * u) @ w[p + "mlp.down_proj.weight"].t()
        return (_rms(x, w["model.norm.weight"], cfg.rms_norm_eps) @ w["lm_head.weight"].t()).unsqueeze(0)
    if kind == "mlp":
        x, dy = _f64(state["x"]), _f64(state["dy"])
        w1, w2 = (_f64(p) for p in state["mlp"].parameters())
        g, u = (x @ w1.t()).chunk(2, dim=1)
        sig = torch.sigmoid(g)
        h, dh = g * sig * u, dy @ w2
        dgu = torch.cat([dh * u * sig * (1 + g * (1 - sig)), dh * g * sig], dim=1)
        return {"y": h @ w2.t(), "dx": dgu @ w1, "dw": [dgu.t() @ x, dy.t() @ h]}
    if kind == "attention":
        hq, hkv = state["hq"], state["hkv"]
        T = case["tokens"]
        q, k, v = _f64(state["qkv"]).view(T, -1, 128).split([hq, hkv, hkv], dim=1)
        o, _, dq, dk, dv = _attention(q, k, v, True, _f64(state["do"]).view(T, hq, 128))
        cos, sin = _f64(state["cos"]), _f64(state["sin"])
        # the gradient goes back through the rotation that the projection's epilogue applied
        d = torch.cat([_rotate(dq, cos, sin, -1.0), _rotate(dk, cos, sin, -1.0), dv], dim=1)
        return {"o": o.reshape(T, -1), "dqkv": d.reshape(T, -1)}
    o, lse, dq, dk, dv = _attention(*(_f64(state[n]) for n in ("q", "k", "v")), False, _f64(state["do"]))
    return {"o": o, "lse": lse, "dq": dq, "dk": dk, "dv": dv}


def work(case):
    """Products at two operations per multiply-add, causal halves not counted; a step's bytes are the optimizer's (fp32
    master and moments read and written, gradient and weight in bf16) and the activations' are left out: a step could keep
    them on the chip.  Checkpointing asks for the layers' forward a second time."""
    kind, T = case["kind"], case["tokens"]
    if kind in ("step", "logits"):
        cfg = _config(case)
        d, i, v, n = cfg.hidden_size, cfg.intermediate_size, cfg.vocab_size, cfg.num_hidden_layers
        layer = d * cfg.q_size + 2 * d * cfg.kv_size + cfg.q_size * d + 3 * d * i
        attn = 2.0 * T * T * cfg.q_size                                   # Q K^T and P V, lower triangle
        fwd = n * (2.0 * T * layer + attn)
        head = 2.0 * T * d * v
        params = cfg.num_parameters()
        if kind == "logits":
            return {"bytes": 2.0 * params - 2.0 * v * d + 2.0 * min(T, v) * d + 2.0 * T * v, "flops": fwd + head}
        flops = 3.0 * (n * 2.0 * T * layer + head) + n * 3.5 * attn + (fwd if case["checkpoint"] else 0.0)
        return {"bytes": 30.0 * params, "flops": flops}
    if kind == "mlp":
        cfg = get_model_config(case["model"])
        w = 3.0 * cfg.hidden_size * cfg.intermediate_size
        return {"bytes": 2.0 * (2 * w + 4.0 * T * cfg.hidden_size), "flops": 6.0 * T * w}
    hq, hkv = case["heads"], case["kv_heads"]
    if kind == "attention":
        return {"bytes": 2.0 * T * 128 * (2 * (hq + 2 * hkv) + 2 * hq), "flops": 3.5 * 2.0 * T * T * hq * 128}
    Tk = case["keys"]
    return {"bytes": 2.0 * 128 * (4.0 * T * hq + 4.0 * Tk * hkv) + 4.0 * T * hq, "flops": 3.5 * 4.0 * T * Tk * hq * 128}


def tolerance(case):
    """bf16 operands with fp32 accumulation, every tensor between two kernels rounded to bf16.  Measured as own kernels
    against the library path (torch matmul, FlashAttention-2) on the same inputs:

    attention, ring block: rel 0.0009 - 0.0031, largest single difference 0.22 of the rms (key gradients of shared heads);
    MLP block: rel 0.0001 (the roundings in between are the same; one that rounds elsewhere differs by half a bf16 step,
    0.002); logits of two layers: rel 0.009 (width 1024) to 0.02 (width 4096); gradients of a step: rel 0.010 (width 1024) to
    0.020 (width 4096), squared ones 0.024, single differences up to 0.83 of the rms."""
    kind = case["kind"]
    if kind in ("step", "logits"):
        return {"rel": 0.03, "max": 0.99}
    if kind == "mlp":
        return {"rel": 0.008, "max": 0.3}
    return {"rel": 0.012, "max": 0.9}
