"""Calls at the edges of what the kernels' dispatch rules take, against plain PyTorch (needs a B200)."""
import math

import pytest
import torch

from test_grad_delivery_cpu import check_recorded_backward

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    from odysseus_transformer_b200.ops import native
    native.set_backend("fused")
    return native.lib()


def _rand(*shape, scale=1.0, dtype=torch.bfloat16):
    return (torch.randn(*shape, device="cuda", dtype=torch.float32) * scale).to(dtype)


def _check_status(lib):
    torch.cuda.synchronize()
    assert lib.status(0) == 0, f"kernel status {lib.status(0)}"


def test_recorded_and_batched_backward_of_the_chunked_loss(lib):
    check_recorded_backward("cuda", torch.bfloat16)


# (300, 8000, 2): keys split over several CTAs; (512, 1024, 64): a full grid, not split
@pytest.mark.parametrize("Tq,Tk,H,lo,hi", [(300, 8000, 2, 0, 128), (300, 8000, 2, 0, 3000), (300, 8000, 2, 3000, 5000),
                                           (300, 8000, 2, 6000, 8000), (512, 1024, 64, 0, 128), (512, 1024, 64, 128, 1024)])
def test_attention_forward_with_keys_out_of_reach(lib, Tq, Tk, H, lo, hi):
    """Keys whose scores are -inf for every row weigh nothing, in whichever block or part they lie.  Bounds as for the other
    forward tests: bf16 output, fp32 statistics."""
    from odysseus_transformer_b200.ops import torch_ref as R
    torch.manual_seed(Tq + lo)
    q, k, v = _rand(Tq, H, 128, scale=0.3).abs() + 0.01, _rand(Tk, H, 128, scale=0.3), _rand(Tk, H, 128)
    k[lo:hi] = float("-inf")
    o, lse = lib.attn_fwd(q, k, v, False, 1.0 / math.sqrt(128))
    _check_status(lib)
    orf, lser = R.attn_fwd(q, k, v, False, 1.0 / math.sqrt(128))
    torch.testing.assert_close(lse, lser, rtol=1e-3, atol=2e-3)
    torch.testing.assert_close(o.float(), orf.float(), rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("lo,hi", [(4096, 4104), (8000, 8192), (0, 64), (4096, 32000)])
def test_cross_entropy_with_words_out_of_reach(lib, lo, hi):
    """Logits of -inf: the loss and its gradient of the other words, as plain fp32 PyTorch gives them."""
    torch.manual_seed(lo)
    logits = _rand(5, 32000, scale=3.0)
    logits[:, lo:hi] = float("-inf")
    tg = torch.randint(100, 4000, (5,), device="cuda")
    x = logits.float().requires_grad_(True)
    want = torch.nn.functional.cross_entropy(x, tg, reduction="none")
    (0.37 * want.sum()).backward()
    scale = torch.full((1,), 0.37, device="cuda")
    loss, _ = lib.ce_fwd(logits, tg, -100)
    got = logits.clone()
    loss1 = lib.ce_grad_(got, tg, scale, -100)
    torch.cuda.synchronize()
    torch.testing.assert_close(loss, want.detach(), rtol=1e-5, atol=1e-5)
    torch.testing.assert_close(loss1, want.detach(), rtol=1e-5, atol=1e-5)
    torch.testing.assert_close(got.float(), x.grad, rtol=1e-2, atol=1e-6)


def test_launches_are_counted(lib):
    """Every kernel a call launches counts, those that sum the parts of a split among them."""
    def count(fn):
        lib.reset_launch_count()
        fn()
        return lib.launch_count()
    g = lambda m, n, k: (lambda a, b: count(lambda: lib.gemm(a, b, None, 0, False)))(_rand(m, k), _rand(n, k))   # noqa: E731
    assert g(512, 1024, 32000) == 2                      # split, sum of the shares
    assert g(128, 256, 4096) == 1                        # shared by the CTAs of a cluster
    assert g(2048, 4096, 1024) == 1

    def attention(Tq, Tk, H, Hkv, causal):
        q, k, v = _rand(Tq, H, 128), _rand(Tk, Hkv, 128), _rand(Tk, Hkv, 128)
        sc = 1.0 / math.sqrt(128)
        o, lse = lib.attn_fwd(q, k, v, causal, sc)
        return (count(lambda: lib.attn_fwd(q, k, v, causal, sc)),
                count(lambda: lib.attn_bwd(q, q, k, v, o, lse, causal, sc, None, None, None)))
    assert attention(4096, 4096, 32, 32, True) == (1, 2)  # full grids: forward; statistics, gradients
    assert attention(2600, 2600, 4, 1, True) == (2, 4)    # both gradient grids split
    assert attention(300, 8000, 2, 2, False) == (2, 3)    # only the queries' gradient is
    try:
        lib.attn_bwd_set_variant(0)
        assert attention(1024, 1024, 4, 4, True)[1] == 3  # statistics, gradients, conversion of dQ
    finally:
        lib.attn_bwd_set_variant(1)
    _check_status(lib)


def test_calls_run_unsplit_when_scratch_cannot_be_had(lib):
    """Scratch only makes these calls faster: without memory for it they run as they would unsplit."""
    q, k, v, do = _rand(300, 2, 128), _rand(8000, 2, 128), _rand(8000, 2, 128), _rand(300, 2, 128)
    dq, dk, dv = torch.empty_like(q), torch.empty_like(k), torch.empty_like(v)
    a, b, c = _rand(512, 32000), _rand(1024, 32000), torch.empty(512, 1024, device="cuda", dtype=torch.bfloat16)
    sc = 1.0 / math.sqrt(128)

    def run():
        o, lse = lib.attn_fwd(q, k, v, False, sc)
        lib.reset_launch_count()
        lib.attn_bwd(do, q, k, v, o, lse, False, sc, dq, dk, dv)
        lib.gemm(a, b, c, 0, False)
        torch.cuda.synchronize()
        return [t.to("cpu", torch.float32) for t in (o, lse, dq, dk, dv, c)], lib.launch_count()
    want, n = run()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    fill = []
    try:
        # two allocator segments of 2 MiB for the calls' small outputs and statistics, but none of 20 MiB, and what is free in
        # those that there are taken up
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (4 << 20)) / total)
        with pytest.raises(torch.cuda.OutOfMemoryError):
            for _ in range(2048):
                fill.append(torch.empty(2 << 20, dtype=torch.uint8, device="cuda"))
        got, m = run()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
        del fill
    assert m < n                                           # it did run without its sums
    for x, y in zip(got, want):
        assert ((x - y).norm() / y.norm()).item() < 5e-3   # the same sums in another order, rounded to bf16
    _check_status(lib)


@pytest.mark.parametrize("bad", [50, -1, 1 << 40])
def test_embedding_gradient_reports_ids_outside_the_table(lib, bad):
    """index_add_ refuses such ids; the kernel skips them, says so, and the other tokens' rows are right."""
    from odysseus_transformer_b200.ops import native
    dy, ids = _rand(40, 64), torch.arange(40, device="cuda")
    ids[7] = bad
    dw = torch.empty(50, 64, device="cuda", dtype=torch.bfloat16)
    lib.embedding_grad_(dy, ids, dw)
    torch.cuda.synchronize()
    assert lib.status(0) == 107
    with pytest.raises(native.KernelStatusError, match="index"):
        native.check_status(0)
    want = torch.zeros_like(dw)
    want[:40] = dy
    want[7] = 0
    assert torch.equal(dw, want)
    _check_status(lib)


def test_evaluation_of_a_tensor_left_over_from_a_transform(lib):
    """A tensor that outlived a functorch transform goes to the kernels as ``apply`` hands it on: unwrapped."""
    from odysseus_transformer_b200.ops import functional as F
    kept, x, w = [], _rand(40, 64), _rand(64)

    def f(t):
        kept.append(t)
        return (t * t).sum()
    torch.func.grad(f)(x)
    with torch.no_grad():
        for fn in (lambda t: F.rmsnorm(t, w, 1e-5), lambda t: F.linear(t, x), F.swiglu):
            assert torch.equal(fn(kept[0]), fn(x))
    _check_status(lib)


def test_back_to_back_launches(lib):
    """Kernels come in while their predecessor drains: a chain in which each reads what the one before wrote gives the bits it
    gives with the GPU waited for after every call, over small and full grids."""
    def chain(T, wait):
        torch.manual_seed(T)
        x, w, wq, wo = _rand(T, 1024), _rand(1024) + 1, _rand(1536, 1024, scale=0.03), _rand(1024, 1024, scale=0.03)
        pos, tg = torch.arange(T, device="cuda"), torch.randint(1024, (T,), device="cuda")
        big = _rand(8192, 8192)
        torch.cuda.synchronize()
        kept = []
        for _ in range(0 if wait else 8):                # about 6 ms of work, so that the calls below queue up behind it
            lib.gemm(big, big, None, 0, False)

        def do(r):
            if wait:
                torch.cuda.synchronize()
            return r
        for _ in range(6):
            cos, sin = do(lib.rope_tables(pos, 128, 10000.0))
            h, rstd = do(lib.rmsnorm_fwd(x, w, 1e-5))
            qkv = do(lib.gemm(h, wq, None, 0, False, (cos, sin, 1280, 1536), None)).view(T, 12, 128)
            q, k, v = qkv[:, :8], qkv[:, 8:10], qkv[:, 10:]
            o, lse = do(lib.attn_fwd(q, k, v, True, 0.1))
            y = do(lib.gemm(o.view(T, 1024), wo, None, 0, False, None, x))
            act = do(lib.swiglu_fwd(torch.cat([y, y], 1)))
            dgu = do(lib.swiglu_bwd(act, torch.cat([y, y], 1)))
            dx, dw = do(lib.rmsnorm_bwd(dgu[:, :1024].contiguous(), x, w, rstd, y))
            d = do(lib.attn_bwd(dx.view(T, 8, 128), q, k, v, o, lse, True, 0.1, None, None, None))
            do(lib.rope_inplace_(d[0], 8, cos, sin, True))
            g = do(lib.gemm(d[0].view(T, 1024), y, None, 2, False))
            loss, l2 = do(lib.ce_fwd(y, tg, -100))
            z = y.clone()
            do(lib.ce_bwd_(z, tg, l2, torch.ones(1, device="cuda"), -100))
            kept += [h, qkv, o, lse, y, act, dgu, dx, dw, *d, g, loss, z]
            x = (y.float() / y.float().pow(2).mean().sqrt()).to(torch.bfloat16)
        return kept
    for T in (1, 300, 4096):
        got, want = chain(T, False), chain(T, True)
        _check_status(lib)
        assert all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("mode", ["odysseus", "tpsp", "ulysses", "ring", "dp"])
@pytest.mark.parametrize("tokens,checkpoint", [(1, False), (300, False), (300, True)])
def test_decoder_layer_as_one_node(lib, monkeypatch, mode, tokens, checkpoint):
    """Logits, gradients and updated weights of a step are those of the blocks' own calls: the loss and all that does not follow the
    embedding's gradient, which is summed in no fixed order, bit for bit.  With a hook on a block its layer keeps those calls."""
    from odysseus_transformer_b200.config import get_model_config
    from odysseus_transformer_b200.mesh import ParallelContext, set_context
    from odysseus_transformer_b200.models import llama
    from odysseus_transformer_b200.ops import functional as F
    from odysseus_transformer_b200.train import Trainer
    ctx = ParallelContext(device=torch.device("cuda", 0), backend="fused")
    set_context(ctx)
    cfg = get_model_config("small-gqa")
    batch = torch.randint(cfg.vocab_size, (1, tokens + 1), generator=torch.Generator().manual_seed(1)).pin_memory()
    made = []
    monkeypatch.setattr(F, "decoder_layer", lambda *a, f=F.decoder_layer: made.append(1) or f(*a))

    def run(limit, prepare=None):
        monkeypatch.setattr(llama, "_ONE_NODE_BYTES", limit)
        tr = Trainer(cfg, mode, ctx, tokens, lr=1e-3, seed=3, grad_checkpoint=checkpoint)
        if prepare is not None:
            prepare(tr.model)
        made.clear()
        loss = tr.train_step(batch).clone()
        n, o, emb = len(made), tr.optimizer, tr.model.embed_tokens.numel()
        got = [loss, o.flat_grad[emb:].clone(), o.master[emb:].clone()]
        with torch.no_grad():
            tr.model.embed_tokens.zero_().add_(0.01)
            got.append(tr.model(batch[:, :-1].cuda(), torch.arange(tokens, device="cuda").unsqueeze(0)))
        torch.cuda.synchronize()
        return n, got
    n0, want = run(0)
    n1, got = run(96 << 20)
    assert n0 == 0 and n1 == 2 * (2 if checkpoint else 1)
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    hooked = []
    n2, other = run(96 << 20, lambda m: m.layers[0].mlp.register_forward_hook(lambda *a: hooked.append(1)))
    assert n2 == n1 // 2 and hooked and torch.equal(other[0], want[0])
    _check_status(lib)


def test_decoder_layer_node_adds_and_returns_gradients(lib):
    """Without ``main_grad`` the gradients come back through autograd; with one that is written they are added to it."""
    from odysseus_transformer_b200.ops import functional as F
    torch.manual_seed(0)
    T, d, hq, hkv, inter = 200, 256, 4, 2, 384
    shapes = [(d,), ((hq + 2 * hkv) * 128, d), (d, hq * 128), (d,), (2 * inter, d), (d, inter)]
    ws = [torch.nn.Parameter(_rand(*s, scale=0.05) + (1 if len(s) == 1 else 0)) for s in shapes]
    x, dy = _rand(T, d).requires_grad_(True), _rand(T, d)
    cos, sin = lib.rope_tables(torch.arange(T, device="cuda"), 128, 10000.0)

    def step():
        for t in (x, *ws):
            t.grad = None
        F.decoder_layer(x, cos, sin, hq, hkv, 1e-5, 128 ** -0.5, ws).backward(dy)
        return x.grad
    dx = step()
    plain = [w.grad.clone() for w in ws]
    for w in ws:
        w.main_grad, w._grad_written = torch.full_like(w, float("nan")), False
    assert torch.equal(step(), dx) and all(w.grad is None and w._grad_written for w in ws)
    assert all(torch.equal(w.main_grad, g) for w, g in zip(ws, plain))
    assert torch.equal(step(), dx)
    _check_status(lib)
    for w, g in zip(ws, plain):                              # twice the gradient, each sum rounded once to bf16
        assert ((w.main_grad.float() - 2 * g.float()).norm() / (2 * g.float()).norm()).item() < 2.0 ** -8
    with pytest.raises(RuntimeError):
        F.decoder_layer(x, cos[:-1], sin[:-1], hq, hkv, 1e-5, 0.1, ws)
    with pytest.raises(RuntimeError):
        F.decoder_layer(x, cos, sin, hq, hkv, 1e-5, 0.1, [*ws[:5], ws[5][:, :-8]])


def test_decoder_layer_with_shared_norm_weight(lib):
    """One weight for both norms of a layer gets the sum of both gradients, in ``main_grad``: what two copies of it get, added."""
    from odysseus_transformer_b200.config import get_model_config
    from odysseus_transformer_b200.mesh import ParallelContext, set_context
    from odysseus_transformer_b200.train import Trainer
    ctx = ParallelContext(device=torch.device("cuda", 0), backend="fused")
    set_context(ctx)
    cfg = get_model_config("small")
    tr = Trainer(cfg, "odysseus", ctx, 300, lr=0.0, seed=3)
    batch = torch.randint(cfg.vocab_size, (1, 301), generator=torch.Generator().manual_seed(1)).pin_memory()
    layer = tr.model.layers[0]
    first, second = layer.input_layernorm, layer.post_attention_layernorm
    tr.train_step(batch)
    want = first.main_grad.float() + second.main_grad.float()
    layer.post_attention_layernorm = first
    tr.train_step(batch)
    _check_status(lib)
    # the contributions and their sum are each rounded to bf16 (2^-9 of them) on either side
    assert ((first.main_grad.float() - want).norm() / want.norm()).item() < 2.0 ** -7


def test_decoder_layer_node_takes_rows_that_lie_apart(lib):
    """Projections, and where their gradients go, as slices of wider matrices, as the single products take them: the bits of packed
    ones, written and added, and nothing beside the slices is touched."""
    from odysseus_transformer_b200.ops import functional as F
    torch.manual_seed(1)
    T, d, hq, hkv, inter = 200, 256, 4, 2, 384
    shapes = [(d,), ((hq + 2 * hkv) * 128, d), (d, hq * 128), (d,), (2 * inter, d), (d, inter)]
    packed = [torch.nn.Parameter(_rand(*s, scale=0.05) + (1 if len(s) == 1 else 0)) for s in shapes]
    wide = [_rand(s[0], s[1] + 40) if len(s) == 2 else None for s in shapes]
    apart = [torch.nn.Parameter(p.detach().clone() if w is None else w[:, 8:8 + p.shape[1]].copy_(p.detach())) for p, w in zip(packed, wide)]
    x, dy = _rand(T, d), _rand(T, d)
    cos, sin = lib.rope_tables(torch.arange(T, device="cuda"), 128, 10000.0)
    grads = [torch.full((*p.shape[:-1], p.shape[-1] + 24), 3.0, device="cuda", dtype=torch.bfloat16) for p in apart]
    for p, g in zip(apart, grads):
        p.main_grad = g[:, 16:16 + p.shape[1]] if p.dim() == 2 else g[:p.shape[0]]
        p._grad_written = False
    for p in packed:
        p.main_grad, p._grad_written = torch.empty_like(p), False
    for _ in range(2):                                       # written, then added to
        out = []
        for ws in (packed, apart):
            xs = x.clone().requires_grad_(True)
            y = F.decoder_layer(xs, cos, sin, hq, hkv, 1e-5, 128 ** -0.5, ws)
            y.backward(dy)
            out.append((y, xs.grad, *[w.main_grad.clone() for w in ws]))
        _check_status(lib)
        assert all(torch.equal(a, b) for a, b in zip(*out))
    assert all((g[:, :16] == 3.0).all() and (g[:, 16 + p.shape[1]:] == 3.0).all() for p, g in zip(apart, grads) if p.dim() == 2)
    with pytest.raises(RuntimeError):                        # columns that lie apart were never taken
        F.decoder_layer(x, cos, sin, hq, hkv, 1e-5, 0.1, [*packed[:5], torch.nn.Parameter(_rand(inter, d).t())])


@pytest.mark.parametrize("mode", ["ulysses", "ring", "dp"])
def test_evaluation_with_rope_tables_of_more_positions(lib, mode):
    """The sequence-parallel attention block takes the rows of its own tokens from longer tables; so does its layer."""
    from odysseus_transformer_b200.config import get_model_config
    from odysseus_transformer_b200.mesh import ParallelContext, set_context
    from odysseus_transformer_b200.parallel.apply import build_model
    ctx = ParallelContext(device=torch.device("cuda", 0), backend="fused")
    set_context(ctx)
    cfg = get_model_config("small")
    layer = build_model(cfg, mode, ctx, dtype=torch.bfloat16, device=ctx.device, seed=0).layers[0]
    cos, sin = lib.rope_tables(torch.arange(200, device="cuda"), cfg.head_dim, 10000.0)
    x = _rand(130, cfg.hidden_size)
    with torch.no_grad():
        y, _ = layer(x, None, cos, sin)
        want, _ = layer(x, None, cos[:130], sin[:130])
    _check_status(lib)
    assert torch.equal(y, want)


@pytest.mark.parametrize("kernel", ["one CTA", "pairs", "cluster", "split"])
def test_rotation_right_behind_its_tables(lib, kernel):
    """The rope tables' kernel is the direct predecessor of the product that rotates with them: the product's blocks are resident
    before the tables are written.  The same bits as with the GPU waited for in between."""
    M, N, K = {"one CTA": (300, 768, 512), "pairs": (600, 768, 512), "cluster": (300, 768, 512), "split": (1, 384, 32000)}[kernel]
    torch.manual_seed(M + N)
    a, b, big = _rand(M, K, scale=0.1), _rand(N, K, scale=0.1), _rand(8192, 8192)
    pos = [torch.randint(0, 9999, (M,), device="cuda") for _ in range(8)]

    def product(p, wait):
        cos, sin = lib.rope_tables(p, 128, 10000.0)
        if wait:
            torch.cuda.synchronize()
        rope = (cos, sin, 256, 384)
        return lib.gemm_cluster(a, b, None, 0, False, rope, None, 128, 2) if kernel == "cluster" else lib.gemm(a, b, None, 0, False, rope, None)
    try:
        lib.gemm_set_variant({"one CTA": 1, "pairs": 2}.get(kernel, 0))
        lib.reset_launch_count()
        want = [product(p, True) for p in pos]
        assert lib.launch_count() == 8 * (3 if kernel == "split" else 2)
        for _ in range(4):                                   # about 3 ms of work, so that the calls below queue up behind it
            lib.gemm(big, big, None, 0, False)
        got = [product(p, False) for p in pos]
    finally:
        lib.gemm_set_variant(0)
    _check_status(lib)
    assert all(torch.equal(x, y) for x, y in zip(got, want))
