"""When a decoder layer runs as one autograd node: the calls that must keep the blocks' own path (no kernel is launched here)."""
import pytest
import torch

from odysseus_transformer_b200.config import get_model_config
from odysseus_transformer_b200.mesh import ParallelContext, set_context
from odysseus_transformer_b200.models import llama
from odysseus_transformer_b200.ops import functional as F
from odysseus_transformer_b200.ops import native

TOKENS = 16
ROW = 2 * (3 * 512 + 1024 + 512 + 192 + 96)      # bytes a token keeps


@pytest.fixture
def layer(request, monkeypatch):
    monkeypatch.setattr(native, "use_native", lambda t: t.dtype == torch.bfloat16)
    monkeypatch.setattr(native, "has_native_attention_bwd", lambda: True)
    ctx = ParallelContext(device=torch.device("cpu"), backend="fused")
    set_context(ctx)
    cfg = get_model_config("small-gqa").replace(hidden_size=512, num_attention_heads=4, num_key_value_heads=2, intermediate_size=96)
    kw = getattr(request, "param", {})
    return llama.DecoderLayer(cfg, ctx, kw.get("mode", "odysseus"), 0, None, kw.get("dtype", torch.bfloat16), torch.device("cpu"),
                              kw.get("zero3", True), kw.get("pack", True))


def _node(layer, dtype=torch.bfloat16, tokens=TOKENS, positions=TOKENS):
    cos, sin = F.rope_tables(torch.arange(positions), 128, 10000.0)
    return layer._one_node(torch.empty(tokens, 512, dtype=dtype), cos, sin)


@pytest.mark.parametrize("layer", [{"mode": m} for m in ("odysseus", "tpsp", "ulysses", "ring", "dp")], indirect=True)
def test_taken_on_one_gpu(layer):
    args = _node(layer)
    weights = args[-1]
    assert args[3:5] == (4, 2) and len(weights) == 6 and all(a.requires_grad for a in weights)
    assert [tuple(t.shape) for t in weights] == [(512,), (1024, 512), (512, 512), (512,), (192, 512), (512, 96)]


@pytest.mark.parametrize("layer", [{"pack": False}, {"zero3": False}, {"dtype": torch.float32}], indirect=True)
def test_other_blocks_keep_their_path(layer):
    assert _node(layer) is None


def test_watched_or_changed_layers_keep_their_path(layer, monkeypatch):
    assert _node(layer) is not None
    for m in (layer.self_attn, layer.mlp, layer.self_attn.qkv_proj, layer.self_attn.o_proj, layer.mlp.gate_up_proj, layer.mlp.down_proj):
        for register in (m.register_forward_hook, m.register_forward_pre_hook, m.register_full_backward_hook):
            h = register(lambda *a: None)
            assert _node(layer) is None
            h.remove()
        m.forward = lambda *a, **k: None
        assert _node(layer) is None
        del m.forward
    h = torch.nn.modules.module.register_module_forward_hook(lambda *a: None)
    assert _node(layer) is None
    h.remove()
    with monkeypatch.context() as p:
        p.setattr(type(layer.mlp), "forward", lambda self, x, residual=None: x)
        assert _node(layer) is None
    layer.self_attn.qkv_proj.sequence_parallel = False
    assert _node(layer) is None
    layer.self_attn.qkv_proj.sequence_parallel = True
    layer.self_attn.o_proj.bias = torch.nn.Parameter(torch.zeros(512, dtype=torch.bfloat16))
    assert _node(layer) is None
    layer.self_attn.o_proj.bias = None
    layer.mlp.down_proj.weight.requires_grad_(False)
    assert _node(layer) is None
    with torch.no_grad():
        assert _node(layer) is not None


def test_layers_with_shared_weights_keep_their_path(layer):
    """Two contributions to one gradient: the layer's backward writes each weight's gradient once, the blocks' nodes add them."""
    own = layer.post_attention_layernorm
    layer.post_attention_layernorm = layer.input_layernorm
    assert _node(layer) is None
    with torch.no_grad():
        assert _node(layer) is not None
    layer.post_attention_layernorm = own
    assert _node(layer) is not None
    weight = torch.nn.Parameter(torch.empty(512, 512, dtype=torch.bfloat16))
    layer.self_attn.o_proj.weight = layer.mlp.down_proj.weight = weight          # as for an MLP as wide as the model
    assert _node(layer) is None
    cos, sin = F.rope_tables(torch.arange(TOKENS), 128, 10000.0)
    norm = layer.input_layernorm
    with pytest.raises(ValueError, match="two places"):
        F.decoder_layer(torch.empty(TOKENS, 512), cos, sin, 4, 2, 1e-5, 0.1, (norm, own.new_empty(1), own.new_empty(2), norm, own, own))


def test_saved_tensor_hooks_see_the_blocks_tensors(layer):
    """A hook that stores, counts or converts what is saved gets the blocks' tensors, not the node's one buffer of bytes."""
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, lambda t: t):
        assert _node(layer) is None
        with torch.no_grad():
            assert _node(layer) is not None
    assert _node(layer) is not None


class _Node(torch.autograd.Function):
    """Stands in for the layer's node on the CPU: the same tensors saved, gradients of ones."""

    @staticmethod
    def forward(ctx, x, cos, sin, hq, hkv, eps, scale, *weights):
        ctx.save_for_backward(x, cos, sin, torch.zeros(64, dtype=torch.uint8), *weights)
        return x.clone()

    @staticmethod
    def backward(ctx, dy):
        x, _, _, _, *weights = ctx.saved_tensors
        return (dy, None, None, None, None, None, None, *[torch.ones_like(w) for w in weights])


@pytest.fixture
def model(monkeypatch):
    """Two checkpointed layers on the CPU that may run as one node; ``calls`` has an entry for each that did."""
    from types import SimpleNamespace
    monkeypatch.setattr(llama, "native", SimpleNamespace(use_native=lambda t: True, has_native_attention_bwd=lambda: True))
    calls = []

    def node(*args):
        calls.append(1)
        return _Node.apply(*args[:-1], *args[-1])
    monkeypatch.setattr(F, "decoder_layer", node)
    ctx = ParallelContext(device=torch.device("cpu"), backend="fused")
    set_context(ctx)
    cfg = get_model_config("small-gqa").replace(hidden_size=512, num_attention_heads=4, num_key_value_heads=2, intermediate_size=96,
                                                num_hidden_layers=2, vocab_size=64)
    m = llama.LlamaForCausalLM(cfg, "odysseus", ctx, dtype=torch.bfloat16, device=torch.device("cpu"))
    m.init_weights(0)
    m.gradient_checkpointing_enable()
    m.calls = calls
    return m


def _loss(m):
    ids = torch.arange(TOKENS).unsqueeze(0)
    return m(ids, ids, labels=ids)


def _profile():
    return torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU])


def test_recomputation_takes_the_way_of_the_forward(model):
    """A checkpoint wants the same tensors saved again; what decides between node and blocks may have changed by then."""
    loss = _loss(model)
    assert len(model.calls) == 2
    with _profile():
        loss.backward()
    assert len(model.calls) == 4 and all(p.grad is not None for p in model.layers.parameters())
    model.calls.clear()
    with _profile():
        loss = _loss(model)
    loss.backward()
    assert not model.calls
    loss = _loss(model)
    model.layers[1].mlp.register_forward_hook(lambda *a: None)
    loss.backward()
    assert len(model.calls) == 4


def test_recomputation_after_memory_was_short(model, monkeypatch):
    """The forward's fallback to the blocks holds for the recomputation; a recomputation that is short of memory says so."""
    node = F.decoder_layer

    def full(*args):
        raise torch.OutOfMemoryError("no memory")
    monkeypatch.setattr(F, "decoder_layer", full)
    loss = _loss(model)
    monkeypatch.setattr(F, "decoder_layer", node)
    loss.backward()
    assert not model.calls
    loss = _loss(model)
    monkeypatch.setattr(F, "decoder_layer", full)
    with pytest.raises(torch.OutOfMemoryError):
        loss.backward()


def test_layers_checkpointed_by_their_user_keep_their_path(model):
    """Here nothing tells the layer what its first run did."""
    from torch.utils.checkpoint import checkpoint
    cos, sin = F.rope_tables(torch.arange(TOKENS), 128, 10000.0)
    y, _ = checkpoint(model.layers[0], torch.randn(TOKENS, 512).to(torch.bfloat16), None, cos, sin, use_reentrant=False)
    with _profile():
        y.sum().backward()
    assert not model.calls and model.layers[0].input_layernorm.grad is not None


def test_replaced_layers_get_four_arguments(model):
    seen = []
    forward = model.layers[0].forward
    model.layers[0].forward = lambda x, delta, cos, sin: seen.append(1) or forward(x, delta, cos, sin)
    _loss(model).backward()
    assert len(seen) == 2


def test_other_calls_keep_their_path(layer):
    assert _node(layer, dtype=torch.float32) is None
    assert _node(layer, tokens=0) is None
    assert _node(layer, positions=TOKENS + 1) is None
    assert _node(layer, tokens=llama._ONE_NODE_BYTES // ROW) is not None
    assert _node(layer, tokens=llama._ONE_NODE_BYTES // ROW + 1) is None
    keep = F.fuse_epilogues()
    try:
        F.fuse_epilogues(rope=False)
        assert _node(layer) is None
    finally:
        F.fuse_epilogues(**keep)
    with torch.autograd.forward_ad.dual_level():
        assert _node(layer) is None
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]):
        assert _node(layer) is None
    seen = []
    torch.func.vmap(lambda t: seen.append(_node(layer)) or t)(torch.zeros(2))
    assert seen == [None]


def test_blocks_run_by_themselves_when_memory_is_short(layer, monkeypatch):
    def full(*args):
        raise torch.OutOfMemoryError("no memory")
    monkeypatch.setattr(F, "decoder_layer", full)
    called = []
    layer.self_attn.forward = lambda h, cos, sin, residual=None: called.append("attention") or residual
    layer.mlp.forward = lambda h, residual=None: called.append("mlp") or residual
    monkeypatch.setattr(layer, "_one_node", lambda *a: (1,))
    monkeypatch.setattr(F, "rmsnorm_keep", lambda x, w, eps: (x, x))
    y, delta = layer(torch.zeros(2, 512, dtype=torch.bfloat16), None, None, None)
    assert called == ["attention", "mlp"] and delta is None and y.shape == (2, 512)
