"""Calls of the autograd functions with gradients off: the same values, and what ``apply`` refuses stays refused."""
import pytest
import torch

from odysseus_transformer_b200.ops import functional as F


def _calls():
    g = torch.Generator().manual_seed(0)
    r = lambda *s: torch.randn(*s, generator=g)   # noqa: E731
    x, w, gu = r(6, 16), r(8, 16), r(6, 32)
    q, k, v = r(6, 4, 8), r(6, 2, 8), r(6, 2, 8)
    cos, sin = F.rope_tables(torch.arange(6), 8, 10000.0)
    return {
        "linear": lambda: F.linear(x, w),
        "rmsnorm": lambda: F.rmsnorm(x, w[0], 1e-5),
        "add_rmsnorm": lambda: F.add_rmsnorm(x, x + 1, w[0], 1e-5),
        "rmsnorm_keep": lambda: F.rmsnorm_keep(x, w[0], 1e-5),
        "rope": lambda: F.rope(q, cos, sin),
        "swiglu": lambda: F.swiglu(gu),
        "attention": lambda: F.attention(q, k, v, True),
        "embedding": lambda: F.embedding(torch.tensor([3, 1, 3]), w),
    }


@pytest.mark.parametrize("name", sorted(_calls()))
def test_same_values_without_gradients(name):
    want = _calls()[name]()
    with torch.no_grad():
        got = _calls()[name]()
    want, got = [(t,) if torch.is_tensor(t) else t for t in (want, got)]
    for a, b in zip(want, got):
        assert torch.equal(a, b) and not b.requires_grad


def test_no_saved_state_is_kept():
    x = torch.randn(4, 8, requires_grad=True)
    with torch.no_grad():
        y = F.rmsnorm(x, torch.ones(8), 1e-5)
    assert y.grad_fn is None


def test_transforms_are_not_bypassed():
    x, w = torch.randn(3, 4, 8), torch.randn(5, 8)
    with torch.no_grad():
        with pytest.raises(RuntimeError):                      # no vmap rule, with or without gradients
            torch.func.vmap(lambda t: F.linear(t, w))(x)
        with torch.autograd.forward_ad.dual_level():
            d = torch.autograd.forward_ad.make_dual(x[0], torch.ones_like(x[0]))
            with pytest.raises((RuntimeError, NotImplementedError)):
                F.linear(d, w)


def test_tensors_left_over_from_a_transform_are_unwrapped():
    """``apply`` unwraps a tensor that outlived its transform; a kernel cannot read one and says so."""
    kept = []

    def f(x):
        kept.append(x)
        return (x * x).sum()
    torch.func.grad(f)(torch.ones(3, 8))

    class Kernel(torch.autograd.Function):
        @staticmethod
        def forward(ctx, x, n):
            if torch._C._functorch.is_functorch_wrapped_tensor(x):
                raise RuntimeError("no storage")
            if n < 0:
                raise RuntimeError("refused")
            return x * n
    with torch.no_grad():
        assert torch.equal(F.call(Kernel, kept[0], 2.0), torch.full((3, 8), 2.0))
        with pytest.raises(RuntimeError, match="refused"):
            F.call(Kernel, torch.ones(2), -1.0)
        with pytest.raises(RuntimeError, match="refused"):
            F.call(Kernel, kept[0], -1.0)


def test_a_profile_names_the_operators():
    calls = _calls()
    with torch.no_grad(), torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]) as prof:
        calls["rmsnorm"]()
        calls["linear"]()
    names = {e.name for e in prof.events()}
    assert {"_RMSNorm", "_Linear"} <= names
