"""How gradients reach ``main_grad`` where a kernel may write them there itself: the switches, hooks and refusals of the
general path hold.  The extension is replaced by a recorder, so the choice of the path is tested without a GPU."""
import pytest
import torch

from odysseus_transformer_b200.ops import functional as F
from odysseus_transformer_b200.ops import native


class _Recorder:
    """Stands in for the extension: notes which kernels were asked for."""

    def __init__(self):
        self.calls = []

    def embedding_grad_(self, dy, ids, dw):
        self.calls.append("embedding_grad_")
        dw.zero_().index_add_(0, ids, dy)


@pytest.fixture
def recorder(monkeypatch):
    rec = _Recorder()
    monkeypatch.setattr(native, "use_native", lambda t: True)
    monkeypatch.setattr(native, "lib", lambda: rec)
    return rec


def _embedding_grad(dtype=torch.bfloat16):
    w = torch.zeros(32, 8, dtype=dtype, requires_grad=True)
    w.main_grad = torch.full((32, 8), float("nan"), dtype=dtype)
    ids = torch.tensor([3, 1, 3, 7])
    dy = torch.arange(32, dtype=dtype).view(4, 8)
    F.embedding(ids, w).backward(dy)
    want = torch.zeros(32, 8, dtype=dtype).index_add_(0, ids, dy)
    assert torch.equal(w.main_grad, want) and w.grad is None


def test_embedding_gradient_takes_the_kernel(recorder):
    _embedding_grad()
    assert recorder.calls == ["embedding_grad_"]


@pytest.mark.parametrize("warn_only", [False, True])
def test_embedding_gradient_obeys_deterministic_algorithms(recorder, warn_only):
    """The kernel adds rows that tokens share in no fixed order; index_add_ has an ordered form under this switch."""
    before, warn = torch.are_deterministic_algorithms_enabled(), torch.is_deterministic_algorithms_warn_only_enabled()
    torch.use_deterministic_algorithms(True, warn_only=warn_only)
    try:
        _embedding_grad()
    finally:
        torch.use_deterministic_algorithms(before, warn_only=warn)
    assert recorder.calls == []


def _chunked_loss(device="cpu", dtype=torch.float32):
    g = torch.Generator().manual_seed(0)
    h = torch.randn(6, 16, generator=g).to(device, dtype).requires_grad_(True)
    w = torch.randn(24, 16, generator=g).to(device, dtype).requires_grad_(True)
    t = torch.randint(24, (6,), generator=g).to(device)
    return h, w, lambda: F.linear_cross_entropy_sum(h, w, t, 0.5, None, 4)


def check_recorded_backward(device, dtype):
    """The incoming gradient is a tensor like any other: a backward that is itself recorded goes through it."""
    h, w, loss = _chunked_loss(device, dtype)
    dh, dw = torch.autograd.grad(loss(), (h, w))
    for main_grad in (False, True):
        if main_grad:
            w.main_grad = torch.zeros_like(w)
        s = torch.tensor(2.0, device=device, requires_grad=True)
        (g,) = torch.autograd.grad(loss() * s, h, create_graph=True) if main_grad else \
            torch.autograd.grad(loss() * s, (h, w), create_graph=True)[:1]
        torch.testing.assert_close(g.detach(), 2 * dh)
        (ds,) = torch.autograd.grad(g.float().sum(), s)
        torch.testing.assert_close(ds, dh.float().sum(), rtol=1e-2, atol=1e-3)
    del w.main_grad
    # several incoming gradients at once
    seeds = torch.tensor([1.0, -2.0, 0.5], device=device)
    many = torch.autograd.grad(loss(), (h, w), seeds, is_grads_batched=True)
    for got, one in zip(many, (dh, dw)):
        torch.testing.assert_close(got, torch.stack([one * c for c in seeds.to(dtype)]))


def test_recorded_backward_of_the_chunked_loss():
    check_recorded_backward("cpu", torch.float32)


def test_chunked_loss_refuses_a_gradient_buffer_of_another_shape():
    h, w, loss = _chunked_loss()
    w.main_grad = torch.zeros(w.numel())
    with pytest.raises(RuntimeError):
        loss().backward()
    assert w.main_grad.shape == (w.numel(),)


@pytest.mark.parametrize("fn", ["rmsnorm", "add_rmsnorm", "rmsnorm_keep"])
def test_norm_refuses_a_gradient_buffer_of_another_shape(recorder, fn):
    """What ``deliver_grad`` refuses - a buffer that the gradient does not broadcast to - the kernel's route refuses too."""
    z = torch.zeros
    recorder.rmsnorm_fwd = lambda x, w, eps: (z(4, 8), z(4))
    recorder.add_rmsnorm_fwd = lambda x, d, w, eps: (z(4, 8), z(4, 8), z(4))

    def bwd(dy, x, w, rstd, ds, dw_out=None):
        recorder.calls.append(dw_out is not None)
        return z(4, 8), z(8)
    recorder.rmsnorm_bwd = bwd
    x = torch.randn(4, 8, requires_grad=True)
    for shape, ok in (((8,), True), ((8, 1), False)):
        w = torch.ones(8, dtype=torch.bfloat16, requires_grad=True)
        w.main_grad = torch.zeros(shape, dtype=torch.bfloat16)
        args = (x, x.detach(), w, 1e-5) if fn == "add_rmsnorm" else (x, w, 1e-5)
        y = getattr(F, fn)(*args)
        y = y if torch.is_tensor(y) else y[0] + y[1]
        if ok:
            y.sum().backward()
        else:
            with pytest.raises(RuntimeError):
                y.sum().backward()
    assert recorder.calls == [True, False]
