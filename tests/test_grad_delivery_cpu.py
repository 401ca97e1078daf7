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
