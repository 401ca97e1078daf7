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
