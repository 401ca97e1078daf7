"""The rule that splits the streamed dimension of the attention kernels (csrc/attn_split.cuh): host code of the extension."""
import ctypes
import os

import pytest

pytest.importorskip("torch")


@pytest.fixture(scope="module")
def cdll():
    import torch  # noqa: F401  (the extension links against libtorch)
    import odysseus_transformer_b200
    path = os.path.join(os.path.dirname(odysseus_transformer_b200.__file__), "_C.so")
    if not os.path.exists(path):
        pytest.skip("extension not built")
    from odysseus_transformer_b200.ops import native
    try:
        native.lib()
    except Exception:
        pass
    lib = ctypes.CDLL(path)
    for f, n in ((lib.ody_flash_fwd_split_bytes, 4), (lib.ody_flash_bwd_split_bytes, 5)):
        f.restype, f.argtypes = ctypes.c_int64, [ctypes.c_int] * n
    return lib


def test_scratch_is_bounded_and_absent_for_full_grids(cdll):
    for T in (1, 127, 128, 129, 1000, 4097, 10007, 32768, 131072):
        for Tk in (1, 128, 1000, 8192, 131072):
            for H, Hkv in ((1, 1), (4, 1), (8, 2), (32, 8), (32, 32)):
                for causal in ((0, 1) if T == Tk else (0,)):
                    f = cdll.ody_flash_fwd_split_bytes(T, Tk, H, causal)
                    b = cdll.ody_flash_bwd_split_bytes(T, Tk, H, Hkv, causal)
                    assert 0 <= f <= 256 << 20 and 0 <= b <= 256 << 20
                    assert f % 16 == 0 and b % 16 == 0
                    if -(-T // 256) * H > 6 * 148:
                        assert f == 0


def test_idle_grids_are_split(cdll):
    assert cdll.ody_flash_bwd_split_bytes(10007, 10007, 4, 1, 1) > 0      # 79 dK/dV CTAs of up to 316 blocks
    assert cdll.ody_flash_fwd_split_bytes(256, 8192, 1, 0) > 0            # one CTA
    assert cdll.ody_flash_fwd_split_bytes(8192, 8192, 32, 1) == 0
    assert cdll.ody_flash_bwd_split_bytes(0, 0, 1, 1, 1) == 0
