"""The rule that sends products with few output tiles to clusters that share K: what it answers is what the kernel takes."""
import ctypes
import os
import random

import pytest

import odysseus_transformer_b200

SO = os.path.join(os.path.dirname(odysseus_transformer_b200.__file__), "_C.so")


@pytest.fixture(scope="module")
def plan():
    if not os.path.exists(SO):
        pytest.skip("extension not built")
    import torch  # noqa: F401  (libtorch symbols must be loaded first)
    lib = ctypes.CDLL(SO)

    def f(M, N, K, rope=0):
        bn, s = ctypes.c_int(), ctypes.c_int()
        return (bn.value, s.value) if lib.ody_gemm_cluster_plan(M, N, K, rope, ctypes.byref(bn), ctypes.byref(s)) else None
    return f


def test_what_the_kernel_takes(plan):
    rng = random.Random(0)
    seen = set()
    for _ in range(20000):
        M, N, K = (max(1, int(2 ** rng.uniform(0, 15))) for _ in range(3))
        N = max(8, N // 8 * 8)
        for rope in (0, 1):
            p = plan(M, N, K, rope)
            if p is None:
                continue
            bn, s = p
            kblocks = -(-K // 64)
            ctas = -(-M // 128) * -(-N // bn) * s
            assert bn in (64, 128) and (bn == 128 or not rope) and 1 <= s <= min(8, kblocks) and s & (s - 1) == 0
            assert ctas <= 148 and -(-kblocks // s) <= 192
            seen.add(p)
    assert len(seen) >= 6                                     # both tiles, several shares


def test_where_the_line_lies(plan):
    assert plan(128, 3072, 1024) and plan(512, 1024, 2816) and plan(2048, 1024, 5632)
    assert plan(8192, 4096, 4096) is None and plan(4096, 1024, 1024) is None          # more tiles than SMs
    assert plan(1024, 1024, 32000) is None                                             # K too long for narrow tiles
    assert plan(128, 256, 4096) and plan(512, 64, 12288)      # also where a split would take more CTAs than a cluster has
    assert plan(128, 256, 32000) is None                      # so long a K that 32 CTAs and a sum are expected to be as fast
    for bad in ((0, 8, 8), (8, 0, 8), (8, 8, 0), (128, 1020, 1024)):
        assert plan(*bad) is None
