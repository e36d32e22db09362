"""Sizes that gla_chunk_fwd_static accepts (no GPU needed: what is accepted goes on to the device, what is not does not)."""
import ctypes

import pytest
import torch

LIMIT = 32 << 20


def _limit_need(T, H, D, C):
    """What the kernels that the limit was set for keep: lam, q^, k^ (or scores), a state and a total decay per chunk."""
    up = lambda n: (4 * n + 255) // 256 * 256
    n = H * (T // C)
    return 2 * up(T * H * D) + up(T * H * max(D, C)) + up(n * D * D) + up(n * D)


def _accepted(T, H, D, C, dtype, impl=0):
    from gla_jax_b200 import build, _lib
    build.build()
    lib = _lib.load()
    assert lib.gla_chunk_fwd_static_max_bytes() == LIMIT
    p, dt = ctypes.c_void_p(4096), _lib.GLA_F32 if dtype == "f32" else _lib.GLA_BF16
    st = lib.gla_chunk_fwd_static(None, 1, T, H, D, C, dt, impl, p, p, p, p, p, p, p)
    assert st != 0
    return st != 8          # 8: too large


no_gpu = pytest.mark.skipif(torch.cuda.is_available(), reason="the pointers are none")


# below 32 MiB for the kernels that keep kv products and scores; the split-operand kernels keep more states than those
@no_gpu
@pytest.mark.parametrize("T,H,C,dtype", [(16256, 1, 128, "f32"), (128, 102, 64, "bf16"), (64, 200, 64, "bf16")])
def test_sizes_at_the_scratch_limit_stay_accepted(T, H, C, dtype):
    assert _limit_need(T, H, 128, C) <= LIMIT and _accepted(T, H, 128, C, dtype)


@no_gpu
@pytest.mark.parametrize("dtype", ["f32", "bf16"])
@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("C", [16, 32, 64, 128, 256])
def test_every_size_up_to_the_limit_is_accepted(D, C, dtype):
    for chunks in (1, 2, 3, 7):                 # the most heads that fit
        heads = 1
        while _limit_need(chunks * C, heads + 1, D, C) <= LIMIT:
            heads += 1
        assert _accepted(chunks * C, heads, D, C, dtype, impl=1)
        assert not _accepted(chunks * C, heads + 1 + heads // 50, D, C, dtype, impl=1)
    n = 1                                       # one head, the longest sequence
    while _limit_need((n + 1) * C, 1, D, C) <= LIMIT:
        n += 1
    assert _accepted(n * C, 1, D, C, dtype, impl=1)
