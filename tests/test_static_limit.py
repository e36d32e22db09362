"""Sizes that gla_chunk_fwd_static accepts (no GPU needed: what is accepted goes on to the device, what is not does not)."""
import ctypes

import pytest
import torch


# below 32 MiB for the kernels that keep kv products and scores, above it with one state more per head
@pytest.mark.parametrize("T,H,C,dtype", [(16256, 1, 128, "f32"), (128, 102, 64, "bf16"), (64, 200, 64, "bf16")])
def test_sizes_at_the_scratch_limit_stay_accepted(T, H, C, dtype):
    from gla_jax_b200 import build, _lib
    build.build()
    lib = _lib.load()
    dt = 0 if dtype == "f32" else _lib.GLA_BF16
    need = lib.gla_chunk_fwd_workspace_bytes(1, T, H, 128, C, dt, 0)
    assert lib.gla_chunk_fwd_static_max_bytes() < need < lib.gla_chunk_fwd_static_max_bytes() + (9 << 20)
    if not torch.cuda.is_available():
        p = ctypes.c_void_p(4096)
        assert lib.gla_chunk_fwd_static(None, 1, T, H, 128, C, dt, 0, p, p, p, p, p, p, p) not in (0, 8)    # 8: too large
