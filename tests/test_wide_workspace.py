"""Size of the forward's workspace at head size 256 (no GPU needed)."""
import pytest


@pytest.mark.parametrize("B,T,H", [(1, 128, 1), (1, 1024, 4), (2, 16384, 8), (16, 16384, 8)])
def test_workspace_at_head_size_256_holds_no_more_than_one_output_per_key_block(B, T, H):
    from gla_jax_b200 import build, _lib
    build.build()
    lib = _lib.load()
    n = lib.gla_chunk_fwd_workspace_bytes(B, T, H, 256, 256 if T >= 256 else 128, _lib.GLA_BF16, _lib.IMPL_BY_NAME["tcgen05"])
    heads, chunks = 4 * B * H, T // 128
    states = heads * chunks * (128 * 128 * 2 + 128 * 4) + 2 * heads * 128 * 128 * 2
    assert states < n <= states + heads * T * 128 * 2         # an output per key block, as callers may have sized it
