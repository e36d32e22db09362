"""Head size 256: a backward block covers both value blocks of a key block, whichever path its gates take."""
import pytest
import torch

from test_gpu_ops import _case, _compare, _oracle, _run_gpu

pytestmark = pytest.mark.gpu

# mean log gate of (key block 0, key block 1): end anchor, middle anchor and all levels
GATES = {"end": (-0.01, -0.3), "end_and_middle": (-0.01, -0.8), "end_and_levels": (-0.01, -2.0), "levels_and_middle": (-2.0, -0.8)}


# (more chunks than SMs: the forward's blocks take several each)
@pytest.mark.parametrize("B,T,H", [(1, 128, 1), (2, 384, 3), (1, 1280, 4)])
@pytest.mark.parametrize("gates", sorted(GATES))
def test_key_blocks_on_different_paths(cuda_device, gates, B, T, H):
    from gla_jax_b200 import chunk_gla, _lib
    h, g, v, k, q, dhf, do = _case(B, T, H, 256, torch.bfloat16, 41, 5.0)
    gen = torch.Generator().manual_seed(5)
    for a, mean in enumerate(GATES[gates]):
        # chunks of one head alternate between the given mean and a mild one, so that a block meets several paths
        x = mean * (1.0 + 0.2 * torch.rand(B, T, H, 128, generator=gen))
        x[:, (torch.arange(T) // 128) % 3 == 1] *= 0.005
        g[..., 128 * a:128 * a + 128] = x
    case = (h, g, v, k, q, dhf, do)
    got = _run_gpu(chunk_gla, cuda_device, *case, chunk_size=128, impl="tcgen05")
    again = _run_gpu(chunk_gla, cuda_device, *case, chunk_size=128, impl="tcgen05")
    assert _lib.load().gla_device_wait_timeouts() == 0
    _compare(_oracle(*case), got, torch.bfloat16, gates)
    assert all(torch.equal(x, y) for x, y in zip((got[0], got[1], *got[2]), (again[0], again[1], *again[2])))
