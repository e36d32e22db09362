"""GPU test (pytest -m gpu): a decode step on a state whose base is not 16-byte aligned (scalar accesses) equals the aligned
one, at every head size."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [32, 64, 128, 256])
def test_decode_step_on_an_unaligned_state(cuda_device, D):
    from gla_jax_b200 import decode_step
    gen = torch.Generator().manual_seed(D)
    x = [torch.randn(2, 3, D, generator=gen).to(cuda_device) for _ in range(4)]
    x[0] = -x[0].abs()
    a = torch.randn(2, 3, D, D, generator=gen).to(cuda_device)
    buf = torch.empty(a.numel() + 1, device=cuda_device)
    b = buf[1:].view(2, 3, D, D)
    b.copy_(a)
    assert b.data_ptr() % 16 != 0 and b.is_contiguous()
    assert torch.equal(decode_step(a, *x), decode_step(b, *x)) and torch.equal(a, b)
