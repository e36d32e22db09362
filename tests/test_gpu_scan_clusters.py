"""GPU parity tests (pytest -m gpu) of the scan kernel where its launch rules change: every column width and alignment, axes
around a block's and a cluster's rows, clusters up to sixteen blocks, both directions, every combine rule."""
import pytest
import torch

from oracle import gla_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,T,D,reverse,dtype", [
    (3, 64, 256, False, torch.float32),      # four columns per lane, a block's rows exactly
    (3, 65, 256, True, torch.float32),       # two per lane from here on
    (2, 129, 192, True, torch.float32),
    (1, 256, 33, False, torch.float32), (1, 257, 31, True, torch.float32),     # one per lane; two blocks of a cluster
    (1, 4096, 32, False, torch.float32),     # sixteen blocks, every one full
    (1, 4097, 40, True, torch.float32),      # ... and one row in the second step
    (2, 9000, 3, False, torch.float32),
    (1, 2049, 64, True, torch.bfloat16), (2, 700, 65, False, torch.bfloat16), (5, 1, 130, False, torch.bfloat16),
    (700, 20, 128, True, torch.float32),     # more blocks than one wave, no cluster
])
def test_cumsum_where_the_launch_rules_change(cuda_device, N, T, D, reverse, dtype):
    from gla_jax_b200 import cumsum_recursive
    gen = torch.Generator().manual_seed(N + T + D)
    x = torch.randn(N, T, D, generator=gen).to(dtype)
    init = torch.randn(N, D, generator=gen).to(dtype)
    ref = O.cumsum(x, 1, init=init, reverse=reverse, out_dtype=torch.float64, compute_dtype=torch.float64)
    y = cumsum_recursive(x.to(cuda_device), axis=1, init=init.to(cuda_device), reverse=reverse).cpu()
    # float32: sqrt(T) roundings of 2^-24 of the running sum; bf16: one rounding of the result
    assert O.rel_l2(ref, y.double()) < (max(T, 16) ** 0.5 * 6e-8 if dtype == torch.float32 else 2.5e-3)


@pytest.mark.parametrize("rule,ref", [("max", lambda x: torch.cummax(x, 1)[0]), ("min", lambda x: torch.cummin(x, 1)[0]),
                                      ("logaddexp", lambda x: torch.logcumsumexp(x, 1)), ("mul", lambda x: torch.cumprod(x, 1))])
def test_rules_across_a_cluster(cuda_device, rule, ref):
    from gla_jax_b200 import scan
    x = 1.0 + 0.01 * torch.randn(2, 3000, 20, generator=torch.Generator().manual_seed(5))
    # running products accumulate a rounding per factor, logaddexp one of the argument's size per step
    assert O.rel_l2(ref(x.double()), scan(rule, x.to(cuda_device), 1).cpu().double()) < 3e-5
