"""GPU parity tests (pytest -m gpu) of packed sequences whose lengths are no multiples of the chunk: tails of every kind, each
regime of the decay anchors in a short chunk, neighbours that must not leak, more sequences than one table launch takes.
Tolerances as everywhere for bfloat16 (relative L2): 1e-2 outputs, 2e-2 gradients."""
import pytest
import torch

from oracle import gla_oracle as O
from test_gpu_ops import _compare, _oracle

pytestmark = pytest.mark.gpu


def _inputs(lengths, H, shift, seed):
    D, T, nseq = 128, sum(lengths), len(lengths)
    cu = [0]
    for L in lengths:
        cu.append(cu[-1] + L)
    _, g, v, k, q = O.make_inputs(1, T, H, D, torch.bfloat16, seed=seed, shift=shift)
    gen = torch.Generator().manual_seed(seed + 1)
    r = lambda *s: torch.randn(*s, generator=gen).to(torch.bfloat16)
    return cu, [r(nseq, H, D, D), g[0], v[0], k[0], q[0]], r(nseq, H, D, D), r(T, H, D)


def _run(dev, cu, x, dhf, do):
    from gla_jax_b200 import chunk_gla_packed, _lib
    leaves = [t.to(dev).requires_grad_(True) for t in x]
    hf, out = chunk_gla_packed(*leaves, cu)
    grads = torch.autograd.grad([hf, out], leaves, [dhf.to(dev), do.to(dev)])
    torch.cuda.synchronize()
    assert _lib.load().gla_device_wait_timeouts() == 0
    return hf.detach().cpu(), out.detach().cpu(), [t.cpu() for t in grads]


def _check(cu, x, dhf, do, got, seqs):
    hf, out, grads = got
    for s in seqs:
        sl = slice(cu[s], cu[s + 1])
        case = (x[0][s:s + 1], *[t[sl].unsqueeze(0) for t in x[1:]], dhf[s:s + 1], do[sl].unsqueeze(0))
        _compare(_oracle(*case), (hf[s:s + 1], out[sl].unsqueeze(0), [grads[0][s:s + 1]] + [t[sl].unsqueeze(0) for t in grads[1:]]),
                 torch.bfloat16, f"sequence {s}, {cu[s + 1] - cu[s]} tokens")


@pytest.mark.parametrize("lengths,H,shift", [
    ([1, 127, 128, 129, 2], 2, 5.0),      # one anchor at the chunk's end
    ([130, 64, 255], 1, 0.0),             # the anchor in the middle (sharp gates)
    ([200, 3, 96], 1, -3.0),              # all levels
    ([513, 31], 3, 2.0),
])
def test_ragged_tails_vs_oracle(cuda_device, lengths, H, shift):
    cu, x, dhf, do = _inputs(lengths, H, shift, 91)
    _check(cu, x, dhf, do, _run(cuda_device, cu, x, dhf, do), range(len(lengths)))


def test_a_sequence_does_not_see_its_neighbour(cuda_device):
    """The tail rows of a chunk hold the next sequence's tokens: not-a-number there must stay there."""
    cu, x, dhf, do = _inputs([70, 90, 40], 1, 5.0, 93)
    for t in x[1:] + [do]:
        t[70:160] = float("nan")
    x[0][1] = float("nan")
    dhf[1] = float("nan")
    got = _run(cuda_device, cu, x, dhf, do)
    _check(cu, x, dhf, do, got, (0, 2))


def test_many_short_sequences(cuda_device):
    lengths = [1 + (7 * i) % 19 for i in range(300)]
    cu, x, dhf, do = _inputs(lengths, 1, 5.0, 95)
    _check(cu, x, dhf, do, _run(cuda_device, cu, x, dhf, do), (0, 1, 254, 255, 256, 299))
