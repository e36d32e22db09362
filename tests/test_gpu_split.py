"""GPU parity tests (pytest -m gpu) of the float32-precision chunk kernels: chunk edges, every head size they serve, element
types, directions, and chunks on both sides of the gate limits, against the float64 oracle.

Tolerances (relative L2).  bfloat16: 1e-2 outputs, 2e-2 gradients.  float32: operand splits keep 24 bits, so what is left is
float32 rounding: a state or a row is a sum of up to T (here <= 300) terms with a running product of up to 64 gates in
front of each, about (sqrt(300) + 64) 2^-24 = 5e-6; the gate gradient is a running sum of terms that cancel, twice that.
With gates around log f = shift < 0 every token's own contribution (the same in q dq and k dk, where it cancels) is
exp(-shift) times what is left of the gate gradient, and so is the rounding error that it leaves there.
"""
import math

import pytest
import torch

from oracle import gla_oracle as O
from test_gpu_ops import NAMES, _case, _oracle, _run_gpu

pytestmark = pytest.mark.gpu


def _check(ref, got, dtype, what, shift=5.0):
    tol_f, tol_g = (1e-2, 2e-2) if dtype == torch.bfloat16 else (5e-6, 1e-5)
    errs = {"hidden_final": O.rel_l2(ref[0], got[0]), "out": O.rel_l2(ref[1], got[1])}
    errs.update({n: O.rel_l2(a, b) for n, a, b in zip(NAMES, ref[2], got[2])})
    tol = {n: tol_f if n in ("hidden_final", "out") else tol_g for n in errs}
    tol["dlog_fgate"] *= math.exp(max(0.0, -shift))
    bad = {n: e for n, e in errs.items() if not e < tol[n]}
    assert not bad, f"{what}: {bad} (all: {errs})"


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("B,T,H,D,shift,reverse", [
    (1, 48, 1, 64, 5.0, False),       # the shortest sequence that takes the chunked form, one partial chunk
    (2, 64, 2, 32, 5.0, False),       # exactly one chunk
    (1, 65, 3, 64, 5.0, True),        # one row in the second chunk, reversed
    (1, 129, 2, 128, 2.0, False),
    (1, 300, 1, 128, 0.0, True),      # sharp gates, reversed, short last chunk
    (2, 97, 1, 32, 0.0, True),
    (1, 127, 2, 64, -4.0, False),     # past the limit: every chunk pair by pair
    (1, 100, 1, 128, -4.0, False),
    (1, 70, 1, 32, -4.0, True),
])
def test_recurrent_gla_in_chunks_vs_oracle(cuda_device, B, T, H, D, shift, reverse, dtype):
    from gla_jax_b200 import recurrent_gla
    case = _case(B, T, H, D, dtype, 7, shift)
    ref = _oracle(*case, reverse=reverse)
    got = _run_gpu(recurrent_gla, cuda_device, *case, reverse=reverse)
    _check(ref, got, dtype, f"recurrent {B, T, H, D, shift, reverse, dtype}", shift)


@pytest.mark.parametrize("D", [32, 64, 128])
def test_gates_that_one_thread_holds(cuda_device, D):
    """Eight consecutive gates just inside and just beyond what the weights of one thread's rows may fall by together."""
    from gla_jax_b200 import recurrent_gla
    for total in (79.0, 81.0):
        case = _case(1, 200, 1, D, torch.float32, 19, 5.0)
        case[1][0, 16:24, 0] = -total / 8
        _check(_oracle(*case), _run_gpu(recurrent_gla, cuda_device, *case), torch.float32, f"group {D, total}")


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("B,T,H,D,shift,reverse", [
    (8, 48, 2, 64, 5.0, False), (4, 65, 4, 64, 5.0, True), (16, 49, 1, 32, 0.0, False), (4, 97, 4, 32, 5.0, True),
    (8, 64, 2, 128, 5.0, False), (4, 65, 4, 128, 0.0, True), (8, 127, 2, 128, -4.0, False),     # enough heads for chunks
    (1, 95, 2, 64, 5.0, False), (1, 96, 2, 64, 5.0, True), (1, 191, 2, 128, 5.0, True), (1, 192, 2, 128, 5.0, False),
    (3, 64, 5, 128, 5.0, False), (4, 64, 4, 128, 5.0, True),                                    # both sides of the rules
])
def test_either_side_of_the_dispatch_by_heads(cuda_device, B, T, H, D, shift, reverse, dtype):
    from gla_jax_b200 import recurrent_gla
    case = _case(B, T, H, D, dtype, 27, shift)
    _check(_oracle(*case, reverse=reverse), _run_gpu(recurrent_gla, cuda_device, *case, reverse=reverse), dtype,
           f"recurrent {B, T, H, D, shift, reverse, dtype}", shift)


@pytest.mark.parametrize("D", [32, 64, 128])
def test_chunks_on_both_sides_of_the_gate_limits(cuda_device, D):
    """Three chunks: mild, one feature past the sum limit, one single gate whose exponential vanishes (and an infinite one)."""
    from gla_jax_b200 import chunk_gla, recurrent_gla
    h, g, v, k, q, dhf, do = _case(1, 192, 2, D, torch.float32, 9, 5.0)
    g[0, 64:128, 1, 3] = -3.0
    g[0, 140, 0, 5] = -95.0
    for fn, kw in ((chunk_gla, dict(chunk_size=64)), (recurrent_gla, {})):
        ref = _oracle(h, g, v, k, q, dhf, do)
        _check(ref, _run_gpu(fn, cuda_device, h, g, v, k, q, dhf, do, **kw), torch.float32, f"limits {D} {fn.__name__}")
    g[0, 150, 1, 7] = -float("inf")       # forget everything: the state row restarts
    hf, out = recurrent_gla(*[x.to(cuda_device) for x in (h, g, v, k, q)])
    hf0, out0 = O.recurrent_gla_naive(*[x[0].double() for x in (h, g, v, k, q)])
    assert O.rel_l2(hf0, hf[0].cpu()) < 5e-6 and O.rel_l2(out0, out[0].cpu()) < 5e-6


@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("gate,at", [(-1e4, (70,)), (-1e4, (5, 64, 100, 127)), (-float("inf"), (3, 40, 41, 90)),
                                     (-100.0, (20, 63, 80)), (-float("inf"), tuple(range(2, 130, 9)))])
def test_resets_in_every_feature(cuda_device, D, gate, at):
    """Tokens whose gate resets the whole state, mild gates in between: what follows a reset keeps its precision."""
    from gla_jax_b200 import recurrent_gla
    case = _case(1, 200, 2, D, torch.float32, 15, 5.0)
    case[1][:, list(at)] = gate
    _check(_oracle(*case), _run_gpu(recurrent_gla, cuda_device, *case), torch.float32, f"resets {D, gate, at}")


@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("shift,gate", [(5.0, None), (0.0, None), (5.0, -30.0), (5.0, -55.0)])
def test_float32_rounding_and_no_more(cuda_device, D, shift, gate):
    """A weight is a product of up to 64 rounded factors, a sum has up to 12 float32 additions of 16 products each; with a
    mean square of 2^-24 / sqrt(3) per rounding that is (8 + 3.5) 3.4e-8 = 4e-7.  The gate gradient (float32 for bf16
    callers too) is a sum of terms that cancel: three times that."""
    from gla_jax_b200 import recurrent_gla
    case = _case(1, 192, 2, D, torch.float32, 17, shift)
    if gate is not None:
        case[1][:, [5, 90, 180]] = gate
    ref, got = _oracle(*case), _run_gpu(recurrent_gla, cuda_device, *case)
    errs = [O.rel_l2(a, b) for a, b in zip((ref[0], ref[1], *ref[2]), (got[0], got[1], *got[2]))]
    bound = [4e-7, 4e-7, *(1.2e-6 if n == "dlog_fgate" else 4e-7 for n in NAMES)]
    assert all(e < b for e, b in zip(errs, bound)), errs
    half = [x if i == 1 else x.to(torch.bfloat16) for i, x in enumerate(case)]
    i = NAMES.index("dlog_fgate")
    assert O.rel_l2(_oracle(*half)[2][i], _run_gpu(recurrent_gla, cuda_device, *half)[2][i]) < 1.2e-6


def _same_where_finite(ref, got, tol, what):
    """Not finite in the same places as the recurrence, and equal elsewhere (an infinity may be either kind)."""
    ok = torch.isfinite(ref)
    assert torch.equal(ok, torch.isfinite(got)), what
    zero = torch.zeros((), dtype=torch.float64)
    assert O.rel_l2(torch.where(ok, ref.double(), zero), torch.where(ok, got.double(), zero)) < tol, what


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("which,bad,t", [("v", float("nan"), 27), ("v", float("inf"), 75), ("k", float("nan"), 90),
                                         ("k", -float("inf"), 5), ("q", float("nan"), 70), ("do", float("inf"), 45)])
@pytest.mark.parametrize("D", [32, 64, 128])
def test_what_is_not_finite_stays_where_the_recurrence_has_it(cuda_device, D, which, bad, t, dtype):
    """One bad value in a token: earlier tokens (later ones for gradients that run backwards) do not see it."""
    from gla_jax_b200 import recurrent_gla
    case = list(_case(1, 200, 2, D, dtype, 21, 5.0))
    case[{"v": 2, "k": 3, "q": 4, "do": 6}[which]][0, t, 1, 7] = bad
    leaves = [x.to(cuda_device).requires_grad_(True) for x in case[:5]]
    hf, out = recurrent_gla(*leaves)
    grads = torch.autograd.grad([hf, out], leaves, [x.to(cuda_device) for x in case[5:]])
    ref = _oracle(*case)
    tol = 5e-6 if dtype == torch.float32 else 1e-2
    for name, a, b in zip(("hidden_final", "out", *NAMES), (ref[0], ref[1], *ref[2]), (hf, out, *grads)):
        if name != "dlog_fgate":        # (a sum over later tokens here, a product per token in the oracle)
            _same_where_finite(a, b.detach().cpu(), tol, name)


@pytest.mark.parametrize("D", [32, 64, 128])
def test_large_values_under_strong_decay(cuda_device, D):
    """Keys whose weighted values exceed float32 although no state or output does."""
    from gla_jax_b200 import recurrent_gla
    case = list(_case(1, 192, 1, D, torch.float32, 23, 5.0))
    case[1][:] = -1.5
    case[3] = case[3] * 1e18
    _check(_oracle(*case), _run_gpu(recurrent_gla, cuda_device, *case), torch.float32, f"large keys {D}", shift=-1.5)


def test_naive_with_bf16_inputs_and_float32_cotangent(cuda_device):
    """bf16 operands with a float32 output and output gradient (recurrent_gla_naive), head size 128: shorter chunks."""
    from gla_jax_b200 import recurrent_gla_naive
    h, g, v, k, q, dhf, do = _case(1, 150, 2, 128, torch.bfloat16, 11, 5.0)
    do = do.float() + 1e-3 * torch.randn(do.shape, generator=torch.Generator().manual_seed(1))
    leaves = [x.to(cuda_device).requires_grad_(True) for x in (h, g, v, k, q)]
    hf, out = recurrent_gla_naive(*leaves)
    assert out.dtype == torch.float32
    grads = torch.autograd.grad([hf, out], leaves, [dhf.to(cuda_device), do.to(cuda_device)])
    ref = _oracle(h, g, v, k, q, dhf, do)
    assert O.rel_l2(ref[1], out.detach().cpu()) < 5e-6
    _check((ref[0], ref[0], ref[2]), (hf.detach().cpu(), hf.detach().cpu(), [x.cpu() for x in grads]), torch.bfloat16, "naive")


def test_without_room_for_the_states_the_tokens_are_walked(cuda_device):
    """recurrent_gla where the device has no room for the chunks' states: it runs as it does without a workspace."""
    from gla_jax_b200 import recurrent_gla, _lib
    case = _case(1, 4096, 4, 128, torch.float32, 25, 5.0)
    x = [t.to(cuda_device).requires_grad_(True) for t in case[:5]]
    co = [t.to(cuda_device) for t in case[5:]]
    with torch.no_grad():
        full = [t.cpu() for t in recurrent_gla(*x)]
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    lib = _lib.load()
    need, least = (lib.gla_recurrent_bwd_workspace_bytes_dout(1, 4096, 4, 128, 0, 0, n) for n in (0, 1))
    assert lib.gla_recurrent_fwd_workspace_bytes(1, 4096, 4, 128, 0) > 16 << 20 and need > 64 << 20 > 3 * least
    # outputs and gradients take about 7 arrays of 8 MiB, the walk's scratch 16 MiB; the states 33 and 67 MB
    total = torch.cuda.get_device_properties(cuda_device).total_memory
    try:
        with torch.no_grad():
            torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (24 << 20)) / total)
            hf, out = recurrent_gla(*x)
        assert O.rel_l2(full[0], hf.cpu()) < 5e-6 and O.rel_l2(full[1], out.cpu()) < 5e-6
        torch.cuda.set_per_process_memory_fraction(1.0)
        hf, out = recurrent_gla(*x)
        torch.cuda.empty_cache()
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (72 << 20)) / total)
        walked = torch.autograd.grad([hf, out], x, co, retain_graph=True)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    for n, a, b in zip(NAMES, torch.autograd.grad([hf, out], x, co), walked):
        assert O.rel_l2(a.cpu(), b.cpu()) < 1e-5, n


def test_wait_for_workspace_is_not_needed(cuda_device):
    """The entry point without a workspace walks the tokens; with one it runs chunks: same results to float32 rounding."""
    from gla_jax_b200 import _lib
    lib = _lib.load()
    h, g, v, k, q, _, _ = [x.to(cuda_device) for x in _case(1, 200, 2, 64, torch.float32, 13, 5.0)]
    st = _lib.stream_of(v.device)
    res = []
    for ws_n in (0, lib.gla_recurrent_fwd_workspace_bytes(1, 200, 2, 64, _lib.GLA_F32)):
        ws = torch.empty(max(ws_n, 1), dtype=torch.uint8, device=cuda_device)
        hf, out = torch.empty_like(h), torch.empty_like(v)
        _lib.check(lib.gla_recurrent_fwd_ws(st, 1, 200, 2, 64, _lib.GLA_F32, h.data_ptr(), g.data_ptr(), v.data_ptr(), k.data_ptr(),
                                            q.data_ptr(), hf.data_ptr(), out.data_ptr(), _lib.GLA_F32, 0,
                                            ws.data_ptr() if ws_n else None, ws_n), "gla_recurrent_fwd_ws")
        res.append((hf.cpu(), out.cpu()))
    assert O.rel_l2(res[0][0], res[1][0]) < 5e-6 and O.rel_l2(res[0][1], res[1][1]) < 5e-6


@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("gate", [-1.4, -1.5, -2.1])
def test_small_values_under_strong_decay(cuda_device, D, gate):
    """Keys and output gradients far below one: the third plane of what the weights shrink must not vanish.  (At the limit of
    100 a weight is exp(-50) = 2e-22, and 2^-126 2^16 / 2e-22 = 4e-12.)"""
    from gla_jax_b200 import recurrent_gla
    case = list(_case(1, 192, 2, D, torch.float32, 29, 5.0))
    case[1][:] = gate * (1.0 + 0.02 * torch.rand(case[1].shape, generator=torch.Generator().manual_seed(3)))
    case[3], case[5], case[6] = case[3] * 1e-6, case[5] * 1e-8, case[6] * 1e-8
    _check(_oracle(*case), _run_gpu(recurrent_gla, cuda_device, *case), torch.float32, f"small values {D, gate}", shift=gate)
