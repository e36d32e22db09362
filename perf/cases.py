"""The calls that users of this framework make, as sizes, inputs and one pass each.

Every case names a public entry point of ``gla_jax_b200`` and the sizes it is called with.  Inputs follow the
distributions of the reference harness (q, k, v, states ~ N(0,1); log_fgate = log_sigmoid(shift + N(0,1)) in float32,
shift 5 for the usual soft gates and 0 for sharp ones); cotangents are N(0,1).
"""
import math

import torch
import torch.nn.functional as F

import gla_jax_b200 as gla
from gla_jax_b200.ops import cumsum_recursive, rnn_recursive

_DTYPES = {"bf16": torch.bfloat16, "f32": torch.float32}
_BYTES = {"bf16": 2, "f32": 4}


def listed():
    return [
        # README shape of the reference: an ordinary training batch of one layer's attention
        dict(name="train_readme", op="chunk", dtype="bf16", B=4, T=4096, H=6, D=128, C=128, shift=5.0, grad=True),
        # one long document per GPU: few heads, a very long time axis; the largest call
        dict(name="train_long_context", op="chunk", dtype="bf16", B=1, T=131072, H=8, D=128, C=128, shift=5.0, grad=True),
        # wide heads with strong decay: the stability stress configuration, one GPU's share of it
        dict(name="train_wide_sharp", op="chunk", dtype="bf16", B=2, T=16384, H=8, D=256, C=256, shift=0.0, grad=True),
        # the usual head size 64 with the usual chunk of 64; an odd number of chunks
        dict(name="train_narrow", op="chunk", dtype="bf16", B=8, T=2112, H=12, D=64, C=64, shift=5.0, grad=True),
        # a correctness run in full precision on a short sequence: small enough that latency and launches count
        dict(name="check_f32", op="chunk", dtype="f32", B=1, T=256, H=2, D=64, C=64, shift=5.0, grad=True),
        # serving: the prompt of one request, forward only
        dict(name="prefill_prompt", op="chunk", dtype="bf16", B=1, T=1152, H=16, D=128, C=128, shift=5.0, grad=False),
        # training with the exact recurrence (no chunk size, any length), on the README shape
        dict(name="train_recurrent", op="recurrent", dtype="bf16", B=4, T=4096, H=6, D=128, shift=5.0, grad=True),
        # serving: one token for a batch of requests, states resident
        dict(name="decode_batch", op="decode", dtype="bf16", B=32, H=16, D=128, shift=5.0),
        # training on documents of different lengths packed on one time axis
        dict(name="train_packed", op="packed", dtype="bf16", T=8192, nseq=11, H=8, D=128, shift=5.0, grad=True),
        # a whole layer of a small model in training: projections, gate, attention, norm, output gate
        dict(name="train_layer", op="layer", dtype="bf16", B=4, T=4096, H=6, D=128, C=128),
        # cumulative log decay over whole sequences
        dict(name="cumsum_gates", op="cumsum", dtype="f32", N=24, T=4096, D=136, init=True, reverse=False),
        # linear-RNN scan of per-chunk states: one state per chunk and head
        dict(name="scan_states", op="rnn", dtype="f32", N=24, T=33, K=128, V=128, init=True, reverse=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges above: token count, heads, head size, gates and direction vary together, and the
    number of (token, head) pairs stays inside what the largest listed case of the same kind has."""
    op = rng.choice(["chunk"] * 5 + ["recurrent", "recurrent", "decode", "decode", "packed", "layer", "cumsum", "rnn"])
    shift = rng.choice([5.0, 5.0, 5.0, 2.0, 0.0])
    if op == "chunk":
        if rng.random() < 0.2:          # full precision: short sequences, any head and chunk size
            D, C = rng.choice([32, 64, 64, 128]), rng.choice([32, 64, 128])
            H, B = rng.randint(1, 6), rng.randint(1, 3)
            n = _log_int(rng, 1, max(1, 2048 // C))
            return dict(op=op, dtype="f32", B=B, T=n * C, H=H, D=D, C=C, shift=shift, grad=rng.random() < 0.7)
        D = rng.choice([64, 128, 128, 128, 256])
        C = {64: 64, 128: rng.choice([64, 128, 128, 256]), 256: rng.choice([128, 256])}[D]
        H = rng.randint(1, 24 if D < 256 else 8)
        B = _log_int(rng, 1, 16)
        # token-heads of the pass: 1 K (a short prompt) to 512 K (a training batch); narrow heads and chunks less
        most = {64: 192 << 10, 128: (512 << 10) if C >= 128 else (128 << 10), 256: 128 << 10}[D]
        T = _log_int(rng, 1 << 10, most) // (B * H)
        return dict(op=op, dtype="bf16", B=B, T=max(1, T // C) * C, H=H, D=D, C=C, shift=shift, grad=rng.random() < 0.7)
    if op == "recurrent":
        D, H, B = rng.choice([64, 128, 128]), rng.randint(1, 12), _log_int(rng, 1, 8)
        T = max(1, min(4096, _log_int(rng, 128, 96 << 10) // (B * H)))
        return dict(op=op, dtype=rng.choice(["bf16", "bf16", "f32"]), B=B, T=T, H=H, D=D, shift=shift, grad=rng.random() < 0.6)
    if op == "decode":
        return dict(op=op, dtype=rng.choice(["bf16", "bf16", "f32"]), B=_log_int(rng, 1, 128), H=rng.randint(2, 24),
                    D=rng.choice([64, 128, 128, 256]), shift=shift)
    if op == "packed":
        nseq = rng.randint(1, 24)
        T = max(nseq * 8, _log_int(rng, 512, 32768))
        return dict(op=op, dtype="bf16", T=T, nseq=nseq, H=rng.randint(2, 16), D=128, shift=shift, grad=rng.random() < 0.8)
    if op == "layer":
        return dict(op=op, dtype="bf16", B=_log_int(rng, 1, 8), T=128 * rng.randint(1, 24), H=rng.randint(4, 12), D=128, C=128)
    if op == "cumsum":
        D = rng.choice([rng.randint(16, 127), 4 * rng.randint(32, 256), rng.randint(128, 768)])
        T, most = _log_int(rng, 64, 16384), 48 << 20
        N = max(1, min(512, _log_int(rng, 1 << 18, most) // (T * D)))
        return dict(op=op, dtype=rng.choice(["f32", "f32", "bf16"]), N=N, T=T, D=D, init=rng.random() < 0.5,
                    reverse=rng.random() < 0.5)
    K, V = rng.choice([64, 128]), rng.choice([64, 128])
    T = _log_int(rng, 8, 2048)
    N = max(1, min(96, _log_int(rng, 1 << 18, 24 << 20) // (T * K * V)))
    return dict(op="rnn", dtype="f32", N=N, T=T, K=K, V=V, init=rng.random() < 0.5, reverse=rng.random() < 0.5)


class _Maker:
    """Seeded normal tensors on the GPU, a new one with every call."""

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda").manual_seed(seed)

    def __call__(self, shape, dtype=torch.float32, scale=1.0):
        x = torch.randn(shape, generator=self.gen, device="cuda")
        return (x if scale == 1.0 else x * scale).to(dtype)

    def gate(self, shape, shift):
        return F.logsigmoid(self(shape).add_(shift))


def _lengths(T, nseq, seed):
    """nseq document lengths that sum to T, none of them round."""
    gen = torch.Generator().manual_seed(seed)
    w = 0.25 + torch.rand(nseq, generator=gen, dtype=torch.float64)
    cu = [0] + [int(x) for x in torch.round(torch.cumsum(w, 0) / w.sum() * T)]
    cu[-1] = T
    return cu


def prepare(case, seed):
    new, op, dt = _Maker(seed), case["op"], _DTYPES[case["dtype"]]
    st = dict(case=case)
    if op in ("chunk", "recurrent", "packed"):
        H, D = case["H"], case["D"]
        if op == "packed":
            lead, tok = (case["nseq"],), (case["T"], H, D)
            st["cu"] = _lengths(case["T"], case["nseq"], seed)
        else:
            lead, tok = (case["B"],), (case["B"], case["T"], H, D)
        state = lead + (H, D, D)
        st["x"] = [new(state, dt), new.gate(tok, case["shift"]), new(tok, dt), new(tok, dt), new(tok, dt)]
        if case["grad"]:
            for x in st["x"]:
                x.requires_grad_(True)
            st["cotangents"] = [new(state, dt), new(tok, dt)]
    elif op == "decode":
        tok = (case["B"], case["H"], case["D"])
        st["state"] = new(tok + (case["D"],))
        st["x"] = [new.gate(tok, case["shift"]), new(tok, dt), new(tok, dt), new(tok, dt)]
    elif op == "layer":
        H, D = case["H"], case["D"]
        with torch.random.fork_rng(devices=[torch.cuda.current_device()]):
            torch.manual_seed(seed)
            st["layer"] = gla.GLALayer(H * D, H, chunk_size=case["C"], device="cuda", dtype=dt)
        tok, state = (case["B"], case["T"], H * D), (case["B"], H, D, D)
        st["x"] = [new(tok, dt).requires_grad_(True), new(state, dt).requires_grad_(True)]
        st["cotangents"] = [new(tok, dt), new(state, dt)]
    elif op == "cumsum":
        st["x"] = new((case["N"], case["T"], case["D"]), dt)
        st["init"] = new((case["N"], case["D"]), dt) if case["init"] else None
    else:
        N, T, K, V = case["N"], case["T"], case["K"], case["V"]
        # decay of a whole chunk under soft gates
        st["x"] = [new((N, T, K)).abs_().neg_(), new((N, T, K, V), dt)]
        st["init"] = [new((N, K)).abs_().neg_(), new((N, K, V), dt)] if case["init"] else [None, None]
    return st


def run(st):
    case = st["case"]
    op = case["op"]
    if op == "decode":
        return gla.decode_step(st["state"], *st["x"]), st["state"]
    if op == "cumsum":
        return cumsum_recursive(st["x"], axis=1, init=st["init"], reverse=case["reverse"])
    if op == "rnn":
        return rnn_recursive(*st["x"], *st["init"], reverse=case["reverse"])
    leaves = st["x"]
    if op == "chunk":
        hidden, out = gla.chunk_gla(*leaves, chunk_size=case["C"])
    elif op == "recurrent":
        hidden, out = gla.recurrent_gla(*leaves)
    elif op == "packed":
        hidden, out = gla.chunk_gla_packed(*leaves, st["cu"])
    else:
        out, hidden = st["layer"](*leaves)
        leaves = leaves + list(st["layer"].parameters())
        return out, hidden, torch.autograd.grad([out, hidden], leaves, st["cotangents"])
    if not case["grad"]:
        return hidden, out
    return hidden, out, torch.autograd.grad([hidden, out], leaves, st["cotangents"])


def work(case):
    op, e = case["op"], _BYTES[case["dtype"]]
    if op == "decode":
        s = case["B"] * case["H"] * case["D"]
        return {"bytes": s * (4 + 4 * e) + 8.0 * s * case["D"], "flops": 5.0 * s * case["D"]}
    if op == "cumsum":
        n = case["N"] * case["T"] * case["D"]
        return {"bytes": 2.0 * e * n, "flops": 1.0 * n}
    if op == "rnn":
        n = case["N"] * case["T"] * case["K"]
        return {"bytes": 2.0 * n * (4 + e * case["V"]), "flops": 2.0 * n * case["V"]}
    D = case["D"]
    B = case.get("B", 1)
    th = 1.0 * B * case["T"] * case["H"]                              # token-heads
    states = 1.0 * case.get("nseq", B) * case["H"] * D * D
    if op == "layer":
        dm = case["H"] * D
        # five projections of d_model x d_model and the low-rank gate, forward and twice that backward
        rows = B * case["T"]
        gemm = 3 * 2.0 * rows * (5 * dm * dm + 2 * 16 * dm)
        # x, its cotangent, y and dx; every weight read and its gradient written; states in and out, both directions
        return {"bytes": e * (4.0 * rows * dm + 2.0 * (5 * dm * dm + 32 * dm) + 4 * states),
                "flops": gemm + th * (6 * case["C"] * D + 12 * D * D)}
    C = 128 if op == "packed" else case.get("C", 0)
    # forward: q, k, v, gate in, out; backward: those and the output's cotangent in, four gradients out
    per = (4 * e + 4) * D + ((7 * e + 8) * D if case["grad"] else 0)
    # contractions of the chunked form; of the plain recurrence where there is no chunk
    if op == "recurrent":
        flops = (5 if not case["grad"] else 17) * D * D
    else:
        flops = (2 * C * D + 4 * D * D) if not case["grad"] else (6 * C * D + 12 * D * D)
    return {"bytes": th * per + states * e * (4 if case["grad"] else 2), "flops": th * flops}


def tolerance(case):
    # bf16: operands of the contractions are rounded to 8 bits.  float32: sums over a chunk and a head, and the gate's
    # gradient is a running sum over the sequence of terms that cancel.
    return {"rel": 1e-2} if case["dtype"] == "bf16" else {"rel": 1e-5 if case["op"] in ("cumsum", "rnn", "decode") else 3e-5}
