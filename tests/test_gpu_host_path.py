"""GPU tests (pytest -m gpu) of the native host path: what it takes, refuses and saves is what the operators' Python form did."""
import pytest
import torch
import torch.autograd.forward_ad as fwAD

from oracle import gla_oracle as O

pytestmark = pytest.mark.gpu


def _call(name, dev):
    """One of the operators with small valid arguments: a callable of its differentiable arguments, and those."""
    import gla_jax_b200 as gla
    dt = torch.bfloat16
    h, g, v, k, q = [x.to(dev) for x in O.make_inputs(1, 256, 2, 128, dt, seed=31)]
    if name == "packed":
        return (lambda *a: gla.chunk_gla_packed(*a, [0, 100, 256])), [torch.cat([h, h]), g[0], v[0], k[0], q[0]]
    if name == "layer":
        torch.manual_seed(0)
        layer = gla.GLALayer(256, 2, device=dev, dtype=dt).requires_grad_(False)
        return (lambda x: layer(x)), [v.reshape(1, 256, 256)]
    return (lambda *a: gla.chunk_gla(*a, chunk_size=128)) if name == "chunk" else gla.recurrent_gla, [h, g, v, k, q]


@pytest.mark.parametrize("grad", [False, True])
@pytest.mark.parametrize("name", ["chunk", "recurrent", "packed", "layer"])
def test_forward_mode_is_refused(cuda_device, name, grad):
    fn, args = _call(name, cuda_device)
    for i in range(len(args)):
        with fwAD.dual_level():
            x = [a.detach().requires_grad_(grad) for a in args]
            x[i] = fwAD.make_dual(x[i], torch.ones_like(x[i]))
            with pytest.raises(NotImplementedError):
                fn(*x)
            with pytest.raises(NotImplementedError), torch.no_grad():
                fn(*x)
    fn(*args)


@pytest.mark.parametrize("name", ["chunk", "recurrent", "packed"])
@pytest.mark.parametrize("dtype", [torch.int32, torch.bool, torch.float16, torch.float64])
def test_gates_of_any_type(cuda_device, name, dtype):
    """log_fgate is converted to float32, whatever it is."""
    fn, args = _call(name, cuda_device)
    g = -(torch.arange(args[1].numel(), device=cuda_device).view(args[1].shape) % 2)
    args[1] = torch.zeros_like(g, dtype=dtype) if dtype == torch.bool else g.to(dtype)      # (a gate of +1 per token overflows)
    want = fn(args[0], args[1].float(), *args[2:])
    got = fn(*[a.requires_grad_(a.is_floating_point()) for a in args])
    assert all(torch.equal(a, b) for a, b in zip(want, got))
    (got[1].float().sum() + got[0].float().sum()).backward()
    assert all(a.grad is not None and a.grad.dtype == a.dtype for a in args if a.is_floating_point())


def test_packed_offsets_on_the_device_in_any_shape(cuda_device):
    import gla_jax_b200 as gla
    _, (h, *x) = _call("packed", cuda_device)
    want = gla.chunk_gla_packed(h, *x, [0, 128, 256])
    for cu in (torch.tensor([[0, 128, 256]], dtype=torch.int32), torch.tensor([[0], [128], [256]])):
        got = gla.chunk_gla_packed(h, *x, cu.to(cuda_device))
        assert all(torch.equal(a, b) for a, b in zip(want, got))


@pytest.mark.parametrize("cu,chunk", [([0, 100, 256], 256), ([0, 128, 256], 512), ([0, 1, 256], 1024)])
def test_packed_chunk_sizes_that_do_not_divide_the_sequences(cuda_device, cu, chunk):
    """Whole chunks of 128 per sequence that `chunk` does not divide, or a chunk beyond the largest, are refused."""
    import gla_jax_b200 as gla
    from gla_jax_b200 import _lib
    _, x = _call("packed", cuda_device)
    with pytest.raises(_lib.GlaError, match="unsupported configuration"):
        gla.chunk_gla_packed(*x, cu, chunk)
    assert torch.equal(gla.chunk_gla_packed(*x, [0, 130, 256], 128)[1], gla.chunk_gla_packed(*x, torch.tensor([0, 130, 256]))[1])


def test_packed_offsets_may_change_before_the_backward(cuda_device):
    import gla_jax_b200 as gla
    _, x = _call("packed", cuda_device)
    cu = torch.tensor([0, 100, 256], dtype=torch.int32)

    def grads(change):
        leaves = [a.detach().requires_grad_(True) for a in x]
        out = gla.chunk_gla_packed(*leaves, cu)[1]
        if change:
            cu[1] = 7
        return torch.autograd.grad(out.float().sum(), leaves)

    assert all(torch.equal(a, b) for a, b in zip(grads(False), grads(True)))
