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
