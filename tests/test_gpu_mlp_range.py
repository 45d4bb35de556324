"""The tensor-core MLP at magnitudes up to FP32's: states up to 1e30 forward,
gradients up to 1e30 backward, against FP64.  Operands are scaled by powers of two
before they are split, so the error is what it is at 1 (1e-5 of a row's or an
array's scale, as in test_gpu_mlp_tc.py)."""
import pytest
import torch

from meshode_gb300 import neuralode

pytestmark = pytest.mark.gpu


def _f64(p):
    q = [t.double() for t in p]

    def f(u):
        for k in (0, 2, 4):
            z = u @ q[k].t() + q[k + 1]
            u = torch.clamp(z, min=0) + torch.log1p(torch.exp(-z.abs()))
        return u @ q[6].t() + q[7]

    return q, f


def _rk4(f, x):
    k1 = f(x)
    k2 = f(x + k1 / 2)
    k3 = f(x + k2 / 2)
    return x + (k1 + 2 * k2 + 2 * k3 + f(x + k3)) / 6


@pytest.mark.parametrize("m", [64, 128, 256])
def test_large_states(cuda, m):
    p = neuralode.init_params(m, 5, cuda)
    g = torch.Generator().manual_seed(m)
    x0 = (torch.rand(310, 3, generator=g) * 10.0 ** (torch.arange(310) % 31)[:, None]).to(cuda)
    got = neuralode.ODEFlow.apply(x0, 1, False, *p).double()
    want = _rk4(_f64(p)[1], x0.double())
    scale = want.abs().max(1).values
    assert torch.isfinite(want.float()).all()
    assert ((got - want).abs().max(1).values <= 1e-5 * scale).all()


@pytest.mark.parametrize("m", [64, 128, 256])
@pytest.mark.parametrize("top", [10, 20, 31])
def test_large_gradients(cuda, m, top):
    p = [t.requires_grad_(True) for t in neuralode.init_params(m, 5, cuda)]
    g = torch.Generator().manual_seed(m)
    x0 = torch.rand(310, 3, generator=g).to(cuda).requires_grad_(True)
    gout = (torch.randn(310, 3, generator=g) * 10.0 ** (torch.arange(310) % top)[:, None]).to(cuda)
    got = torch.autograd.grad(neuralode.ODEFlow.apply(x0, 1, False, *p), [x0] + p, gout)
    q, f = _f64([t.detach() for t in p])
    q = [t.requires_grad_(True) for t in q]

    def f64(u):
        for k in (0, 2, 4):
            u = torch.nn.functional.softplus(u @ q[k].t() + q[k + 1], threshold=60)
        return u @ q[6].t() + q[7]

    x = x0.detach().double().requires_grad_(True)
    want = torch.autograd.grad(_rk4(f64, x), [x] + q, gout.double())
    row = want[0].abs().max(1).values
    assert ((got[0].double() - want[0]).abs().max(1).values <= 1e-5 * row).all()
    for a, b in zip(got[1:], want[1:]):
        assert (a.double() - b).abs().max() <= 1e-5 * b.abs().max()
