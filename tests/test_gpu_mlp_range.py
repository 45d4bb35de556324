"""The tensor-core MLP at magnitudes up to FP32's: states up to 1e30 forward,
gradients up to 1e30 backward, against FP64.  Operands are scaled by powers of two
before they are split, so the error is what it is at 1 (1e-5 of a row's or an
array's scale, as in test_gpu_mlp_tc.py)."""
import pytest
import torch

from meshode_gb300 import _lib as L
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


@pytest.mark.parametrize("W", [64, 128, 256])
@pytest.mark.parametrize("gmax,hmax", [(1e38, 1e38), (1e38, 1e-3), (1e-3, 1e38), (1e-20, 1e30), (1.0, 1.0)])
def test_weight_gradient_scales(cuda, W, gmax, hmax):
    """The arrays' two scales, whose product is no float: sums that are zero stay
    zero, others are right."""
    rows, s, lib = 1024, L.stream_ptr(), L.lib()
    P = neuralode._Packed(neuralode.init_params(W, 5, cuda))
    bounds = P.buf[-32:-16].view(torch.float32)  # of |H1|, |H2|, |G2|, |G3|
    bounds.copy_(torch.tensor([hmax, hmax, gmax, gmax]))
    g = torch.Generator().manual_seed(W)
    G, H = [(torch.rand(rows * W, generator=g) * 2 - 1).to(cuda) for _ in range(2)]
    H *= hmax
    n = int(lib.mo_mlp_tc_wgrad_floats(rows, W))

    def sums(G):
        part = torch.full((n,), float("nan"), device=cuda)
        L.call("mo_mlp_tc_wgrad", L.ptr(G), L.ptr(H), rows, L.ptr(P.buf), W, 2, L.ptr(part), 1, s)
        splits = n // (W * W + (2 if W < 128 else 1) * W)
        return part[:splits * W * W].view(splits, W, W).double().sum(0)

    assert (sums(torch.zeros_like(G)) == 0).all()
    scale = gmax if gmax * hmax < 1e35 else 1e35 / hmax if 1e35 / hmax > gmax * 2.0 ** -16 else None
    if scale is not None:  # the sums are finite, and G not 17 binades below its bound
        got = sums(G * scale)
        cols = [t.double().view(rows // 128, W // 8, 128, 8).permute(0, 2, 1, 3).reshape(rows, W) for t in (G * scale, H)]
        want = cols[0].t() @ cols[1]
        assert (got - want).abs().max() <= 1e-5 * want.abs().max()
