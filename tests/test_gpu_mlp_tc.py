"""The tensor-core MLP kernels (mo_mlp_tc_*) against the same model in FP64, at
the sizes where they can go wrong: one row, around a 128-row tile, more tiles
than SMs, hidden widths at and beside the padded widths 64, 128 and 256, rows
whose gradients differ by 20 orders of magnitude, activations in the thousands,
and a row of NaN.

Tolerance: every operand carries 22 bits and every sum of at most 256 products
FP32 accuracy, so a layer is within a few 1e-7 of its scale and a gradient,
through six layers, within 1e-5 of its own (the bound of the velocity-field
configuration)."""
import pytest
import torch

from meshode_gb300 import neuralode

pytestmark = pytest.mark.gpu


def _params(m, seed, gain=1.0):
    g = torch.Generator().manual_seed(seed)
    shapes = [(m, 3), (m,), (m, m), (m,), (m, m), (m,), (3, m), (3,)]
    out = []
    for k, s in enumerate(shapes):
        a = (6.0 / sum(s)) ** 0.5 if len(s) == 2 else 0.1
        out.append(((torch.rand(s, generator=g) * 2 - 1) * a * (gain if k == 2 else 1.0)).cuda())
    return out


def _flow64(x, p, steps):
    def f(u):
        for k in (0, 2, 4):
            u = torch.nn.functional.softplus(u @ p[k].t() + p[k + 1], threshold=60)
        return u @ p[6].t() + p[7]
    h = 1.0 / steps
    for _ in range(steps):
        k1 = f(x)
        k2 = f(x + h / 2 * k1)
        k3 = f(x + h / 2 * k2)
        k4 = f(x + h * k3)
        x = x + h / 6 * (k1 + 2 * k2 + 2 * k3 + k4)
    return x


def _both(x0, p, gout, steps, store):
    x = x0.clone().requires_grad_(True)
    q = [t.clone().requires_grad_(True) for t in p]
    y = neuralode.ODEFlow.apply(x, steps, store, *q)
    got = [y.detach()] + list(torch.autograd.grad(y, [x] + q, gout))
    x = x0.double().requires_grad_(True)
    q = [t.double().requires_grad_(True) for t in p]
    y = _flow64(x, q, steps)
    ref = [y.detach()] + list(torch.autograd.grad(y, [x] + q, gout.double()))
    return got, ref


def _close(got, ref, names):
    for name, a, b in zip(names, got, ref):
        assert a.shape == b.shape
        err, scale = (a.double() - b).abs().max().item(), b.abs().max().item()
        assert err <= 1e-5 * scale, (name, err, scale)


NAMES = ("x", "x0") + neuralode.PARAM_NAMES


@pytest.mark.parametrize("n,m", [(1, 1), (127, 16), (128, 64), (129, 65), (300, 128), (257, 129), (1, 256), (500, 200),
                                 (19457, 64), (19457, 256)])
def test_sizes(cuda, n, m):
    g = torch.Generator().manual_seed(n + m)
    x0 = torch.rand(n, 3, generator=g).cuda()
    gout = torch.randn(n, 3, generator=g).cuda()
    for store in (False, True):
        got, ref = _both(x0, _params(m, 3), gout, 2, store)
        _close(got, ref, NAMES)


@pytest.mark.parametrize("m", [64, 128, 256])
def test_ranges(cuda, m):
    g = torch.Generator().manual_seed(m)
    x0 = torch.rand(260, 3, generator=g).cuda()
    gout = torch.randn(260, 3, generator=g).cuda() * (10.0 ** -(torch.arange(260).float() % 21)).cuda()[:, None]
    got, ref = _both(x0, _params(m, 5), gout, 1, False)
    _close(got, ref, NAMES)
    # every row's own gradient, however small
    err = (got[1].double() - ref[1]).abs().max(1).values / ref[1].abs().max(1).values
    assert err.max().item() <= 1e-5
    # activations in the thousands
    got, ref = _both(x0 * 100.0, _params(m, 6, gain=20.0), gout, 1, False)
    _close(got, ref, NAMES)


def test_nan_stays_in_its_row(cuda):
    x0 = torch.rand(200, 3, generator=torch.Generator().manual_seed(1)).cuda()
    p = _params(128, 7)
    clean = neuralode.ODEFlow.apply(x0, 2, False, *p)
    x0[17, 1] = float("nan")
    y = neuralode.ODEFlow.apply(x0, 2, False, *p)
    bad = torch.isnan(y).any(1)
    assert bad[17] and bad.sum() == 1
    keep = ~bad
    assert torch.equal(y[keep], clean[keep])
