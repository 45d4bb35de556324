"""A flow issued in one call against its evaluations called one by one, bit for
bit: one and several steps, partial tiles, every kernel width; both adjoint
modes agree; scratch that is too small is refused."""
import pytest
import torch

from meshode_gb300 import _lib as L
from meshode_gb300 import neuralode

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden", [5, 64, 100, 256])
@pytest.mark.parametrize("n, steps", [(1, 1), (127, 3), (129, 2), (1000, 5)])
def test_flow_is_its_evaluations(cuda, n, steps, hidden):
    params = neuralode.init_params(hidden, 3, cuda)
    g = torch.Generator().manual_seed(n)
    x0 = torch.rand(n, 3, generator=g).to(cuda)
    P = neuralode._Packed(params)
    s, h, x = L.stream_ptr(), 1.0 / steps, x0
    for _ in range(steps):
        acc, u = torch.empty_like(x), x
        for k, (a, w) in enumerate([(h / 2, h / 6), (h / 2, h / 3), (h, h / 3), (0.0, h / 6)]):
            nxt = torch.empty_like(x)
            L.call("mo_mlp_tc_fwd", L.ptr(u), L.ptr(x), n, L.ptr(P.buf), P.M, a, w, int(k == 0),
                   L.ptr(nxt) if k < 3 else None, L.ptr(acc), None, 0, s)
            u = nxt
        x = acc
    ps = [p.requires_grad_(True) for p in params]
    xr = x0.clone().requires_grad_(True)
    gout = torch.randn(n, 3, generator=g).to(cuda)
    grads = []
    for store in (False, True):
        y = neuralode.ODEFlow.apply(xr, steps, store, *ps)
        assert torch.equal(y.detach(), x)
        grads.append(torch.autograd.grad(y, [xr] + ps, gout))
    assert all(torch.equal(a, b) for a, b in zip(*grads))


def test_refused(cuda):
    P = neuralode._Packed(neuralode.init_params(64, 3, cuda))
    n = 40
    t = torch.zeros(10 * n, device=cuda)
    nb = int(L.lib().mo_ode_backward_floats(n, P.M, 0))
    scratch = torch.zeros(nb, device=cuda)
    grads = [L.ptr(g) for g in P.grads()]
    with pytest.raises(RuntimeError, match="too small"):
        L.call("mo_ode_flow_backward", L.ptr(t), n, 1, L.ptr(P.buf), P.M, P.m, None, None, L.ptr(t), L.ptr(scratch),
               nb - 1, L.ptr(t), L.ptr(t), *grads, L.stream_ptr())
    with pytest.raises(ZeroDivisionError):
        neuralode.ODEFlow.apply(t[:9].view(3, 3), 0, False, *neuralode.init_params(64, 3, cuda))
