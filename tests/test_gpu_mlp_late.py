"""A wait of the MLP kernels that ran out leaves NaN for the scales of the packed
weights; whatever a backward pass makes after it is NaN, parameter gradients
included, and never a plausible number.  The scales are set here as a kernel sets
them."""
import pytest
import torch

from meshode_gb300 import _lib as L
from meshode_gb300 import neuralode

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [300, 153 * 128 + 7])
@pytest.mark.parametrize("m", [64, 128, 256])
@pytest.mark.parametrize("stored", [False, True])
@pytest.mark.parametrize("late", [0, 1])
def test_scales(cuda, n, m, stored, late):
    steps, s, lib = 2, L.stream_ptr(), L.lib()
    g = torch.Generator().manual_seed(n)
    x0, aout = torch.rand(n, 3, generator=g).to(cuda), torch.randn(n, 3, generator=g).to(cuda)
    P = neuralode._Packed(neuralode.init_params(m, 7, cuda))
    ckpt, out = torch.zeros(steps, n, 3, device=cuda), torch.zeros(n, 3, device=cuda)
    u = torch.zeros(steps if stored else 1, 3, n, 3, device=cuda)
    act = torch.zeros(steps, int(lib.mo_ode_act_floats(n, P.M)), device=cuda) if stored else None
    L.call("mo_ode_flow", L.ptr(x0), n, steps, L.ptr(P.buf), P.M, L.ptr(ckpt), L.ptr(act), L.ptr(u), L.ptr(out), s)
    scales = P.buf[16 * P.M ** 2 + 36 * P.M:][:8].view(torch.float32)  # behind the images and vectors
    assert torch.isfinite(out).all() and torch.isfinite(scales).all()
    assert torch.equal(scales, torch.exp2(torch.log2(scales).round())) and (scales > 0).all()  # powers of two
    if late:
        scales.fill_(float("nan"))
    nb = int(lib.mo_ode_backward_floats(n, P.M, int(stored)))
    scratch, dx, grads = torch.zeros(nb, device=cuda), torch.zeros(2, n, 3, device=cuda), P.grads()
    L.call("mo_ode_flow_backward", L.ptr(ckpt), n, steps, L.ptr(P.buf), P.M, m, L.ptr(act), L.ptr(u), L.ptr(aout),
           L.ptr(scratch), nb, L.ptr(dx[0]), L.ptr(dx[1]), *[L.ptr(t) for t in grads], s)
    for name, t in zip(("x0",) + neuralode.PARAM_NAMES, [dx[0]] + grads):
        assert torch.isnan(t).all() if late else torch.isfinite(t).all(), name
