"""A flow in one launch, and a step's four vector-Jacobian products in one,
against a launch each, bit for bit: one tile a block with a ragged last one,
blocks of one and two tiles, of two, of two and three, of three and four, and
more steps than one launch takes."""
import pytest
import torch

from meshode_gb300 import _lib as L
from meshode_gb300 import neuralode

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tiles,extra,steps", [(0, 1, 300), (1, 0, 3), (21, -72, 3), (152, 0, 2), (152, 1, 2), (303, 0, 2),
                                               (304, 0, 2), (304, 5, 2), (456, -1, 2), (470, 3, 2), (1400, 9, 3)])
@pytest.mark.parametrize("m", [64, 128, 256])
@pytest.mark.parametrize("stored", [False, True])
def test_one_launch_gives_the_same(cuda, tiles, extra, steps, m, stored):
    n = tiles * 128 + extra
    params = neuralode.init_params(m, 7, cuda)
    params[6].mul_(20.0)
    gen = torch.Generator(device="cpu").manual_seed(n + m)
    x0 = torch.rand(n, 3, generator=gen).to(cuda)
    s = L.stream_ptr()
    rows, W = int(L.lib().mo_mlp_tc_rows(n)), m

    def outputs():
        return (torch.full((steps, n, 3), -1.0, device=cuda),
                torch.full((steps if stored else 1, 3, n, 3), -1.0, device=cuda),
                torch.full((steps, 3, 4, rows * W), -1.0, device=cuda) if stored else None,
                torch.full((n, 3), -1.0, device=cuda))

    P = neuralode._Packed(params)
    ckpt, u, act, out = outputs()
    L.call("mo_ode_flow", L.ptr(x0), n, steps, L.ptr(P.buf), W, L.ptr(ckpt), L.ptr(act), L.ptr(u), L.ptr(out), s)
    Q = neuralode._Packed(params)
    rc, ru, ract, rout = outputs()
    rc[0] = x0
    h = 1.0 / steps
    for k in range(steps):
        nxt = rc[k + 1] if k + 1 < steps else rout
        us = ru[k if stored else 0]
        for e in range(4):
            L.call("mo_mlp_tc_fwd", L.ptr(us[e - 1] if e else rc[k]), L.ptr(rc[k]), n, L.ptr(Q.buf), W,
                   (h / 2, h / 2, h, 0.0)[e], (h / 6, h / 3, h / 3, h / 6)[e], int(e == 0),
                   L.ptr(us[e]) if e < 3 else None, L.ptr(nxt), L.ptr(ract[k, 0, e]) if stored else None,
                   4 * rows * W if stored else 0, s)
    assert torch.isfinite(out).all()
    assert torch.equal(out, rout) and torch.equal(ckpt, rc) and torch.equal(u, ru)
    assert not stored or torch.equal(act, ract)
    assert torch.equal(P.buf, Q.buf)  # the bounds of the activations, kept behind the parameters


@pytest.mark.parametrize("n", [1, 128, 2563, 152 * 128 - 1, 153 * 128 + 7, 304 * 128 + 1, 460 * 128])
@pytest.mark.parametrize("m", [64, 128, 256])
def test_a_steps_products_give_the_same(cuda, n, m):
    steps, W, s, lib = 2, m, L.stream_ptr(), L.lib()
    params = neuralode.init_params(m, 7, cuda)
    params[6].mul_(20.0)
    gen = torch.Generator(device="cpu").manual_seed(n + m)
    x0, aout = torch.rand(n, 3, generator=gen).to(cuda), torch.randn(n, 3, generator=gen).to(cuda)
    rows = int(lib.mo_mlp_tc_rows(n))
    size, h = rows * W, 1.0 / steps

    def floats(*shape):
        return torch.zeros(*shape, device=cuda)

    P = neuralode._Packed(params)
    ckpt, u, act, out = floats(steps, n, 3), floats(steps, 3, n, 3), floats(steps, 3, 4, size), floats(n, 3)
    L.call("mo_ode_flow", L.ptr(x0), n, steps, L.ptr(P.buf), W, L.ptr(ckpt), L.ptr(act), L.ptr(u), L.ptr(out), s)
    buf = P.buf.clone()  # the backward pass adds its bounds
    nb = int(lib.mo_ode_backward_floats(n, W, 1))
    scratch, dx, grads = floats(nb), floats(2, n, 3), P.grads()
    L.call("mo_ode_flow_backward", L.ptr(ckpt), n, steps, L.ptr(P.buf), W, m, L.ptr(act), L.ptr(u), L.ptr(aout),
           L.ptr(scratch), nb, L.ptr(dx[0]), L.ptr(dx[1]), *[L.ptr(g) for g in grads], s)
    partial = floats(int(lib.mo_mlp_tc_partial_floats(n, W)))
    wpart = [floats(int(lib.mo_mlp_tc_wgrad_floats(4 * rows, W))) for _ in range(2)]
    gz, gu, a = floats(2, 4, size), floats(2, n, 3), aout
    for k in reversed(range(steps)):
        d = floats(n, 3)
        for e in (3, 2, 1, 0):
            L.call("mo_mlp_tc_bwd", L.ptr(a), (h / 6, h / 3, h / 3, h / 6)[e], L.ptr(gu[e & 1]) if e < 3 else None,
                   (h / 2, h / 2, h, 0.0)[e], L.ptr(u[k, e - 1] if e else ckpt[k]), n, L.ptr(buf), W,
                   L.ptr(act[k, 0, e]), 4 * size, L.ptr(gz[0, e]), L.ptr(gz[1, e]), L.ptr(a if e == 3 else d),
                   L.ptr(d), L.ptr(gu[1 - (e & 1)]), L.ptr(partial), int(k == steps - 1 and e == 3), s)
        for l in range(2):
            L.call("mo_mlp_tc_wgrad", L.ptr(gz[l]), L.ptr(act[k, l]), 4 * rows, L.ptr(buf), W, 2 + l,
                   L.ptr(wpart[l]), int(k == steps - 1), s)
        a = d
    ref = P.grads()
    L.call("mo_mlp_tc_reduce", L.ptr(partial), n, L.ptr(wpart[0]), L.ptr(wpart[1]), 4 * rows, W, m,
           *[L.ptr(g) for g in ref], s)
    assert torch.isfinite(a).all() and torch.equal(dx[0], a) and torch.equal(P.buf, buf)
    assert all(torch.equal(g, q) for g, q in zip(grads, ref))
