"""A flow in one launch against an evaluation a launch, bit for bit: one tile a
block with a ragged last one, blocks of one and two tiles (an evaluation a
launch), of two, of two and three, of three and four, and more steps than one
launch takes."""
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
