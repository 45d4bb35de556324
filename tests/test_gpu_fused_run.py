"""mo_fused_run (all steps of a pair in one launch) against mo_fused_step, a
launch per step: positions, moments and losses bit for bit, at one vertex, around
a slice of 32 and a tile of 8 slices, with more than the 12 records a thread
keeps, with isolated vertices, with weights, a mask and an odd number of steps,
in two calls, with one to three vertices a thread, and at the largest size that fits; one vertex more is refused."""
import numpy as np
import pytest
import torch

from meshode_gb300 import _lib as L
from meshode_gb300 import fused, meshgen
from meshode_gb300 import pyDeform as PD

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def target(cuda):
    rng = np.random.Generator(np.random.PCG64(2))
    V, F = meshgen.icosphere(4)
    return torch.from_numpy(meshgen.displace(V, rng).astype(np.float32)), torch.from_numpy(F.astype(np.int32))


def _mesh(nv, kind):
    n = max(2, int(np.ceil(np.sqrt(max(nv - 2, 6) / 6.0))))
    V, F = meshgen.cubesphere(n)
    F = F[(F < nv).all(1)]
    if kind == "star":  # vertex 0 in many faces
        extra = np.stack([np.zeros(30, np.int64), np.arange(30) % nv, (np.arange(30) + 1) % nv], 1)
        F = np.concatenate([F, extra])
    if kind == "sparse":
        F = F[::5]
    return V[:nv].astype(np.float32), F.astype(np.int32)


def _pairs(target, nv, kind, layout, **kw):
    V, F = _mesh(nv, kind)
    pid = PD.InitializeDeformTemplate(*target, 0, 32, layout=layout)
    X = torch.from_numpy(V).cuda()
    PD.NormalizeByTemplate(X, pid)
    Fd = torch.from_numpy(F).cuda()
    if kind == "cad":
        E = torch.from_numpy(meshgen.edges_from_faces(F)[::3].copy()).cuda()
        PD.StoreCadInformation(X, Fd, E, pid)
    else:
        PD.StoreRigidityInformation(X, Fd, pid)
    X = X + 0.01 * torch.sin(40 * X)
    out = [fused.pair_from_template(pid, X, 27, **kw) for _ in range(2)]
    PD.ReleaseTemplate(pid)
    return out


@pytest.mark.parametrize("nv,kind,layout,kw", [
    (1, "plain", L.MO_LAYOUT_CELL, {}), (31, "plain", L.MO_LAYOUT_LINEAR, {}), (33, "star", L.MO_LAYOUT_CELL, {}),
    (256, "plain", L.MO_LAYOUT_BRICK4, {}), (257, "sparse", L.MO_LAYOUT_CELL, {"mask_thresh": 0.5 * 0.03 ** 2}),
    (5000, "cad", L.MO_LAYOUT_CELL, {"w_edge": 0.3}), (9729, "plain", L.MO_LAYOUT_CELL, {}),
    (40_000, "star", L.MO_LAYOUT_CELL, {"w_edge": 2.0}),
    # more than a vertex a thread: two, three, with rows of more than 12 records, weights and a mask
    (77_900, "plain", L.MO_LAYOUT_CELL, {}), (90_001, "cad", L.MO_LAYOUT_LINEAR, {"w_edge": 0.3}),
    (160_003, "star", L.MO_LAYOUT_CELL, {}), (200_003, "cad", L.MO_LAYOUT_CELL, {"mask_thresh": 0.5 * 0.03 ** 2})])
def test_same_bits_as_a_launch_per_step(target, nv, kind, layout, kw):
    a, b = _pairs(target, nv, kind, layout, **kw)
    runner = fused.StepGroupRunner(a.device, 1, a.ntiles, group_steps=27, use_graph=False, weighted=a.sell_w is not None)
    runner.upload([a], [0])
    runner.run_group()
    want = runner.pair_losses(27)[:, 0]
    a.t = 27
    got = torch.cat([b.run(8, True), b.run(19, True)])
    assert b.done
    assert torch.equal(a.positions(), b.positions())
    assert torch.equal(a.m, b.m) and torch.equal(a.v, b.v)
    assert torch.allclose(got, want, rtol=1e-6, atol=0)  # the partials' sums may contract differently


def test_largest_and_refused(target):
    lib = L.lib()
    lo, hi = 1, 1 << 22
    while hi - lo > 1:
        mid = (lo + hi) // 2
        lo, hi = (mid, hi) if lib.mo_fused_run_fits(mid) else (lo, mid)
    a, b = _pairs(target, lo, "plain", L.MO_LAYOUT_CELL)
    runner = fused.StepGroupRunner(a.device, 1, a.ntiles, group_steps=27, use_graph=False)
    runner.upload([a], [0])
    runner.run_group()
    a.t = 27
    b.run(27)
    assert torch.equal(a.positions(), b.positions())
    c = _pairs(target, hi, "plain", L.MO_LAYOUT_CELL)[0]
    with pytest.raises(RuntimeError, match="do not fit"):
        c.run(1)


def test_long_rows(target):
    """Vertices with hundreds of records: the same bits as a launch per step, and
    the rule that keeps large pairs with such rows on a launch per step."""
    lib = L.lib()
    assert lib.mo_fused_run_pays(5000, 10 ** 6) == 1 and lib.mo_fused_run_pays(77_824, 10 ** 6) == 1
    assert lib.mo_fused_run_pays(77_825, 20) == 1 and lib.mo_fused_run_pays(77_825, 21) == 0
    assert lib.mo_fused_run_pays(10 ** 7, 1) == 0 and lib.mo_fused_run_pays(0, 1) == 0
    for nv, fan in ((700, 200), (90_000, 40)):
        V, F = _mesh(nv, "plain")
        k = np.arange(fan)
        F = np.concatenate([F, np.stack([np.full(fan, 5), 10 + k, 11 + k], 1)]).astype(np.int32)
        pid = PD.InitializeDeformTemplate(*target, 0, 32)
        X = torch.from_numpy(V).cuda()
        PD.NormalizeByTemplate(X, pid)
        PD.StoreRigidityInformation(X, torch.from_numpy(F).cuda(), pid)
        X = X + 0.01 * torch.sin(40 * X)
        a, b = [fused.pair_from_template(pid, X, 9) for _ in range(2)]
        assert b.run_pays() == (nv == 700)
        runner = fused.StepGroupRunner(a.device, 1, a.ntiles, group_steps=9, use_graph=False)
        runner.upload([a], [0])
        runner.run_group()
        a.t = 9
        b.run(9)
        assert torch.equal(a.positions(), b.positions())
        PD.ReleaseTemplate(pid)
