"""fused_fit's one-launch run from several threads at once, on pairs of different sizes
that take the same kernel with different amounts of shared memory: no launch is
refused, and the results are those of a run alone, bit for bit."""
import ctypes
import threading

import numpy as np
import pytest
import torch

from meshode_gb300 import _lib as L
from meshode_gb300 import fused, meshgen
from meshode_gb300 import pyDeform as PD

pytestmark = pytest.mark.gpu
SIZES = (82_000, 145_000)  # 17 and 30 warps a block on 152 SMs


def _pair(nv, steps):
    V, F = meshgen.cubesphere(int(np.ceil(np.sqrt((nv - 2) / 6.0))))
    F = F[(F < nv).all(1)]
    Vd, Fd = torch.from_numpy(V[:nv].astype(np.float32)).cuda(), torch.from_numpy(F.astype(np.int32)).cuda()
    pid = PD.InitializeDeformTemplate(*[torch.from_numpy(a) for a in _target()], 0, 32)
    PD.NormalizeByTemplate(Vd, pid)
    PD.StoreRigidityInformation(Vd, Fd, pid)
    pair = fused.pair_from_template(pid, Vd + 0.01 * torch.sin(40 * Vd), steps)
    PD.ReleaseTemplate(pid)
    return pair


def _target():
    V, F = meshgen.icosphere(4)
    return meshgen.displace(V, np.random.Generator(np.random.PCG64(2))).astype(np.float32), F.astype(np.int32)


def _on_threads(pairs, work):
    errors = []
    streams = [torch.cuda.Stream() for _ in pairs]
    start = threading.Barrier(len(pairs))
    torch.cuda.synchronize()

    def body(pair, stream):
        try:
            with torch.cuda.stream(stream):
                start.wait()
                work(pair)
                stream.synchronize()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=body, args=a) for a in zip(pairs, streams)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


def test_many_launches(cuda):
    """Runs of one step of the large pair beside calls of no steps of the small one."""
    pairs = [_pair(nv, 2) for nv in SIZES[:1] * 4 + SIZES[1:]]
    running = [True]

    def work(pair):
        fn, s = L.lib().mo_fused_run, L.stream_ptr()
        row = pair.struct(0, 0, fused.tiles_for(pair.nslices))
        sync = torch.empty(2, dtype=torch.int32, device=cuda)
        large = pair.nv == SIZES[1]
        try:
            for _ in range(4000) if large else iter(lambda: running[0], False):  # the same step again and again
                L.check(fn(ctypes.byref(row), 0, int(large), None, 0, L.ptr(sync), s), "mo_fused_run")
        finally:
            running[0] = running[0] and not large

    _on_threads(pairs, work)
    assert all(torch.isfinite(p.positions()).all() for p in pairs)


def test_same_bits_as_alone(cuda):
    pairs = [_pair(nv, 200) for nv in SIZES]
    alone = [_pair(nv, 200) for nv in SIZES]
    for p in alone:
        p.run(200)
    _on_threads(pairs, lambda pair: [pair.run(20) for _ in range(10)])
    for p, q in zip(pairs, alone):
        assert torch.equal(p.positions(), q.positions())
