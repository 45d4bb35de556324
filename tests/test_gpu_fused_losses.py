"""A long fit with its losses: the partial sums that it holds do not grow with the
number of steps, and losses and positions are those of shorter runs."""
import numpy as np
import pytest
import torch

from meshode_gb300 import fused, meshgen
from meshode_gb300 import pyDeform as PD

pytestmark = pytest.mark.gpu


def _pair(steps):
    V, F = meshgen.icosphere(4)
    tar = torch.from_numpy(meshgen.displace(V, np.random.Generator(np.random.PCG64(2))).astype(np.float32))
    pid = PD.InitializeDeformTemplate(tar, torch.from_numpy(F.astype(np.int32)), 0, 32)
    Vs, Fs = meshgen.cubesphere(50)
    X = torch.from_numpy(Vs.astype(np.float32)).cuda()
    PD.NormalizeByTemplate(X, pid)
    PD.StoreRigidityInformation(X, torch.from_numpy(Fs.astype(np.int32)).cuda(), pid)
    pair = fused.pair_from_template(pid, X, steps)
    PD.ReleaseTemplate(pid)
    return pair


def test_memory_and_losses(cuda):
    steps = 20_000
    a, b = _pair(steps), _pair(steps)
    per_step = 4 * fused.tiles_for(a.nslices) * fused.SLICES_PER_TILE
    torch.cuda.synchronize()
    base = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    losses = a.run(steps, True)
    torch.cuda.synchronize()
    peak = torch.cuda.max_memory_allocated() - base
    assert peak <= 5000 * per_step + 8 * steps + (1 << 20), (peak, per_step)
    parts = []
    for n in (1, 999, 4000, 5000, 10_000):
        parts.append(b.run(n, True))
    assert torch.equal(torch.cat(parts), losses) and losses.shape == (steps,)
    assert torch.equal(a.positions(), b.positions()) and a.done and b.done
