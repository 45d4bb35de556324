"""SolveLinear's one-launch solver where its work split changes: one block, a
vertex more than one block takes, blocks with more vertices than threads (state
in memory instead of registers), cells so large that a block sums one, cells of
one vertex, a vertex without edges.  Against the oracle's direct solve, within
1e-6 of the bounding-box diagonal (the result is float32, both solvers are
double), as in test_gpu_linear.py."""
import numpy as np
import pytest
import torch

from meshode_gb300 import meshgen
from meshode_gb300 import pyDeform as PD

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,cut,ncells", [(2, 3, 2), (3, 0, 56), (7, 1, 5), (21, 0, 2), (21, 0, 2000), (95, 5, 900)])
def test_against_direct_solve(cuda, orc, n, cut, ncells):
    rng = np.random.Generator(np.random.PCG64(n))
    V, F = meshgen.cubesphere(n)
    V = (0.4 * V + 0.5).astype(np.float32)
    F = F[(F < len(V) - cut).all(1)].astype(np.int32)  # the cut vertices keep no faces
    ref = (np.arange(len(V)) * ncells // len(V)).astype(np.int32)
    ncells = int(ref.max()) + 1
    G = np.zeros((ncells, 3))
    np.add.at(G, ref, V)
    G /= np.bincount(ref, minlength=ncells)[:, None]
    G = ((G - 0.5) * 1.1 + 0.5 + 0.005 * rng.standard_normal(G.shape)).astype(np.float32)
    E = np.stack([np.arange(8) % len(V), (np.arange(8) + 3) % len(V)], 1).astype(np.int32)
    want = orc.solve_linear(V, F, E, ref, G, 1.0, 0)
    X = torch.from_numpy(V.copy()).cuda()
    it, res = PD.SolveLinear(X, torch.from_numpy(F), torch.from_numpy(E), torch.from_numpy(ref), torch.from_numpy(G),
                             1.0, 0)
    assert res <= 1e-13 and it > 0
    diag = float(np.linalg.norm(V.max(0) - V.min(0)))
    assert np.abs(X.cpu().numpy() - want).max() <= 1e-6 * diag


def test_a_vertex_with_a_thousand_neighbours(cuda, orc):
    """A block's rows that do not fit its shared memory."""
    rng = np.random.Generator(np.random.PCG64(5))
    n = 1500
    V = rng.uniform(0.2, 0.8, (n, 3)).astype(np.float32)
    k = np.arange(1, 1200)
    F = np.stack([np.zeros_like(k), k, k + 1], 1).astype(np.int32)
    ref = (np.arange(n) // 25).astype(np.int32)
    G = np.stack([V[ref == g].mean(0) for g in range(ref.max() + 1)]).astype(np.float32)
    E = np.stack([np.arange(8), np.arange(8) + 1201], 1).astype(np.int32)
    want = orc.solve_linear(V, F, E, ref, G, 1.0, 0)
    X = torch.from_numpy(V.copy()).cuda()
    it, res = PD.SolveLinear(X, torch.from_numpy(F), torch.from_numpy(E), torch.from_numpy(ref), torch.from_numpy(G),
                             1.0, 0)
    assert res <= 1e-13 and it > 0
    assert np.abs(X.cpu().numpy() - want).max() <= 1e-6 * float(np.linalg.norm(V.max(0) - V.min(0)))
