"""SolveLinear with more cells than the solver has warps: a cell a vertex, cells of
two, cells of very different sizes, empty cells, against the oracle's direct solve
(1e-6 of the box's diagonal, as in test_gpu_linear.py); and the time of an iteration
with a cell a vertex, beside that with cells of 50."""
import time

import numpy as np
import pytest
import torch

from meshode_gb300 import meshgen
from meshode_gb300 import pyDeform as PD

pytestmark = pytest.mark.gpu
E0 = torch.zeros(0, 2, dtype=torch.int32)


def _system(n, kind):
    V, F = meshgen.cubesphere(n)
    V = (0.4 * V + 0.5).astype(np.float32)
    k = len(V)
    if kind == "one":
        ref = np.arange(k)
    elif kind == "two":
        ref = np.arange(k) // 2
    elif kind == "mixed":  # one of a third of the vertices, some of nine, the others of one
        ref = np.where(np.arange(k) < k // 3, 0, np.arange(k) - k // 3 + 1)
        ref = np.where(np.arange(k) > k // 2, ref[k // 2] + 1 + (np.arange(k) - k // 2) // 9, ref)
    else:
        ref = np.arange(k) // 50
    ref = ref.astype(np.int32)
    G = np.zeros((ref.max() + 1, 3))
    np.add.at(G, ref, V)
    G = (G / np.maximum(np.bincount(ref), 1)[:, None] * 1.03).astype(np.float32)
    if kind == "two":  # cells without a vertex
        G = np.concatenate([G, G])
    return [torch.from_numpy(np.ascontiguousarray(a)) for a in (V, F.astype(np.int32), ref, G)]


@pytest.mark.parametrize("kind", ["one", "two", "mixed"])
@pytest.mark.parametrize("n", [15, 36])
def test_against_direct_solve(cuda, orc, kind, n):
    V, F, ref, G = _system(n, kind)
    want = orc.solve_linear(V.numpy(), F.numpy(), E0.numpy(), ref.numpy(), G.numpy(), 1.0, 0)
    X = V.cuda()
    _, res = PD.SolveLinear(X, F, E0, ref, G, 1.0, 0)
    assert res <= 1e-13
    assert np.abs(X.cpu().numpy() - want).max() <= 1e-6 * float(np.linalg.norm((V.max(0).values - V.min(0).values).numpy()))


def test_time_of_an_iteration(cuda):
    def iteration(kind):
        V, F, ref, G = [t.cuda() for t in _system(182, kind)]
        best = []
        for _ in range(4):
            t = []
            for its in (32, 160):  # more iterations, the same preparation
                X = V.clone()
                torch.cuda.synchronize()
                a = time.perf_counter()
                try:
                    PD.SolveLinear(X, F, E0.cuda(), ref, G, 1.0, 0, tol=1e-300, max_iter=its)
                except RuntimeError:
                    pass  # not converged: its iterations are what is timed
                torch.cuda.synchronize()
                t.append(time.perf_counter() - a)
            best.append((t[1] - t[0]) / 128)
        return min(best)

    # as many additions: a cell's sum is one addition a member and coordinate either way,
    # and a cell a vertex has three loads a sum where cells of 50 have one
    one, fifty = iteration("one"), iteration("fifty")
    assert one <= 3 * fifty, (one, fifty)
