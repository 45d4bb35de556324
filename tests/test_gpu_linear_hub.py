"""SolveLinear with a vertex of many neighbours: on either side of the number of
half-edges up to which neighbours are merged, against the oracle's direct solve
(1e-6 of the box's diagonal, as in test_gpu_linear.py).  A large one takes no
second pass over its pairs of half-edges: the list of them, whose sort is one,
takes longer than half of all that a solve of one iteration does before it."""
import time

import numpy as np
import pytest
import torch

from meshode_gb300 import _lib as L
from meshode_gb300 import pyDeform as PD

pytestmark = pytest.mark.gpu


def _hub(faces, n):
    """A fan of `faces` triangles around vertex 0, which has twice as many half-edges."""
    rng = np.random.Generator(np.random.PCG64(faces))
    V = rng.uniform(0.2, 0.8, (n, 3)).astype(np.float32)
    k = np.arange(1, faces + 1)
    F = np.stack([np.zeros_like(k), k, k + 1], 1).astype(np.int32)
    ref = (np.arange(n) // 25).astype(np.int32)
    G = np.stack([V[ref == g].mean(0) for g in range(ref.max() + 1)]).astype(np.float32)
    return V, F, np.zeros((0, 2), np.int32), ref, G


@pytest.mark.parametrize("faces", [63, 64, 65, 300])
@pytest.mark.parametrize("with_edge", [False, True])  # one half-edge more
def test_against_direct_solve(cuda, orc, faces, with_edge):
    V, F, E, ref, G = _hub(faces, 900)
    if with_edge:
        E = np.array([[0, 5]], np.int32)
    want = orc.solve_linear(V, F, E, ref, G, 1.0, 0)
    X = torch.from_numpy(V.copy()).cuda()
    _, res = PD.SolveLinear(X, *[torch.from_numpy(a) for a in (F, E, ref, G)], 1.0, 0)
    assert res <= 1e-13
    assert np.abs(X.cpu().numpy() - want).max() <= 1e-6 * float(np.linalg.norm(V.max(0) - V.min(0)))


def test_time_of_a_large_hub(cuda):
    V, F, E, ref, G = _hub(1600, 2000)
    dev = [torch.from_numpy(a).to(cuda) for a in (F, E, ref, G)]
    nb = int(L.lib().mo_edge_csr_bytes(len(V), len(F), L.MO_EDGES_FACES))
    csr = torch.empty(nb, dtype=torch.uint8, device=cuda)

    def seconds(fn):
        best = 1e9
        for _ in range(4):
            X = torch.from_numpy(V.copy()).to(cuda)
            torch.cuda.synchronize()
            t = time.perf_counter()
            fn(X)
            torch.cuda.synchronize()
            best = min(best, time.perf_counter() - t)
        return best

    lists = seconds(lambda X: L.call("mo_edge_csr_build", L.ptr(dev[0]), len(F), L.MO_EDGES_FACES, len(V), L.ptr(csr), nb,
                                     None, L.stream_ptr()))
    # one iteration, with any residual
    solve = seconds(lambda X: PD.SolveLinear(X, *dev, 1.0, 0, tol=1e9, max_iter=1))
    assert solve <= 2.0 * lists, (solve, lists)
