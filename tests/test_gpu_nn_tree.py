"""The nearest-point query where its tree's parts change hands: points around a
chunk of 256 leaves and the sizes at which a node's box is left to a warp or a
block, few queries and many, clustered points (deep trees), and more near-ties
than a query's list holds.  Indices and distances equal the brute force's."""
import numpy as np
import pytest
import torch

from meshode_gb300 import _lib as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 16, 17, 18, 255, 256, 257, 512, 1024, 1025, 1026, 5000, 40000])
@pytest.mark.parametrize("kind, nq", [("even", 1), ("even", 300), ("clusters", 300), ("ties", 300)])
def test_equals_brute_force(cuda, n, kind, nq):
    rng = np.random.Generator(np.random.PCG64(n))
    P = rng.uniform(0, 1, (n, 3))
    Q = rng.uniform(-0.1, 1.1, (nq, 3))
    if kind == "clusters":
        P = 0.5 + 0.3 * np.round(P) + 1e-4 * rng.standard_normal((n, 3)) ** 3
    elif kind == "ties":  # points on a sphere around every tenth query: the same distance but for the last bits
        u = rng.standard_normal((n, 3))
        P = Q[rng.integers(0, nq, n) // 10 * 10] + 0.05 * u / np.linalg.norm(u, axis=1, keepdims=True)
    P, Q = P.astype(np.float32), Q.astype(np.float32)
    Pd, Qd = torch.from_numpy(P).to(cuda), torch.from_numpy(Q).to(cuda)
    idx = torch.full((nq,), -7, dtype=torch.int32, device=cuda)
    d2 = torch.full((nq,), -7.0, dtype=torch.float64, device=cuda)
    L.call("mo_nn_query", L.ptr(Pd), n, L.ptr(Qd), nq, L.ptr(idx), L.ptr(d2), None, 0, L.stream_ptr())
    d = Pd.double()[None] - Qd.double()[:, None]
    D = (d[..., 0] * d[..., 0] + d[..., 1] * d[..., 1]) + d[..., 2] * d[..., 2]
    want = D.min(1).values
    first = torch.where(D == want[:, None], torch.arange(n, device=cuda)[None], n).min(1).values
    assert torch.equal(idx.long(), first) and torch.equal(d2, want)
