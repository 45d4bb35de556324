"""The nearest-point query's float culling where it could cut too much: points
and queries of very large, very small and denormal coordinates, queries far from
a dense cluster (all distances equal in float), exact duplicates and queries that
are points, and source points with infinite or NaN coordinates.  Indices and
double distances must equal the brute force's (lowest index among ties) exactly:
the query promises the minimum of the same double expression."""
import numpy as np
import pytest
import torch

from meshode_gb300 import _lib as L

pytestmark = pytest.mark.gpu


def _nn(P, Q):
    Pd, Qd = torch.from_numpy(P).cuda(), torch.from_numpy(Q).cuda()
    idx = torch.empty(len(Q), dtype=torch.int32, device="cuda")
    d2 = torch.empty(len(Q), dtype=torch.float64, device="cuda")
    L.call("mo_nn_query", L.ptr(Pd), len(P), L.ptr(Qd), len(Q), L.ptr(idx), L.ptr(d2), None, 0, L.stream_ptr())
    return idx.cpu().numpy(), d2.cpu().numpy()


def _brute(P, Q):
    with np.errstate(all="ignore"):
        d = P[None].astype(np.float64) - Q[:, None].astype(np.float64)
        D = (d[..., 0] * d[..., 0] + d[..., 1] * d[..., 1]) + d[..., 2] * d[..., 2]
    D = np.where(D < np.finfo(np.float64).max, D, np.inf)
    i = D.argmin(1)  # the first of equal ones
    return i, D[np.arange(len(Q)), i]


@pytest.mark.parametrize("kind", ["unit", "huge", "tiny", "denormal", "far", "duplicates", "nonfinite"])
@pytest.mark.parametrize("n", [2, 33, 1000])
def test_equals_brute_force(cuda, n, kind):
    rng = np.random.Generator(np.random.PCG64(n))
    P, Q = rng.uniform(-1, 1, (n, 3)), rng.uniform(-1.2, 1.2, (700, 3))
    if kind == "huge":
        P, Q = P * 2e38, Q * 2e38
    elif kind == "tiny":
        P, Q = P * 1e-21, Q * 1e-21
    elif kind == "denormal":
        P, Q = P * 1e-43, Q * 1e-43
    elif kind == "far":
        P, Q = 1e-6 * P, Q + 1000.0
    elif kind == "duplicates":
        P = np.concatenate([P[: n // 2 + 1]] * 2)
        Q = np.concatenate([P, Q])
    P, Q = P.astype(np.float32), Q.astype(np.float32)
    if kind == "nonfinite":
        P[::3, 0] = np.inf
        P[1::5, 1] = np.nan
        P[-1] = 0.5  # one finite point at least
    idx, d2 = _nn(P, Q)
    want, dist = _brute(P, Q)
    assert np.array_equal(idx, want)
    assert np.array_equal(d2, dist)
