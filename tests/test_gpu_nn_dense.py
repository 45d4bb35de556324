"""Nearest points among many that floats cannot tell apart from the query: lines,
clusters seen from afar, circles around the queries and exact ties, against every
pair in double (lowest index among equals); and the time of the worst of them."""
import time

import pytest
import torch

from meshode_gb300 import _lib as L

pytestmark = pytest.mark.gpu


def _query(P, Q):
    idx = torch.empty(len(Q), dtype=torch.int32, device=P.device)
    d2 = torch.empty(len(Q), dtype=torch.float64, device=P.device)
    L.call("mo_nn_query", L.ptr(P), len(P), L.ptr(Q), len(Q), L.ptr(idx), L.ptr(d2), None, 0, L.stream_ptr())
    return idx.long(), d2


def _sets(kind, n, g):
    P, Q = torch.rand(n, 3, generator=g), torch.rand(1500, 3, generator=g)
    if kind == "line":
        P[:, 1:] = 0.5
    elif kind == "diagonal":
        P[:, 1:] = P[:, :1]
    elif kind == "cluster":
        P *= 1e-4
    elif kind == "far":
        Q += 1000.0
    elif kind == "circle":  # queries near its axis
        a = P[:, 0] * 6.2831853
        P = torch.stack([a.cos(), a.sin(), torch.zeros(n)], 1)
        Q = Q * 1e-6
    elif kind == "ties":
        P = P[torch.randint(0, min(7, n), (n,), generator=g)]
    elif kind == "steps":  # many at a few distances that differ in the last bits
        P[:, 0] = 1.0 + torch.randint(0, 5, (n,), generator=g) * 1.2e-7
        P[:, 1:] = 0.0
        Q[:] = 0.0
    return P, Q


@pytest.mark.parametrize("kind", ["line", "diagonal", "cluster", "far", "circle", "ties", "steps"])
@pytest.mark.parametrize("n", [2, 7, 40, 3000, 20_000])
def test_every_pair_in_double(cuda, kind, n):
    g = torch.Generator().manual_seed(n)
    P, Q = [t.to(cuda) for t in _sets(kind, n, g)]
    idx, d2 = _query(P, Q)
    p, q = P.double(), Q.double()
    best, at = torch.full((len(Q),), float("inf"), dtype=torch.float64, device=cuda), torch.zeros_like(idx)
    for k in range(0, n, 2000):  # x, y, z in turn, every operation rounded
        d = p[None, k:k + 2000] - q[:, None]
        d = (d[..., 0] * d[..., 0] + d[..., 1] * d[..., 1]) + d[..., 2] * d[..., 2]
        m = d.min(1).values
        first = (d == m[:, None]).int().argmax(1) + k
        at = torch.where(m < best, first, at)
        best = torch.minimum(best, m)
    assert torch.equal(d2, best)
    assert torch.equal(idx, at)


def test_time_of_a_dense_line(cuda):
    P, Q = torch.rand(300_000, 3, device=cuda), torch.rand(300_000, 3, device=cuda)
    P[:, 1:] = 0.5
    best = 1e9
    for _ in range(6):
        torch.cuda.synchronize()
        t = time.perf_counter()
        _query(P, Q)
        best = min(best, time.perf_counter() - t)
    assert best <= 2 * 8.9e-3  # 8.9 ms: every box in double
