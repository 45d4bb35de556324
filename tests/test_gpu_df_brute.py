"""The brute-force build at its edges (packets that stick out of the grid,
one to eight warps a packet, counts around the 32 triangles a warp bounds at
a time) against the tree's grid, bit for bit, exact and with a band; and a
triangle with a NaN corner, which counts as the edge between its other two."""
import ctypes

import numpy as np
import pytest
import torch

from meshode_gb300 import _lib as L
from meshode_gb300 import meshgen

pytestmark = pytest.mark.gpu


def _grid(V, F, N, method, band):
    s = L.stream_ptr()
    bbox = torch.empty(6, dtype=torch.int32, device=V.device)
    prm = torch.empty(4, dtype=torch.float64, device=V.device)
    L.call("mo_bbox", L.ptr(V), V.shape[0], L.ptr(bbox), s)
    L.call("mo_norm_params", L.ptr(bbox), L.ptr(prm), s)
    g = torch.full((N ** 3,), float("nan"), dtype=torch.float32, device=V.device)
    opt = L.MoDfOptions(method, L.MO_PACKET_4x4x2, band)
    L.call("mo_df_build_ex", L.ptr(V), V.shape[0], L.ptr(F), F.shape[0], N, L.ptr(prm), ctypes.byref(opt), None, 0,
           L.ptr(g), None, s)
    return g


def _mesh(nf, seed, squash):
    rng = np.random.Generator(np.random.PCG64(seed))
    V, F = meshgen.cubesphere_for_triangles(max(nf, 12))
    V = (meshgen.displace(V, rng) * squash).astype(np.float32)
    F = np.ascontiguousarray(F[rng.permutation(len(F))[np.arange(nf) % len(F)]], np.int32)
    F[::13, 2] = F[::13, 1]
    return V, F


@pytest.mark.parametrize("N", [2, 3, 5, 16, 31, 33, 47, 68])
@pytest.mark.parametrize("nf", [1, 2, 31, 33, 256, 257, 700])
def test_brute_force_grid_is_the_tree_grid(cuda, N, nf):
    for squash in ((1, 1, 1), (1, 0.3, 0.1)):
        V, F = _mesh(nf, N * nf, np.array(squash))
        V, F = torch.from_numpy(V).to(cuda), torch.from_numpy(F).to(cuda)
        for band in (0.0, L.lib().mo_df_loss_band(N), 0.01):
            assert torch.equal(_grid(V, F, N, L.MO_DF_BRUTE, band), _grid(V, F, N, L.MO_DF_LBVH, band)), (squash, band)


def test_many_triangles_on_a_coarse_grid(cuda):
    V, F = _mesh(20011, 3, np.ones(3))
    V, F = torch.from_numpy(V).to(cuda), torch.from_numpy(F).to(cuda)
    assert torch.equal(_grid(V, F, 8, L.MO_DF_BRUTE, 0.0), _grid(V, F, 8, L.MO_DF_LBVH, 0.0))


def test_nan_corner_leaves_the_other_edge(cuda):
    V, F = _mesh(320, 5, np.ones(3))
    V = np.concatenate([V, [[np.nan, 0.1, 0.2]]]).astype(np.float32)
    bad = np.array([[len(V) - 1, 3, 9], [4, len(V) - 1, 11], [5, 7, len(V) - 1]], np.int32)
    Vd = torch.from_numpy(V).to(cuda)
    edge = np.array([[3, 3, 9], [4, 4, 11], [5, 7, 7]], np.int32)
    got, want = (_grid(Vd, torch.from_numpy(np.concatenate([F[:100], f, F[100:]])).to(cuda), 32, L.MO_DF_BRUTE, 0.0)
                 for f in (bad, edge))
    # the doubled edge is measured in both directions, a few roundings apart
    assert torch.isfinite(got).all() and (got - want).abs().max() <= 1e-6
