"""The traversal packet the library picks when a build names none
(mo_df_packet_for): both sides of each of its lines give the grid of the
4x4x2 packet bit for bit, exact and with the loss band, on a target with
degenerate triangles; and the lines themselves."""
import ctypes

import numpy as np
import pytest
import torch

from meshode_gb300 import _lib as L
from meshode_gb300 import meshgen


@pytest.mark.parametrize("N, nf, band, packet", [
    (2, 1, 0.0, L.MO_PACKET_2x4x4_TRI2), (71, 10 ** 6, 0.0, L.MO_PACKET_2x4x4_TRI2),
    (72, 7776, 0.0, L.MO_PACKET_4x4x4), (72, 7777, 0.0, L.MO_PACKET_2x4x4_TRI2),
    (99, 20214, 0.5, L.MO_PACKET_4x4x4), (99, 20215, 0.5, L.MO_PACKET_2x4x4_TRI2),
    (100, 20833, 0.3, L.MO_PACKET_4x4x4), (100, 20834, 0.3, L.MO_PACKET_2x4x4),
    (120, 216_000, 0.3, L.MO_PACKET_4x4x4), (120, 216_001, 0.3, L.MO_PACKET_2x4x4),
    (100, 250_000, 0.0, L.MO_PACKET_4x4x4), (100, 250_001, 0.0, L.MO_PACKET_2x4x4),
])
def test_lines(N, nf, band, packet):
    assert L.lib().mo_df_packet_for(nf, N, band) == packet


@pytest.mark.gpu
@pytest.mark.parametrize("N, nf", [(33, 9001), (71, 839), (72, 7776), (72, 7777), (99, 20215), (100, 20834),
                                   (100, 250_001)])
def test_chosen_packet_gives_the_same_grid(cuda, N, nf):
    V, F = meshgen.cubesphere_for_triangles(nf)
    V = meshgen.displace(V, np.random.Generator(np.random.PCG64(N)))
    F = np.ascontiguousarray(F[np.arange(nf) % len(F)], np.int32)
    F[:: 97, 2] = F[:: 97, 1]  # zero area: the segment tests
    T = torch.from_numpy(np.asarray(V, np.float32)).to(cuda)
    Fd = torch.from_numpy(F).to(cuda)
    s = L.stream_ptr()
    bbox = torch.empty(6, dtype=torch.int32, device=cuda)
    prm = torch.empty(4, dtype=torch.float64, device=cuda)
    L.call("mo_bbox", L.ptr(T), T.shape[0], L.ptr(bbox), s)
    L.call("mo_norm_params", L.ptr(bbox), L.ptr(prm), s)
    assert L.lib().mo_df_method_for(nf, N) == L.MO_DF_LBVH
    for band in (0.0, L.lib().mo_df_loss_band(N)):
        grids = []
        for method in (L.MO_DF_LBVH, L.MO_DF_AUTO):
            opt = L.MoDfOptions(method, L.MO_PACKET_4x4x2, band)
            g = torch.full((N ** 3,), float("nan"), dtype=torch.float32, device=cuda)
            L.call("mo_df_build_ex", L.ptr(T), T.shape[0], L.ptr(Fd), nf, N, L.ptr(prm), ctypes.byref(opt),
                   None, 0, L.ptr(g), None, s)
            grids.append(g)
        assert torch.equal(*grids)
    g = torch.empty_like(grids[0])
    L.call("mo_df_build", L.ptr(T), T.shape[0], L.ptr(Fd), nf, N, L.ptr(prm), L.MO_DF_AUTO, None, 0, L.ptr(g), None, s)
    opt = L.MoDfOptions(L.MO_DF_LBVH, L.MO_PACKET_4x4x2, 0.0)
    L.call("mo_df_build_ex", L.ptr(T), T.shape[0], L.ptr(Fd), nf, N, L.ptr(prm), ctypes.byref(opt), None, 0,
           L.ptr(grids[0]), None, s)
    assert torch.equal(g, grids[0])
