"""Tree builds over so few triangles that the root is a bucket's size itself (and
around it), in scratch memory that holds other numbers: the grid is brute force's,
bit for bit, and the tree does not depend on what the scratch held."""
import ctypes

import numpy as np
import pytest
import torch

from meshode_gb300 import _lib as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nf", [1, 2, 3, 4, 5, 6, 7, 8, 13])
@pytest.mark.parametrize("N", [5, 16, 33])
def test_grid_and_tree(cuda, nf, N):
    rng = np.random.Generator(np.random.PCG64(nf))
    V = torch.from_numpy(rng.random((3 * nf, 3)).astype(np.float32)).to(cuda)
    F = torch.arange(3 * nf, dtype=torch.int32, device=cuda).view(-1, 3)
    s, lib = L.stream_ptr(), L.lib()
    bbox = torch.empty(6, dtype=torch.int32, device=cuda)
    prm = torch.empty(4, dtype=torch.float64, device=cuda)
    L.call("mo_bbox", L.ptr(V), 3 * nf, L.ptr(bbox), s)
    L.call("mo_norm_params", L.ptr(bbox), L.ptr(prm), s)

    def grid(method, fill, band):
        nb = int(lib.mo_df_build_scratch_bytes(3 * nf, nf, N, method))
        scratch = torch.full(((nb + 3) // 4,), fill, device=cuda)
        g = torch.empty(N ** 3, device=cuda)
        opt = L.MoDfOptions(method, L.MO_PACKET_4x4x2, band)
        L.call("mo_df_build_ex", L.ptr(V), 3 * nf, L.ptr(F), nf, N, L.ptr(prm), ctypes.byref(opt), L.ptr(scratch), nb,
               L.ptr(g), None, s)
        return g

    def tree(fill):
        nb = int(lib.mo_df_tree_scratch_bytes(3 * nf, nf))
        scratch = torch.full(((nb + 3) // 4,), fill, device=cuda)
        t = torch.zeros(int(lib.mo_df_tree_bytes(nf)) // 4, dtype=torch.int32, device=cuda)
        st = torch.zeros(1, dtype=torch.int32, device=cuda)
        L.call("mo_df_tree_build", L.ptr(V), 3 * nf, L.ptr(F), nf, L.ptr(prm), L.ptr(scratch), nb, L.ptr(t), L.ptr(st), s)
        assert int(st) == 0
        return t

    for band in (0.0, L.lib().mo_df_loss_band(N)):
        want = grid(L.MO_DF_BRUTE, 0.0, band)
        for fill in (0.0, 10.0, 1e6):
            assert torch.equal(grid(L.MO_DF_LBVH, fill, band), want), (fill, band)
    assert torch.equal(tree(0.0), tree(1e6)) and torch.equal(tree(0.0), tree(10.0))
