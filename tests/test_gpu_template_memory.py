"""A template whose laid-out grid is large: the grid is not held beside the build's
scratch, a resolution out of range is refused before it is asked for, and it holds
what a small one's path would put there."""
import numpy as np
import pytest
import torch

from meshode_gb300 import _lib as L
from meshode_gb300 import meshgen
from meshode_gb300 import pyDeform as PD

pytestmark = pytest.mark.gpu


def _mesh(nt):
    V, F = meshgen.cubesphere_for_triangles(nt)
    return torch.from_numpy(V.astype(np.float32)), torch.from_numpy(np.ascontiguousarray(F, np.int32))


def test_scratch_is_free_when_the_grid_is_made(cuda):
    V, F = _mesh(700_000)
    N = 330
    grid, linear = int(L.lib().mo_grid_bytes(N, L.MO_LAYOUT_CELL)), 4 * N ** 3
    scratch = int(L.lib().mo_df_build_scratch_bytes(len(V), len(F), N, L.MO_DF_AUTO))
    inputs = 4 * (V.numel() + F.numel())
    assert scratch > 1 << 27
    torch.cuda.synchronize()
    base = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    pid = PD.InitializeDeformTemplate(V, F, 0, N)
    peak = torch.cuda.max_memory_allocated() - base
    PD.ReleaseTemplate(pid)
    assert peak <= linear + max(grid, scratch) + inputs + (1 << 20)


def test_resolution_out_of_range(cuda):
    with pytest.raises(L.MeshodeError, match="out of range"):
        PD.InitializeDeformTemplate(*_mesh(1000), 0, 2049)


@pytest.mark.parametrize("layout", [L.MO_LAYOUT_LINEAR, L.MO_LAYOUT_CELL, L.MO_LAYOUT_BRICK4])
def test_both_ways_give_the_same(cuda, layout, monkeypatch):
    grids = []
    for at_once in (1 << 30, 0):
        monkeypatch.setattr(PD, "GRID_AT_ONCE", at_once, raising=False)
        pid = PD.InitializeDeformTemplate(*_mesh(3000), 0, 19, layout=layout)
        p = PD.GetParams(pid)
        grids.append((p.grid.clone(), PD.GetDistanceField(pid).clone(), p.params.clone()))
        PD.ReleaseTemplate(pid)
    assert all(torch.equal(a, b) for a, b in zip(*grids))
