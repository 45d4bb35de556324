"""Distance fields of thin and repeated-vertex triangles: angles whose sine
runs from 0.3 to 1e-9, and exactly collinear and coincident vertices.  Both
build methods give one grid, and it is the FP64 oracle's within 1e-5 of the
target's diagonal (the tolerance of the build's other tests)."""
import numpy as np
import pytest
import torch

from meshode_gb300 import _lib as L
from meshode_gb300 import pyDeform as PD

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sine", [0.3, 0.11, 0.09, 1e-2, 1e-4, 1e-6, 1e-8, 0.0])
@pytest.mark.parametrize("nt, N", [(1, 9), (7, 16), (700, 24)])
def test_thin_triangles_vs_fp64(cuda, orc, sine, nt, N):
    rng = np.random.Generator(np.random.PCG64(nt))
    a = rng.random((nt, 3))
    u = rng.standard_normal((nt, 3))
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    w = np.cross(u, rng.standard_normal((nt, 3)))
    w /= np.linalg.norm(w, axis=1, keepdims=True)
    b = a + u * rng.uniform(0.01, 0.3, (nt, 1))
    c = a + (u + sine * w) * rng.uniform(-0.3, 0.3, (nt, 1))
    V = np.stack([a, b, c], 1).reshape(-1, 3).astype(np.float32)
    F = np.arange(3 * nt, dtype=np.int32).reshape(-1, 3)
    F[::5, 2] = F[::5, 1]  # B == C
    F[2::5, 1] = F[2::5, 0]  # A == B
    F[4::5, 2] = F[4::5, 0]  # A == C
    V = np.concatenate([V, [[0, 0, 0], [1, 1, 1]]]).astype(np.float32)  # a box with an extent in every case
    grids = []
    for method in (L.MO_DF_BRUTE, L.MO_DF_LBVH):
        pid = PD.InitializeDeformTemplate(torch.from_numpy(V), torch.from_numpy(F), 0, N, df_method=method)
        grids.append(PD.GetDistanceField(pid).clone())
        PD.ReleaseTemplate(pid)
    assert torch.equal(*grids)
    scale, trans = orc.normalize_params(V)
    Vn = orc.normalized_double(V, scale, trans)
    ref = orc.df_build(Vn, F, N, method="brute")
    err = np.abs(grids[0].cpu().numpy().reshape(-1) - ref).max()
    assert err <= 1e-5 * np.linalg.norm(Vn.max(0) - Vn.min(0)), err
