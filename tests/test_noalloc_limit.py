"""The allocation-free build's fixed scratch holds the targets that it held when a
tree took 405 bytes a triangle and 12 a vertex: closed meshes of 20,429 triangles."""
import pytest
import torch

from meshode_gb300 import _lib as L

LARGEST = 20_429  # triangles, with half as many vertices


def test_scratch_of_the_largest():
    lib = L.lib()
    cap = int(lib.mo_df_noalloc_scratch_capacity())
    for N in (64, 128, 256):
        assert int(lib.mo_df_build_scratch_bytes(LARGEST // 2 + 2, LARGEST, N, L.MO_DF_AUTO)) <= cap
    assert int(lib.mo_df_build_scratch_bytes(3 * 19_037, 19_037, 64, L.MO_DF_AUTO)) <= cap  # three vertices each


@pytest.mark.gpu
def test_builds_the_largest(cuda):
    g = torch.Generator().manual_seed(1)
    nv, N = LARGEST // 2 + 2, 64
    V = torch.rand(nv, 3, generator=g).to(cuda)
    F = torch.randint(0, nv, (LARGEST, 3), generator=g, dtype=torch.int32).to(cuda)
    bbox = torch.empty(6, dtype=torch.int32, device=cuda)
    prm = torch.empty(4, dtype=torch.float64, device=cuda)
    s = L.stream_ptr()
    L.call("mo_bbox", L.ptr(V), nv, L.ptr(bbox), s)
    L.call("mo_norm_params", L.ptr(bbox), L.ptr(prm), s)
    a, b = torch.empty(N ** 3, device=cuda), torch.empty(N ** 3, device=cuda)
    L.call("mo_df_build_noalloc", L.ptr(V), nv, L.ptr(F), LARGEST, N, L.ptr(prm), L.ptr(a), s)
    L.call("mo_df_build", L.ptr(V), nv, L.ptr(F), LARGEST, N, L.ptr(prm), L.MO_DF_LBVH, None, 0, L.ptr(b), None, s)
    assert torch.equal(a, b)
