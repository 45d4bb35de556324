"""Brute force on a target far outside the unit cube (mo_df_build takes any
transform): a point and the tip of a triangle on either side of the grid's one
packet, as far from the voxel in its corner as float tells apart.  A triangle that is sorted out is never
the nearest of a voxel: the grid is the least of the two single-triangle grids,
bit for bit."""
import pytest
import torch

from meshode_gb300 import _lib as L

pytestmark = pytest.mark.gpu


def _grid(V, F, N):
    dev = V.device
    prm = torch.tensor([1.0, 0.0, 0.0, 0.0], dtype=torch.float64, device=dev)
    nb = int(L.lib().mo_df_build_scratch_bytes(V.shape[0], F.shape[0], N, L.MO_DF_BRUTE))
    scratch = torch.empty(nb, dtype=torch.uint8, device=dev)
    g = torch.empty(N ** 3, device=dev)
    L.call("mo_df_build", L.ptr(V), V.shape[0], L.ptr(F), F.shape[0], N, L.ptr(prm), L.MO_DF_BRUTE, L.ptr(scratch), nb,
           L.ptr(g), None, L.stream_ptr())
    return g


@pytest.mark.parametrize("far", [0.3, 10.0, 300.0, 5e3, 1e5, 3e7])
def test_nothing_near_is_sorted_out(cuda, far):
    N = 4
    g = torch.Generator().manual_seed(int(far * 10))
    F = torch.tensor([[0, 0, 0], [1, 2, 3]], dtype=torch.int32, device=cuda)
    centre, R = 0.375, 3 ** 0.5 * 0.375
    u = torch.ones(3, dtype=torch.float64) / 3 ** 0.5
    for k in range(400):
        gap, size, wide = torch.rand(3, generator=g, dtype=torch.float64).tolist()
        gap, size = (gap * 2 - 1) * 1e-6 * (far + 1), size * far
        side = torch.linalg.cross(u, torch.randn(3, generator=g, dtype=torch.float64))
        side *= 0.5 * wide * size / side.norm()
        tip = centre + (far + 2 * R + gap) * u
        corners = [tip, tip + size * u + side, tip + size * u - side]
        order = torch.randperm(3, generator=g)
        V = torch.stack([centre - far * u] + [corners[i] for i in order]).float().to(cuda)
        want = torch.minimum(_grid(V, F[:1].contiguous(), N), _grid(V, F[1:].contiguous(), N))
        assert torch.equal(_grid(V, F, N), want), k
