"""A few triangles on a large grid, where a packet's index arithmetic and bounds are
most of the work: the grid is the least over single triangles' grids, bit for bit,
on either side of the number that is tested without bounds, and the build takes no
longer than about the relayout of its grid, which moves nine times its bytes."""
import time

import numpy as np
import pytest
import torch

from meshode_gb300 import _lib as L

pytestmark = pytest.mark.gpu


def _builder(nf, N, dev, seed=1):
    g = torch.Generator().manual_seed(seed)
    V = torch.rand(3 * nf, 3, generator=g).to(dev)
    F = torch.arange(3 * nf, dtype=torch.int32, device=dev).view(-1, 3)
    prm = torch.tensor([1.1, -0.05, -0.05, -0.05], dtype=torch.float64, device=dev)
    nb = int(L.lib().mo_df_build_scratch_bytes(3 * nf, nf, N, L.MO_DF_BRUTE))
    scratch = torch.empty(nb, dtype=torch.uint8, device=dev)
    st = torch.zeros(4, dtype=torch.int32, device=dev)

    def build(faces, out):
        L.call("mo_df_build", L.ptr(V), 3 * nf, L.ptr(faces), faces.shape[0], N, L.ptr(prm), L.MO_DF_BRUTE, L.ptr(scratch),
               nb, L.ptr(out), L.ptr(st), L.stream_ptr())
        return out

    return F, build


@pytest.mark.parametrize("nf", [1, 2, 4, 5, 9])
@pytest.mark.parametrize("N", [4, 67, 130])
def test_least_of_single_triangles(cuda, nf, N):
    F, build = _builder(nf, N, cuda)
    want = torch.full((N ** 3,), float("inf"), device=cuda)
    for k in range(nf):
        want = torch.minimum(want, build(F[k:k + 1].contiguous(), torch.empty(N ** 3, device=cuda)))
    assert torch.equal(build(F, torch.empty(N ** 3, device=cuda)), want)


def test_time(cuda):
    N = 256
    F, build = _builder(1, N, cuda)
    lin = torch.empty(N ** 3, device=cuda)
    cells = torch.empty(int(L.lib().mo_grid_bytes(N, L.MO_LAYOUT_CELL)) // 4, device=cuda)

    def median(fn):
        out = []
        for _ in range(15):
            torch.cuda.synchronize()
            t = time.perf_counter()
            fn()
            torch.cuda.synchronize()
            out.append(time.perf_counter() - t)
        return float(np.median(out))

    relayout = median(lambda: L.call("mo_grid_relayout", L.ptr(lin), N, L.MO_LAYOUT_CELL, L.ptr(cells), L.stream_ptr()))
    assert median(lambda: build(F, lin)) <= 1.25 * relayout
