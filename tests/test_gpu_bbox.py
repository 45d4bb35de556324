"""The vertex box and the normalisation made from it, in one call and in two,
at the edges of the cluster kernel (a coordinate a thread, 16 reads in
flight) and past the vertices it takes: exact against numpy, NaNs ignored."""
import numpy as np
import pytest
import torch

from meshode_gb300 import _lib as L

pytestmark = pytest.mark.gpu


def _float(o):
    o = o.astype(np.int32)
    return np.where(o >= 0, o, o ^ 0x7FFFFFFF).astype(np.int32).view(np.float32)


@pytest.mark.parametrize("n", [1, 2, 33, 2559, 2560, 2561, 40959, 40961, 2 ** 20, 2 ** 20 + 1])
def test_box_and_params(cuda, n):
    rng = np.random.Generator(np.random.PCG64(n))
    V = rng.standard_normal((n, 3)).astype(np.float32)
    V[rng.integers(0, n, n // 7), rng.integers(0, 3, n // 7)] = np.nan
    V[-1] = [-3e8, 0.5, 7e7]  # the last vertex is a corner of the box
    Vd = torch.from_numpy(np.concatenate([[0], V.ravel()]).astype(np.float32)).to(cuda)[1:]  # 4-byte aligned
    s = L.stream_ptr()
    boxes, params = [], []
    for one in (True, False):
        bbox = torch.full((6,), 7, dtype=torch.int32, device=cuda)
        prm = torch.full((4,), 7.0, dtype=torch.float64, device=cuda)
        if one:
            L.call("mo_bbox_params", L.ptr(Vd), n, L.ptr(bbox), L.ptr(prm), s)
        else:
            L.call("mo_bbox", L.ptr(Vd), n, L.ptr(bbox), s)
            L.call("mo_norm_params", L.ptr(bbox), L.ptr(prm), s)
        boxes.append(bbox.cpu().numpy())
        params.append(prm.cpu().numpy())
    assert np.array_equal(boxes[0], boxes[1]) and np.array_equal(params[0], params[1])
    lo, hi = np.nanmin(V, 0), np.nanmax(V, 0)
    assert np.array_equal(_float(boxes[0]), np.concatenate([lo, hi]))
    assert params[0][0] == np.max(hi.astype(np.float64) - lo.astype(np.float64)) * 1.1


def test_no_vertices(cuda):
    bbox = torch.zeros(6, dtype=torch.int32, device=cuda)
    L.call("mo_bbox", None, 0, L.ptr(bbox), L.stream_ptr())
    assert bbox.tolist() == [2 ** 31 - 1] * 3 + [-2 ** 31] * 3
