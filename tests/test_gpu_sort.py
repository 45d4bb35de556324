"""The radix sort of the builders (through mo_lbvh_build's sorted codes and
order, exactly the oracle's stable sort) where its tiles change: one key beside
a tile, the step from small to large tiles, many tiles to look back over; random
codes, one code for all, and codes in two runs."""
import numpy as np
import pytest
import torch

from meshode_gb300 import _lib as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["random", "equal", "runs"])
@pytest.mark.parametrize("nf", [2, 511, 512, 513, 20_001, 131_072, 131_073, 133_120, 700_001])
def test_sorted_codes(cuda, orc, nf, kind):
    rng = np.random.Generator(np.random.PCG64(nf))
    V = rng.uniform(0, 1, (4096, 3)).astype(np.float32)
    if kind == "random":
        F = rng.integers(0, len(V), (nf, 3))
    elif kind == "equal":
        F = np.tile([[1, 2, 3]], (nf, 1))
    else:
        F = np.where((np.arange(nf) % 7 < 3)[:, None], [[1, 2, 3]], [[4, 5, 6]])
    F = F.astype(np.int32)
    dev = torch.device("cuda")
    Vd, Fd = torch.from_numpy(V).to(dev), torch.from_numpy(F).to(dev)
    bbox = torch.empty(6, dtype=torch.int32, device=dev)
    prm = torch.empty(4, dtype=torch.float64, device=dev)
    s = L.stream_ptr()
    L.call("mo_bbox", L.ptr(Vd), len(V), L.ptr(bbox), s)
    L.call("mo_norm_params", L.ptr(bbox), L.ptr(prm), s)
    codes, order = (torch.empty(nf, dtype=torch.int32, device=dev) for _ in range(2))
    left, right = (torch.empty(nf, dtype=torch.int32, device=dev) for _ in range(2))
    L.call("mo_lbvh_build", L.ptr(Vd), len(V), L.ptr(Fd), nf, L.ptr(prm), None, 0, L.ptr(codes), L.ptr(order),
           L.ptr(left), L.ptr(right), None, s)
    scale, trans = orc.normalize_params(V)
    want, perm = orc.sort_codes(orc.morton_codes(orc.normalized_double(V, scale, trans).astype(np.float32), F))
    assert np.array_equal(codes.cpu().numpy().view(np.uint32), want)
    assert np.array_equal(order.cpu().numpy(), perm)
