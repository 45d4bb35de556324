"""The vertex box on either side of the number of vertices up to which one cluster
makes it: the same box, and no more time than past it for nearly as many."""
import numpy as np
import pytest
import torch

from meshode_gb300 import _lib as L

pytestmark = pytest.mark.gpu


def _box(V):
    out = torch.full((6,), 7, dtype=torch.int32, device=V.device)
    prm = torch.empty(4, dtype=torch.float64, device=V.device)
    L.call("mo_bbox_params", L.ptr(V), len(V), L.ptr(out), L.ptr(prm), L.stream_ptr())
    return out, prm


@pytest.mark.parametrize("n", [599_999, 600_000, 600_001, 900_000])
def test_box(cuda, n):
    V = torch.randn(n, 3, generator=torch.Generator().manual_seed(n))
    V[n // 2] = torch.tensor([-40.0, 50.0, float("nan")])
    V[-1] = torch.tensor([60.0, -70.0, 80.0])
    out, prm = _box(V.to(cuda))
    o = out.cpu().numpy()
    box = np.where(o >= 0, o, o ^ 0x7FFFFFFF).astype(np.int32).view(np.float32)
    want = np.concatenate([np.nanmin(V.numpy(), 0), np.nanmax(V.numpy(), 0)])
    assert np.array_equal(box, want)
    assert prm[0].item() == np.max(want[3:].astype(np.float64) - want[:3].astype(np.float64)) * 1.1


def test_time(cuda):
    def us(n):
        V = torch.rand(n, 3, device=cuda)
        box = torch.empty(6, dtype=torch.int32, device=cuda)
        prm = torch.empty(4, dtype=torch.float64, device=cuda)
        out = []
        for _ in range(40):
            torch.cuda.synchronize()
            a, b = torch.cuda.Event(True), torch.cuda.Event(True)
            torch.cuda._sleep(300_000)  # the calls are queued before the first one runs
            a.record()
            L.call("mo_bbox_params", L.ptr(V), n, L.ptr(box), L.ptr(prm), L.stream_ptr())
            b.record()
            b.synchronize()
            out.append(a.elapsed_time(b) * 1e3)
        return float(np.median(out))

    assert us(1_048_000) <= 1.2 * us(1_060_000)
