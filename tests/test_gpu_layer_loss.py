"""A layer's loss and gradient in one pass against the separate calls: the
gradient bit for bit, the loss within a float's rounding of the terms' sum in
double; vertex and edge counts around a block's, the three grid layouts, and
tensors on the host."""
import numpy as np
import pytest
import torch

from meshode_gb300 import _lib as L
from meshode_gb300 import layers, meshgen
from meshode_gb300 import pyDeform as PD

pytestmark = pytest.mark.gpu


def _problem(cuda, nv, layout, seed=3):
    rng = np.random.Generator(np.random.PCG64(seed))
    Vt, Ft = meshgen.icosphere(3)
    pid = PD.InitializeDeformTemplate(torch.from_numpy(meshgen.displace(Vt, rng).astype(np.float32)),
                                      torch.from_numpy(Ft.astype(np.int32)), 0, 24, layout=layout)
    V, F = meshgen.cubesphere(max(2, int(np.ceil(np.sqrt(max(nv - 2, 6) / 6)))))
    F = np.ascontiguousarray(F[(F < nv).all(1)], np.int32)
    if not len(F):
        F = np.zeros((1, 3), np.int32)
    V = torch.from_numpy((V[:nv] * 0.9).astype(np.float32)).to(cuda)
    PD.NormalizeByTemplate(V, pid)
    moved = V + torch.from_numpy(rng.normal(0, 2e-2, (nv, 3)).astype(np.float32)).to(cuda)
    return pid, V, moved, torch.from_numpy(F).to(cuda)


@pytest.mark.parametrize("layout", [L.MO_LAYOUT_LINEAR, L.MO_LAYOUT_CELL, L.MO_LAYOUT_BRICK4])
@pytest.mark.parametrize("nv", [1, 255, 256, 257, 10242])
def test_rigid(cuda, nv, layout):
    pid, V, X, F = _problem(cuda, nv, layout)
    PD.StoreRigidityInformation(V, F, pid)
    d = PD.DistanceFieldLoss_forward(X, pid) * 0.5
    r = PD.RigidEdgeLoss_forward(X, F, pid) * 0.5
    want = float(d.double().sum() + r.double().sum())
    grad = 0.7 * (PD.DistanceFieldLoss_backward(X, pid) + PD.RigidEdgeLoss_backward(X, F, pid))
    for host in (False, True):
        Y = (X.cpu() if host else X.clone()).requires_grad_(True)
        loss = layers.RigidLossFunction.apply(Y, F.cpu() if host else F, pid)
        (loss * 0.7).backward()
        assert loss.shape == () and loss.device == Y.device and loss.dtype == torch.float32
        assert abs(float(loss) - want) <= 3e-7 * want
        assert torch.equal(Y.grad.to(cuda), grad)
    PD.ReleaseTemplate(pid)


@pytest.mark.parametrize("layout", [L.MO_LAYOUT_LINEAR, L.MO_LAYOUT_CELL, L.MO_LAYOUT_BRICK4])
@pytest.mark.parametrize("nv", [3, 256, 5000])
def test_graph(cuda, nv, layout):
    pid, V, X, F = _problem(cuda, nv, layout)
    E = torch.cat([F[:, :2], F[:, 1:]]).contiguous()
    PD.StoreGraphInformation(V, E, pid)
    r2 = float(torch.tensor(0.3))
    d, gd = PD.DistanceFieldLoss_fwd_bwd(X, pid, mask_thresh=layers.GraphLossFunction.MASK)
    r = PD.GraphEdgeLoss_forward(X, E, pid) * 0.5
    want = float((d * 0.5).double().sum() + r.double().sum() * r2)
    grad = 0.7 * (gd + PD.GraphEdgeLoss_backward(X, E, pid) * r2)
    Y = X.clone().requires_grad_(True)
    loss = layers.GraphLossFunction.apply(Y, E, r2, pid)
    (loss * 0.7).backward()
    assert abs(float(loss) - want) <= 3e-7 * want
    assert torch.equal(Y.grad, grad)
    PD.ReleaseTemplate(pid)
