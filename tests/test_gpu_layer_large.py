"""A layer's loss over more vertices and half-edges than its blocks have threads:
within a float's rounding of the terms' sum in double, with infinite and NaN terms as
the separate calls have them, and in no more time than these take."""
import time

import numpy as np
import pytest
import torch

from meshode_gb300 import layers, meshgen
from meshode_gb300 import pyDeform as PD

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def problem(cuda):
    Vt, Ft = meshgen.icosphere(3)
    pid = PD.InitializeDeformTemplate(torch.from_numpy(Vt.astype(np.float32)), torch.from_numpy(Ft.astype(np.int32)), 0, 24)
    V, F = meshgen.cubesphere_for_triangles(8_000_000)
    V, F = torch.from_numpy((V * 0.9).astype(np.float32)).to(cuda), torch.from_numpy(F.astype(np.int32)).to(cuda)
    PD.NormalizeByTemplate(V, pid)
    PD.StoreRigidityInformation(V, F, pid)
    X = V + 0.02 * torch.sin(50 * V)
    yield pid, X, F
    PD.ReleaseTemplate(pid)


def _separate(X, F, pid):
    return PD.DistanceFieldLoss_forward(X, pid) * 0.5, PD.RigidEdgeLoss_forward(X, F, pid) * 0.5


def test_loss(problem):
    pid, X, F = problem
    d, r = _separate(X, F, pid)
    want = float(d.double().sum() + r.double().sum())
    loss = float(layers.RigidLossFunction.apply(X, F, pid))
    # both sums and their sum are rounded to float
    assert abs(loss - want) <= 2 * 2.0 ** -24 * want * 1.001
    assert loss == float(layers.RigidLossFunction.apply(X, F, pid))


@pytest.mark.parametrize("value", [float("nan"), float("inf"), 1e25, 1e15])
def test_large_and_bad_terms(problem, value):
    pid, X, F = problem
    Y = X.clone()
    Y[1234567] = value
    d, r = _separate(Y, F, pid)
    want = (d.double().sum() + r.double().sum()).float()
    loss = layers.RigidLossFunction.apply(Y, F, pid)
    assert torch.equal(torch.isnan(loss), torch.isnan(want)) and torch.equal(torch.isinf(loss), torch.isinf(want))
    if torch.isfinite(want):
        assert abs(float(loss) - float(want)) <= 3e-7 * float(want)


def test_time(problem):
    pid, X, F = problem

    def median(fn):
        out = []
        for _ in range(15):
            torch.cuda.synchronize()
            t = time.perf_counter()
            fn()
            torch.cuda.synchronize()
            out.append(time.perf_counter() - t)
        return float(np.median(out))

    def apart():
        d, r = _separate(X, F, pid)
        return d.sum() + r.sum()

    assert median(lambda: layers.RigidLossFunction.apply(X, F, pid)) <= median(apart)
