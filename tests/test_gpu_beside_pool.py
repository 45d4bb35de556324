"""Calls of one launch whose blocks wait on one another (SolveLinear, fused_fit) and
flows, on a stream of their own beside a busy serving pool: the results of a quiet
GPU, bit for bit, on both sides.  And a flow with its gradient captured in a graph,
and from two threads at once."""
import threading

import numpy as np
import pytest
import torch

from meshode_gb300 import fused, meshgen, neuralode, pool, serving
from meshode_gb300 import pyDeform as PD

pytestmark = pytest.mark.gpu


def _requests(dev):
    specs = meshgen.serving_requests(n=24, seed=3, rate=400.0, steps=400, v_range=(3000, 60_000), t_range=(2000, 40_000),
                                     grids=(32, 64))
    meshes = [meshgen.request_meshes(s) for s in specs]
    return [serving.requests_from_meshes(meshes, specs, device=dev) for _ in range(2)]


def _work(dev):
    """The results of a solve, a fit and a flow with its gradients."""
    V, F = meshgen.cubesphere(40)
    V = (0.4 * V + 0.5).astype(np.float32)
    ref = (np.arange(len(V)) * 60 // len(V)).astype(np.int32)
    G = np.stack([V[ref == g].mean(0) for g in range(60)]).astype(np.float32) * 1.02
    X = torch.from_numpy(V.copy()).to(dev)
    PD.SolveLinear(X, torch.from_numpy(F.astype(np.int32)), torch.zeros(0, 2, dtype=torch.int32), torch.from_numpy(ref),
                   torch.from_numpy(G), 1.0, 0)
    pid = PD.InitializeDeformTemplate(torch.from_numpy(V), torch.from_numpy(F.astype(np.int32)), 0, 32)
    Vs, Fs = meshgen.cubesphere(120)
    Y = torch.from_numpy((0.4 * Vs + 0.5).astype(np.float32)).to(dev)
    PD.StoreRigidityInformation(Y, torch.from_numpy(Fs.astype(np.int32)).to(dev), pid)
    fit, _ = fused.fused_fit(pid, Y, 100)
    PD.ReleaseTemplate(pid)
    return [X, fit] + _flow(*_flow_inputs(dev))


def _flow_inputs(dev, n=3000, m=64):
    p = [t.requires_grad_(True) for t in neuralode.init_params(m, 3, dev)]  # seeds torch's generator
    return torch.rand(n, 3, generator=torch.Generator().manual_seed(1)).to(dev), p


def _flow(x0, p):
    y = neuralode.ODEFlow.apply(x0, 4, False, *p)
    return [y.detach()] + list(torch.autograd.grad(y.square().sum(), p))


def test_beside_a_busy_pool(cuda):
    quiet, busy = _requests(cuda)
    P = pool.NativePool(group_steps=10, results_to_host=False)
    P.run(quiet)
    want = _work(cuda)
    torch.cuda.synchronize()
    done = threading.Event()
    errors = []

    def serve():
        try:
            P.run(busy)
        except Exception as e:  # noqa: BLE001
            errors.append(e)
        finally:
            done.set()

    t = threading.Thread(target=serve)
    t.start()
    rounds = 0
    with torch.cuda.stream(torch.cuda.Stream()):
        while not done.is_set() or rounds == 0:
            got = _work(cuda)
            torch.cuda.current_stream().synchronize()
            assert all(torch.equal(a, b) for a, b in zip(got, want)), rounds
            rounds += 1
    t.join()
    P.close()
    assert not errors, errors
    for a, b in zip(quiet, busy):
        assert b.error is None and torch.equal(a.out, b.out)


def test_flow_in_a_graph(cuda):
    for n, m in ((3000, 64), (40_000, 256)):
        x0 = torch.rand(n, 3, generator=torch.Generator().manual_seed(1)).to(cuda)
        p = [t.requires_grad_(True) for t in neuralode.init_params(m, 3, cuda)]

        def step():
            y = neuralode.ODEFlow.apply(x0, 2, False, *p)
            return [y.detach()] + list(torch.autograd.grad(y.square().sum(), p))

        want = [t.clone() for t in step()]
        with torch.cuda.stream(torch.cuda.Stream()):
            step()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            got = step()
        for t in got:
            t.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, want))


def test_flows_from_two_threads(cuda):
    sizes = ((3000, 64), (25_000, 256))
    inputs = [_flow_inputs(cuda, n, m) for n, m in sizes]
    want = [_flow(*a) for a in inputs]
    torch.cuda.synchronize()
    errors = []

    def body(k):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(10):
                    got = _flow(*inputs[k])
                    torch.cuda.current_stream().synchronize()
                    assert all(torch.equal(a, b) for a, b in zip(got, want[k]))
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=body, args=(k,)) for k in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
