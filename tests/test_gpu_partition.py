"""Calls that launch a grid whose blocks wait on one another, in a context that has
only part of the GPU's SMs (a green context): such a grid does not fit there at
the size that fills the GPU."""
import os
import subprocess
import sys

import pytest
import torch

from meshode_gb300 import _lib as L
from meshode_gb300 import fused, meshgen
from meshode_gb300 import pyDeform as PD

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

BODY = r'''
import ctypes, sys
import numpy as np, torch
sys.path.insert(0, sys.argv[1])
from meshode_gb300 import _lib as L, fused, meshgen, pyDeform as PD

torch.cuda.init()
cu = ctypes.CDLL("libcuda.so.1")
P = ctypes.c_void_p

def check(rc, what):
    if rc:
        print("SKIP", what, rc)
        sys.exit(0)

def partition(sms):
    """Makes a context with `sms` of the GPU's SMs the current one; returns how many it got to ask for."""
    whole, part, rest = (ctypes.create_string_buffer(1024) for _ in range(3))  # CUdevResource, opaque here
    n, desc, green, ctx = ctypes.c_uint(1), P(), P(), P()
    check(cu.cuDeviceGetDevResource(0, whole, 1), "cuDeviceGetDevResource")
    check(cu.cuDevSmResourceSplitByCount(part, ctypes.byref(n), whole, rest, 0, sms), "cuDevSmResourceSplitByCount")
    check(cu.cuDevResourceGenerateDesc(ctypes.byref(desc), part, 1), "cuDevResourceGenerateDesc")
    check(cu.cuGreenCtxCreate(ctypes.byref(green), desc, 0, 1), "cuGreenCtxCreate")
    check(cu.cuCtxFromGreenCtx(ctypes.byref(ctx), green), "cuCtxFromGreenCtx")
    return ctx

def in_partition(ctx, fn):
    old = P()
    check(cu.cuCtxGetCurrent(ctypes.byref(old)), "cuCtxGetCurrent")
    check(cu.cuCtxSetCurrent(ctx), "cuCtxSetCurrent")
    try:
        return fn()
    finally:
        cu.cuCtxSynchronize()
        cu.cuCtxSetCurrent(old)

ctx = partition(16)
lib, dev = L.lib(), torch.device("cuda")

# --- SolveLinear
V, F = meshgen.cubesphere(40)
V = (0.4 * V + 0.5).astype(np.float32)
nv, ng = len(V), 60
ref = (np.arange(nv) * ng // nv).astype(np.int32)
G = np.stack([V[ref == g].mean(0) for g in range(ng)]).astype(np.float32) * 1.02
Fd, refd, Gd = [torch.from_numpy(np.ascontiguousarray(a)).to(dev) for a in (F.astype(np.int32), ref, G)]
nb = int(lib.mo_solve_linear_scratch_bytes(nv, len(F), 0, ng, 0))
scratch = torch.empty(nb, dtype=torch.uint8, device=dev)

def solve(X):
    it, res = ctypes.c_int(), ctypes.c_double()
    rc = lib.mo_solve_linear(L.ptr(X), nv, L.ptr(Fd), len(F), None, 0, L.ptr(refd), L.ptr(Gd), ng, 1.0, 0, 1e-13, 20000,
                             L.ptr(scratch), nb, ctypes.byref(it), ctypes.byref(res), None)
    return rc, lib.mo_last_error(), it.value

whole = torch.from_numpy(V.copy()).to(dev)
torch.cuda.synchronize()
rc, msg, it = solve(whole)
assert rc == 0, msg
part = torch.from_numpy(V.copy()).to(dev)
torch.cuda.synchronize()
rc, msg, it2 = in_partition(ctx, lambda: solve(part))
print("solve", rc, msg, it, it2)
if sys.argv[2] == "solve":
    assert rc == 0, msg
    assert (whole - part).abs().max().item() <= 1e-6
    print("OK")
    sys.exit(0)

# --- a fit in one launch
Vs, Fs = meshgen.cubesphere(90)
pid = PD.InitializeDeformTemplate(torch.from_numpy(V), torch.from_numpy(F.astype(np.int32)), 0, 32)
X = torch.from_numpy((0.4 * Vs + 0.5).astype(np.float32)).to(dev)
PD.StoreRigidityInformation(X, torch.from_numpy(Fs.astype(np.int32)).to(dev), pid)
pair = fused.pair_from_template(pid, X, 20)
before = pair.positions().clone()
row = pair.struct(0, 0, fused.tiles_for(pair.nslices))
sync = torch.empty(2, dtype=torch.int32, device=dev)
torch.cuda.synchronize()
rc = in_partition(ctx, lambda: lib.mo_fused_run(ctypes.byref(row), 0, 20, None, 0, L.ptr(sync), None))
print("fit", rc, lib.mo_last_error())
assert rc == 5, rc  # MO_ERR_TOO_LARGE: nothing has run
assert torch.equal(pair.positions(), before)
print("OK")
'''


@pytest.mark.parametrize("what", ["solve", "fit"])
def test_part_of_the_gpu(cuda, what):
    r = subprocess.run([sys.executable, "-c", BODY, ROOT, what], capture_output=True, text=True, timeout=300)
    out = r.stdout + r.stderr
    if "SKIP" in r.stdout:
        pytest.skip(r.stdout.strip())
    assert r.returncode == 0 and r.stdout.rstrip().endswith("OK"), out


@pytest.mark.parametrize("record", [False, True])
def test_fit_goes_on_with_a_launch_per_step(cuda, record, monkeypatch):
    V, F = meshgen.cubesphere(20)
    V, F = torch.from_numpy((0.4 * V + 0.5).astype("float32")), torch.from_numpy(F.astype("int32"))
    pid = PD.InitializeDeformTemplate(V, F, 0, 32)
    PD.StoreRigidityInformation(V, F, pid)
    X = V + 0.01 * torch.sin(40 * V)
    want, losses = fused.fused_fit(pid, X, 30, record_loss=record)
    real = fused.call

    def call(name, *args):
        if name == "mo_fused_run":
            err = L.MeshodeError("too large")
            err.status = L.MO_ERR_TOO_LARGE
            raise err
        return real(name, *args)

    monkeypatch.setattr(fused, "call", call)
    got, losses2 = fused.fused_fit(pid, X, 30, record_loss=record)
    PD.ReleaseTemplate(pid)
    assert torch.equal(got, want)
    assert losses is None and losses2 is None if not record else torch.allclose(losses, losses2, rtol=1e-6, atol=0)
