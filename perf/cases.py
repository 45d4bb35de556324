"""The work that a user of meshode_gb300 has it do, as cases to be timed.

Sizes are those of the repository's own workloads (the ico-5 rigid pair at 64^3, the 1.3 M-triangle target at 256^3
with a 200k-vertex source, the serving stream's 2k-100k vertices and 5k-500k triangles at 64^3 or 128^3, the 50k-vertex
velocity field, the 41k-vertex linear propagation) and of the ranges around them.  Meshes are cube-spheres of the
generator in meshgen, cut to the exact counts asked for (so they are open at one end and their counts are ragged);
targets are displaced, scaled and rotated by the seed.
"""
import functools
import math

import numpy as np
import torch

from meshode_gb300 import layers, meshgen, neuralode, pool, serving
from meshode_gb300 import fused
from meshode_gb300 import pyDeform as PD


def listed():
    return [
        # a handful of primitives as a target: launches and their latency are all there is
        {"name": "template_320_32", "kind": "template", "nt": 320, "N": 32},
        # the ordinary target: InitializeDeformTemplate of the rigid pair at the reference's 64^3
        {"name": "template_20k_64", "kind": "template", "nt": 20480, "N": 64},
        # a dense scan as a target, exact grid
        {"name": "template_355k_128", "kind": "template", "nt": 355001, "N": 128},
        # one step of the reference's Python loop: RigidLossLayer forward and backward
        {"name": "rigid_layer_10k", "kind": "layer", "edges": "rigid", "nv": 10242, "nt": 20480, "N": 64},
        # the whole loop of one pair on the fused step
        {"name": "fit_10k_64", "kind": "fit", "nv": 10242, "nt": 20480, "N": 64, "steps": 500},
        {"name": "fit_200k_256", "kind": "fit", "nv": 200003, "nt": 1310720, "N": 256, "steps": 500},
        # the serving stream: requests of its mixed sizes offered together to the native pool
        {"name": "serve_32", "kind": "serve", "requests": 32, "stream": 5, "steps": 500},
        # the reverse (target to source) term of a step of inverse_deform and cad_deform2
        {"name": "reverse_50k", "kind": "reverse", "nv": 49688, "nt": 49999},
        # the propagation of a fitted graph to the whole mesh at the end of a CAD deformation
        {"name": "solve_41k", "kind": "solve", "nv": 40963, "cell": 0.06, "rigidity": 1.0},
        # one gradient of a small velocity field, activations kept
        {"name": "ode_2k_w64_stored", "kind": "ode", "nv": 2563, "hidden": 64, "steps": 10, "store": True},
        # one gradient of the full velocity field, checkpointed
        {"name": "ode_50k_w256", "kind": "ode", "nv": 49688, "hidden": 256, "steps": 20, "store": False},
        # a fitted field applied to a denser mesh
        {"name": "flow_200k_w256", "kind": "flow", "nv": 200003, "hidden": 256, "steps": 20},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["template", "template", "layer", "fit", "fit", "serve", "reverse", "solve", "ode", "ode", "flow"])
    if kind == "template":
        N = rng.choice([32, 47, 64, 64, 96, 128, 128])
        return {"kind": kind, "nt": _log(rng, 100, 500_000), "N": N}
    if kind == "layer":
        return {"kind": kind, "edges": rng.choice(["rigid", "graph"]), "nv": _log(rng, 1_000, 200_000),
                "nt": _log(rng, 1_000, 100_000), "N": rng.choice([64, 64, 128])}
    if kind == "fit":
        return {"kind": kind, "nv": _log(rng, 1_000, 200_000), "nt": _log(rng, 1_000, 100_000),
                "N": rng.choice([64, 64, 128]), "steps": _log(rng, 50, 1000)}
    if kind == "serve":
        return {"kind": kind, "requests": _log(rng, 1, 24), "stream": rng.randrange(1 << 20),
                "steps": _log(rng, 100, 500)}
    if kind == "reverse":
        return {"kind": kind, "nv": _log(rng, 1_000, 200_000), "nt": _log(rng, 1_000, 200_000)}
    if kind == "solve":
        return {"kind": kind, "nv": _log(rng, 2_000, 41_000), "cell": rng.uniform(0.03, 0.06),
                "rigidity": rng.choice([0.5, 1.0, 2.0])}
    if kind == "ode":
        return {"kind": kind, "nv": _log(rng, 500, 49_000), "hidden": rng.choice([32, 64, 128, 256, 256]),
                "steps": rng.randint(4, 20), "store": rng.choice([False, True])}
    return {"kind": kind, "nv": _log(rng, 1_000, 200_000), "hidden": rng.choice([64, 256, 256]),
            "steps": rng.randint(4, 20)}


# ---------------------------------------------------------------------------
# meshes
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=96)
def _sphere(n):
    return meshgen.cubesphere(n)


def _source(nv):
    """Unit cube-sphere cut to its first nv vertices: (float64 [nv,3], int32 [nf,3])."""
    V, F = _sphere(max(2, math.ceil(math.sqrt(max(nv - 2, 6) / 6.0))))
    F = F[(F < nv).all(1)]
    return V[:nv], np.ascontiguousarray(F, np.int32)


def _target(nt, rng):
    """Displaced cube-sphere cut to its first nt triangles."""
    V, F = _sphere(max(2, math.ceil(math.sqrt(max(nt, 12) / 12.0))))
    return meshgen.displace(V, rng), np.ascontiguousarray(F[:nt], np.int32)


def _cuda(a, dtype):
    return torch.from_numpy(np.ascontiguousarray(a, dtype)).cuda()


def _pair(case, seed):
    """(source V, source F, target V, target F) on the GPU."""
    rng = np.random.Generator(np.random.PCG64(seed))
    Vs, Fs = _source(case["nv"])
    Vs = Vs * rng.uniform(0.9, 1.0)
    Vt, Ft = _target(case["nt"], rng)
    return _cuda(Vs, np.float32), _cuda(Fs, np.int32), _cuda(Vt, np.float32), _cuda(Ft, np.int32)


class _Template:
    """A template handle that is released with the state that holds it."""

    def __init__(self, pid):
        self.pid = int(pid)

    def __del__(self):
        try:
            PD.ReleaseTemplate(self.pid)
        except Exception:
            pass


def _noise(shape, scale, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(shape, generator=g, device="cuda") * scale


def _field(case, seed):
    """(start positions in the unit cube, parameters of a fitted velocity field, gradient of the loss at the end)."""
    V, _ = _source(case["nv"])
    x0 = _cuda(V * 0.4 + 0.5, np.float32)
    params = neuralode.init_params(case["hidden"], seed)
    for k, p in enumerate(params):
        if k % 2:
            p.add_(_noise(p.shape, 0.05, seed + k))
    params[6].mul_(0.3)
    return x0, params, _noise(x0.shape, 1e-2, seed + 100)


def _cells(V, cell):
    key = np.floor(V / cell).astype(np.int64)
    _, ref = np.unique(key[:, 0] * 10000 + key[:, 1] * 100 + key[:, 2], return_inverse=True)
    return ref.reshape(-1).astype(np.int32)


def _solve_inputs(case, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    V, F = _source(case["nv"])
    V = (0.4 * V + 0.5).astype(np.float32)
    ref = _cells(V, case["cell"])
    ng = int(ref.max()) + 1
    cent = np.zeros((ng, 3))
    np.add.at(cent, ref, V)
    cent /= np.bincount(ref, minlength=ng)[:, None]
    G = ((cent - 0.5) * rng.uniform(0.9, 1.1) + 0.5 + 0.005 * rng.standard_normal(cent.shape)).astype(np.float32)
    i = rng.integers(0, len(V), 200)
    E = np.stack([i, (i + 1) % len(V)], 1).astype(np.int32)
    return _cuda(V, np.float32), _cuda(F, np.int32), _cuda(E, np.int32), _cuda(ref, np.int32), _cuda(G, np.float32)


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind == "template":
        rng = np.random.Generator(np.random.PCG64(seed))
        Vt, Ft = _target(case["nt"], rng)
        st["V"], st["F"] = _cuda(Vt, np.float32), _cuda(Ft, np.int32)
    elif kind == "layer":
        Vs, Fs, Vt, Ft = _pair(case, seed)
        if case["edges"] == "rigid":
            st["idx"] = Fs
            st["layer"] = layers.RigidLossLayer(Vs, Fs, Vt, Ft, grid_resolution=case["N"])
        else:
            st["idx"] = _cuda(meshgen.edges_from_faces(Fs.cpu().numpy()), np.int32)
            st["layer"] = layers.GraphLossLayer(Vs, st["idx"], Vt, Ft, 0.5, grid_resolution=case["N"])
        st["held"] = _Template(st["layer"].param_id)
        st["V"] = (Vs + _noise(Vs.shape, 2e-3, seed)).requires_grad_(True)  # some steps into a fit
    elif kind == "fit":
        Vs, Fs, Vt, Ft = _pair(case, seed)
        st["held"] = _Template(PD.InitializeDeformTemplate(Vt, Ft, 0, case["N"]))
        PD.NormalizeByTemplate(Vs, st["held"].pid)
        PD.StoreRigidityInformation(Vs, Fs, st["held"].pid)
        st["V"] = Vs
    elif kind == "serve":
        specs = meshgen.serving_requests(case["requests"], seed=case["stream"], steps=case["steps"])
        rng = np.random.Generator(np.random.PCG64(seed))
        st["requests"] = []
        for s in specs:
            Vs, Fs = _source(s["nv"])
            Vt, Ft = _target(s["nt"], rng)
            st["requests"].append(serving.Request(s["id"], _cuda(Vs, np.float32), _cuda(Fs, np.int32),
                                                  _cuda(Vt, np.float32), _cuda(Ft, np.int32), N=s["N"],
                                                  steps=s["steps"]))
        st["pool"] = pool.NativePool(group_steps=10, max_building=32, results_to_host=False)
    elif kind == "reverse":
        rng = np.random.Generator(np.random.PCG64(seed))
        Vs, _ = _source(case["nv"])
        Vt, _ = _source(case["nt"])
        st["S"] = _cuda(Vs * 0.9, np.float32).requires_grad_(True)
        st["T"] = _cuda(meshgen.displace(Vt, rng), np.float32)
        st["layer"] = layers.ReverseLossLayer()
    elif kind == "solve":
        st["V"], st["F"], st["E"], st["ref"], st["G"] = _solve_inputs(case, seed)
    else:
        x0, params, gout = _field(case, seed)
        st["x0"], st["gout"] = x0, gout
        st["params"] = [p.requires_grad_(kind == "ode") for p in params]
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "template":
        pid = PD.InitializeDeformTemplate(st["V"], st["F"], 0, case["N"])
        grid = PD.GetDistanceField(pid)
        PD.ReleaseTemplate(pid)
        return grid
    if kind == "layer":
        V = st["V"]
        V.grad = None
        loss = st["layer"](V, st["idx"])
        loss.backward()
        return [loss.detach(), V.grad]
    if kind == "fit":
        out, _ = fused.fused_fit(st["held"].pid, st["V"], case["steps"])
        return out
    if kind == "serve":
        st["pool"].run(st["requests"])
        return [r.out for r in st["requests"]]
    if kind == "reverse":
        S = st["S"]
        S.grad = None
        loss = st["layer"](S, st["T"])
        loss.backward()
        return [loss.detach(), S.grad]
    if kind == "solve":
        V = st["V"].clone()  # solved in place
        PD.SolveLinear(V, st["F"], st["E"], st["ref"], st["G"], case["rigidity"], 0)
        return V
    if kind == "ode":
        x = neuralode.ODEFlow.apply(st["x0"], case["steps"], case["store"], *st["params"])
        return [x.detach()] + list(torch.autograd.grad(x, st["params"], st["gout"]))
    with torch.no_grad():
        return neuralode.ODEFlow.apply(st["x0"], case["steps"], False, *st["params"])


def work(case):
    """Inputs read once and outputs written once; the operations that the results are made of."""
    kind = case["kind"]
    nv, nt, N = case.get("nv", 0), case.get("nt", 0), case.get("N", 0)
    step = 220 * nv + 16 * 6 * nv  # a lookup and its jet, Adam, and six half-edges a vertex
    if kind == "template":  # the nearest triangle's distance, once a voxel
        return {"bytes": 6 * nt + 12 * nt + 4 * N ** 3, "flops": 55 * N ** 3}
    if kind == "layer":
        return {"bytes": (12 + 32 + 12) * nv + (4 + 12) * 6 * nv, "flops": 2 * step}
    if kind == "fit":
        return {"bytes": (12 + 12 + 32) * nv + 4 * 6 * nv, "flops": case["steps"] * step}
    if kind == "serve":
        b = f = 0
        for s in meshgen.serving_requests(case["requests"], seed=case["stream"], steps=case["steps"]):
            b += (12 + 24 + 12) * s["nv"] + 18 * s["nt"]
            f += case["steps"] * 316 * s["nv"] + 55 * s["N"] ** 3
        return {"bytes": b, "flops": f}
    if kind == "reverse":
        return {"bytes": 24 * nv + 12 * nt, "flops": 8 * nt * max(1.0, math.log2(nv)) + 9 * nt}
    if kind == "solve":  # some hundreds of products with the matrix
        return {"bytes": (12 + 24 + 4 + 12) * nv, "flops": 500 * (3 * 2 * 12 + 30) * nv}
    m, ev = case["hidden"], 4 * case["steps"]
    flops = ev * nv * 2 * (6 * m + 2 * m * m) * (3 if kind == "ode" else 1)
    return {"bytes": (36 if kind == "ode" else 24) * nv + 8 * (2 * m * m + 9 * m), "flops": flops}


# ---------------------------------------------------------------------------
# the same in 64 bits, in plain torch
# ---------------------------------------------------------------------------
def _segment_d2(P, A, B):
    AB, AP = B - A, P - A
    t = ((AP * AB).sum(-1) / (AB * AB).sum(-1).clamp_min(1e-300)).clamp(0, 1)
    Q = AP - t[..., None] * AB
    return (Q * Q).sum(-1)


def _triangles_d2(P, A, B, C):
    """Squared distances of points [p,1,3] to triangles [1,t,3]."""
    n = torch.linalg.cross(B - A, C - A)
    nn = (n * n).sum(-1)
    inside = torch.ones((P.shape[0], A.shape[1]), dtype=torch.bool, device=P.device)
    for X, Y in ((A, B), (B, C), (C, A)):
        inside &= (torch.linalg.cross(Y - X, n).expand(1, -1, 3) * (P - X)).sum(-1) <= 0
    d = torch.minimum(torch.minimum(_segment_d2(P, A, B), _segment_d2(P, B, C)), _segment_d2(P, C, A))
    h = ((P - A) * n).sum(-1)
    return torch.where(inside & (nn > 0), h * h / nn.clamp_min(1e-300), d)


def _transform(V):
    """scale and translation of a target's normalisation."""
    lo, hi = V.double().min(0).values, V.double().max(0).values
    scale = (hi - lo).max() * 1.1
    return scale, lo - 0.05 * scale


_BRICK = 8


def _grid(V, F, N):
    """Distances of the voxels x/N to the normalised triangles, [z][y][x] in 64 bits; None where that takes too long."""
    nb = -(-N // _BRICK)
    if nb ** 3 * F.shape[0] > 3e9:
        return None
    scale, trans = _transform(V)
    T = ((V.double() - trans) / scale)[F.long()]
    A, B, C = T[:, 0], T[:, 1], T[:, 2]
    cen = T.mean(1)
    rad = (T - cen[:, None]).norm(dim=-1).max(1).values
    g = torch.empty(nb * _BRICK, nb * _BRICK, nb * _BRICK, dtype=torch.float64, device=V.device)
    k = torch.arange(_BRICK, device=V.device, dtype=torch.float64)
    off = torch.stack(torch.meshgrid(k, k, k, indexing="ij"), -1).reshape(-1, 3).flip(-1)  # x fastest
    reach = math.sqrt(3.0) * (_BRICK - 1) / 2 / N
    for z in range(nb):
        for y in range(nb):
            row = torch.tensor([[x * _BRICK, y * _BRICK, z * _BRICK] for x in range(nb)], device=V.device).double()
            mid = (row + (_BRICK - 1) / 2) / N
            far = torch.cdist(mid, cen, compute_mode="donot_use_mm_for_euclid_dist")
            near = far - rad <= (far + rad).min(1, keepdim=True).values + 2 * reach + 1e-9
            for x in range(nb):
                at = near[x].nonzero()[:, 0]
                P = ((row[x] + off) / N)[:, None]
                best = None
                for part in at.split(4096):
                    d = _triangles_d2(P, A[None, part], B[None, part], C[None, part]).min(1).values
                    best = d if best is None else torch.minimum(best, d)
                g[z * _BRICK:(z + 1) * _BRICK, y * _BRICK:(y + 1) * _BRICK, x * _BRICK:(x + 1) * _BRICK] = \
                    best.sqrt().view(_BRICK, _BRICK, _BRICK)
    return g[:N, :N, :N].contiguous()


def _lookup(grid, P):
    """(distance, its gradient) of points in the unit cube: trilinear, 0 above 0.2, a linear penalty outside."""
    N = grid.shape[0]
    s = P * N
    i = torch.trunc(s).long()
    out = ((i < 0) | (i >= N - 1)).any(1)
    far = N - 1 - 1e-3
    pen = torch.where(i < 0, -s, torch.where(i >= N, s - far, torch.zeros_like(s)))
    gpen = torch.where(i < 0, -float(N), torch.where(i >= N, float(N), 0.0)).double()
    j = i.clamp(0, N - 2)
    w = s - j
    d = torch.zeros(P.shape[0], dtype=torch.float64, device=P.device)
    g = torch.zeros_like(P)
    for b in range(8):
        bit = [(b >> k) & 1 for k in range(3)]
        f = [w[:, k] if bit[k] else 1 - w[:, k] for k in range(3)]
        c = grid[j[:, 2] + bit[2], j[:, 1] + bit[1], j[:, 0] + bit[0]]
        d = d + f[0] * f[1] * f[2] * c
        for k in range(3):
            g[:, k] += (N if bit[k] else -N) * f[(k + 1) % 3] * f[(k + 2) % 3] * c
    cut = d > 0.2
    d, g = torch.where(cut, 0.0, d), torch.where(cut[:, None], 0.0, g)
    return torch.where(out, pen.sum(1), d), torch.where(out[:, None], gpen, g)


def _ends(idx):
    if idx.shape[1] == 3:
        idx = torch.stack([idx, idx.roll(-1, 1)], -1).reshape(-1, 2)
    return idx[:, 0].long(), idx[:, 1].long()


def _objective(grid, idx, rest, weight, mask):
    a, b = _ends(idx)
    off = rest[b] - rest[a]

    def f(V):
        d, g = _lookup(grid, V)
        gd = d[:, None] * g
        if mask is not None:
            gd = gd * (0.5 * d * d < mask)[:, None]
        r = V[b] - V[a] - off
        gr = torch.zeros_like(V).index_add_(0, b, r).index_add_(0, a, -r)
        return 0.5 * (d * d).sum() + weight * 0.5 * (r * r).sum(), gd + weight * gr
    return f


def _normalised(V, T):
    scale, trans = _transform(T)
    return ((V.double() - trans) / scale).float()


def _mlp(p, x):
    sp = torch.nn.functional.softplus
    for k in (0, 2, 4):
        x = sp(x @ p[k].t() + p[k + 1], threshold=40)
    return x @ p[6].t() + p[7]


def _rk4(p, x, h):
    k1 = _mlp(p, x)
    k2 = _mlp(p, x + h / 2 * k1)
    k3 = _mlp(p, x + h / 2 * k2)
    k4 = _mlp(p, x + h * k3)
    return x + h / 6 * (k1 + 2 * k2 + 2 * k3 + k4)


def _flow(case, seed):
    x, params, gout = _field(case, seed)
    p = [q.detach().double().requires_grad_(case["kind"] == "ode") for q in params]
    h = 1.0 / case["steps"]
    states = [x.double()]
    with torch.no_grad():
        for _ in range(case["steps"]):
            states.append(torch.cat([_rk4(p, part, h) for part in states[-1].split(65536)]))
    if case["kind"] == "flow":
        return states[-1]
    grads = [torch.zeros_like(q) for q in p]
    a = gout.double()
    for x in reversed(states[:-1]):
        x = x.requires_grad_(True)
        got = torch.autograd.grad(_rk4(p, x, h), [x] + p, a)
        a = got[0]
        for t, q in zip(grads, got[1:]):
            t += q
    return [states[-1].detach()] + grads


def _solved(case, seed):
    """The linear propagation by conjugate gradients run until nothing changes."""
    V, F, E, ref, G = _solve_inputs(case, seed)
    V, G, ref = V.double(), G.double(), ref.long()
    a, b = (torch.cat(t) for t in zip(_ends(F), _ends(E)))
    w = ((case["rigidity"] * 0.02 / ((V[a] - V[b]).norm(dim=1) + 1e-8)) ** 2)[:, None]
    wg = 1.0 / torch.bincount(ref, minlength=G.shape[0]).clamp_min(1).double()

    def spring(d):
        return torch.zeros_like(V).index_add_(0, a, w * d).index_add_(0, b, -w * d)

    def A(x):
        s = torch.zeros_like(G).index_add_(0, ref, x)
        return 1e-6 * x + (wg * wg)[ref][:, None] * s[ref] + spring(x[a] - x[b])

    rhs = (1e-6 + wg[ref])[:, None] * G[ref] + spring(V[a] - V[b])
    diag = torch.full((V.shape[0], 1), 1e-6, dtype=torch.float64, device=V.device) + (wg * wg)[ref][:, None]
    diag = diag.index_add_(0, a, w).index_add_(0, b, w)
    x = V.clone()
    r = rhs - A(x)
    z = r / diag
    p = z
    rz = (r * z).sum(0)
    for it in range(6000):
        q = A(p)
        alpha = rz / (p * q).sum(0)
        x = x + alpha * p
        r = r - alpha * q
        if it % 50 == 49 and bool((r.norm(dim=0) <= 1e-15 * rhs.norm(dim=0)).all()):
            break
        z = r / diag
        new = (r * z).sum(0)
        p = z + new / rz * p
        rz = new
    return x


def exact(case, seed):
    kind = case["kind"]
    if kind in ("ode", "flow"):
        return _flow(case, seed)
    if kind == "solve":
        return _solved(case, seed)
    if kind == "template":
        Vt, Ft = _target(case["nt"], np.random.Generator(np.random.PCG64(seed)))
        return _grid(_cuda(Vt, np.float32), _cuda(Ft, np.int32), case["N"])
    if kind == "reverse":
        st = prepare(case, seed)
        S, T = st["S"].detach().double(), st["T"].double()
        ii = torch.cat([torch.cdist(t, S, compute_mode="donot_use_mm_for_euclid_dist").argmin(1)
                        for t in T.split(2048)])
        d = S[ii] - T
        return [0.5 * (d * d).sum(), torch.zeros_like(S).index_add_(0, ii, d)]
    if kind == "layer":
        Vs, Fs, Vt, Ft = _pair(case, seed)
        grid = _grid(Vt, Ft, case["N"])
        if grid is None:
            return None
        rest = _normalised(Vs, Vt)
        V = (rest + _noise(rest.shape, 2e-3, seed)).double()
        if case["edges"] == "rigid":
            f = _objective(grid, Fs, rest.double(), 1.0, None)
        else:
            f = _objective(grid, _cuda(meshgen.edges_from_faces(Fs.cpu().numpy()), np.int32), rest.double(), 0.25,
                           0.5 * 0.03 * 0.03)
        return list(f(V))
    if kind == "fit":
        Vs, Fs, Vt, Ft = _pair(case, seed)
        grid = _grid(Vt, Ft, case["N"])
        if grid is None:
            return None
        V = _normalised(Vs, Vt).double()
        f = _objective(grid, Fs, V, 1.0, None)
        m, v = torch.zeros_like(V), torch.zeros_like(V)
        for t in range(1, case["steps"] + 1):
            g = f(V)[1]
            m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
            V = V - 1e-3 / (1 - 0.9 ** t) * m / (v.sqrt() / math.sqrt(1 - 0.999 ** t) + 1e-8)
        return V
    return None  # a stream of whole fits takes too long here
