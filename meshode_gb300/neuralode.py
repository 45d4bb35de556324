"""Velocity-field ODE deformation with a checkpointed RK4 adjoint.

The reference's NeuralODE variant (src/python/layers/neuralode_fast.py:7-64,
driven by src/python/cad_neural_deform2.py:51-86) deforms the source by
integrating a learned velocity field with torchdiffeq's RK4 and fits it with
the graph/DF losses, back-propagating through the stored RK4 graph.  Here:

* the velocity field is an MLP 3 -> m -> m -> m -> 3 with softplus
  (m = 256, Xavier-uniform weights from ``torch.manual_seed(seed)``, zero
  biases), autonomous (no time input);
* x(1) = RK4(x(0)) with ``steps`` fixed steps over t in [0, 1];
* the fit loss at t = 1 is the GPU DistanceFieldLoss (0.5 sum d^2) plus
  rigidity^2 * RigidEdgeLoss (0.5 sum |r|^2) over the source faces;
* the backward pass is a checkpointed adjoint: only the state at the start
  of every RK4 step is kept; each step's four stage activations are
  recomputed and back-propagated in reverse, accumulating the parameter
  gradients (``store_activations=True`` keeps every stage's activations
  from the forward instead: plain autograd's memory, no recompute, the same
  gradients bit for bit).

Every evaluation of the MLP is one fused libmeshode kernel (mo_mlp_tc_fwd:
the four layers of 128-vertex tiles with their activations kept on chip, and
the RK4 stage update), its vector-Jacobian product another (mo_mlp_tc_bwd), and
the hidden weights' gradients a split-K kernel over the four stages of a step
(mo_mlp_tc_wgrad).  Their contractions run on the tensor cores in FP16 pairs
that carry 22 bits, accumulated in FP32; everything else is FP32.
"""
import math

import torch
from torch.autograd import Function

from . import _lib as L
from . import pyDeform as PD
from ._lib import call, ptr, stream_ptr

PARAM_NAMES = ("W1", "b1", "W2", "b2", "W3", "b3", "W4", "b4")


def init_params(hidden=256, seed=4, device="cuda"):
    """Xavier-uniform weights (torch.manual_seed(seed)), zero biases."""
    torch.manual_seed(seed)
    shapes = [(hidden, 3), (hidden, hidden), (hidden, hidden), (3, hidden)]
    out = []
    for shp in shapes:
        W = torch.empty(shp, dtype=torch.float32)
        torch.nn.init.xavier_uniform_(W)
        out += [W.to(device), torch.zeros(shp[0], dtype=torch.float32, device=device)]
    return out


MLP_WIDTH = 256  # the fused kernels' hidden width; narrower MLPs run zero-padded


class _Packed:
    """The parameters as the fused kernels take them (mo_mlp_tc_pack): split
    and laid out for the tensor cores, zero-padded to the kernels' width
    (exact: a padded unit's pre-activation and outgoing weights are 0)."""

    def __init__(self, params):
        params = [p.detach().float().contiguous() for p in params]
        m = params[0].shape[0]
        if m > MLP_WIDTH:
            raise RuntimeError("hidden width %d exceeds the fused kernels' %d" % (m, MLP_WIDTH))
        self.m = m
        self.M = int(L.lib().mo_mlp_tc_width(m))
        self.dev = params[0].device
        self.buf = torch.empty(int(L.lib().mo_mlp_tc_pack_bytes(self.M)), dtype=torch.uint8, device=self.dev)
        call("mo_mlp_tc_pack", *[ptr(p) for p in params], m, ptr(self.buf), stream_ptr())

    def grads(self):
        m = self.m
        return [torch.zeros(sh, dtype=torch.float32, device=self.dev)
                for sh in ((m, 3), (m,), (m, m), (m,), (m, m), (m,), (3, m), (3,))]


def _fwd(P, u, x, a, w, init_acc, unext, acc, store=None, astride=0):
    """One fused MLP evaluation k = f(u) with the RK4 update
    unext = x + a*k, acc = (init ? x : acc) + w*k (mo_mlp_tc_fwd); store: the
    stage's H1 H2 H3 at stride astride."""
    call("mo_mlp_tc_fwd", ptr(u), ptr(x), u.shape[0], ptr(P.buf), P.M, float(a), float(w), int(init_acc), ptr(unext),
         ptr(acc), ptr(store), int(astride), stream_ptr())


class _StepStore:
    """The activations of one RK4 step's four evaluations:
    act [3][4][rows][M] (H1 H2 H3 of stages 1..4; rows: n padded to whole
    tiles) and the stage inputs u2..u4."""

    def __init__(self, n, M, dev):
        self.n = int(L.lib().mo_mlp_tc_rows(n)) * M  # floats of one array of one stage
        self.act = torch.empty(3 * 4 * self.n, dtype=torch.float32, device=dev)
        self.u = [None, torch.empty(n, 3, dtype=torch.float32, device=dev),
                  torch.empty(n, 3, dtype=torch.float32, device=dev), torch.empty(n, 3, dtype=torch.float32, device=dev)]

    def stage(self, s):
        return self.act[s * self.n:], 4 * self.n

    def array(self, a):
        """Array a (0 H1, 1 H2, 2 H3) of all four stages."""
        return self.act[a * 4 * self.n:(a + 1) * 4 * self.n]


def _rk4_step(P, x, h, st=None):
    """One classic RK4 step of the fused evaluations; with st, the stages'
    activations and inputs are kept there.  Returns x_next."""
    acc = torch.empty_like(x)
    if st is None:
        u2, u3, u4 = torch.empty_like(x), torch.empty_like(x), torch.empty_like(x)
    else:
        u2, u3, u4 = st.u[1], st.u[2], st.u[3]
    ss = [st.stage(k) if st is not None else (None, 0) for k in range(4)]
    _fwd(P, x, x, h / 2, h / 6, 1, u2, acc, *ss[0])
    _fwd(P, u2, x, h / 2, h / 3, 0, u3, acc, *ss[1])
    _fwd(P, u3, x, h, h / 3, 0, u4, acc, *ss[2])
    _fwd(P, u4, x, 0.0, h / 6, 0, None, acc, *ss[3])
    return acc


class _Backward:
    """Work buffers of the adjoint: the stage gradients g_z2, g_z3 of the
    four evaluations of a step ([2][4][rows][M]) and the partial sums of the
    parameter gradients, added to by every step (each block and split of the
    kernels adds to its own, in step order) and reduced once at the end."""

    def __init__(self, n, M, dev):
        lib = L.lib()
        self.n = n
        self.rows = int(lib.mo_mlp_tc_rows(n))
        self.size = self.rows * M

        def floats(k):
            return torch.empty(int(k), dtype=torch.float32, device=dev)

        self.gz = floats(2 * 4 * self.size)
        self.partial = floats(lib.mo_mlp_tc_partial_floats(n, M))
        self.wpart = [floats(lib.mo_mlp_tc_wgrad_floats(4 * self.rows, M)) for _ in range(2)]
        self.gu = [torch.empty(n, 3, dtype=torch.float32, device=dev) for _ in range(2)]
        self.dx = [torch.empty(n, 3, dtype=torch.float32, device=dev) for _ in range(2)]
        self.evals = self.steps = 0

    def stage_vjp(self, P, st, s, u, a, ca, cg, dx_in, dx_out):
        """Evaluation s (0..3) of the step: dL/dk = ca*a + cg*(dL/du of the
        evaluation handled before); dx_out = dx_in + dL/du."""
        act, astride = st.stage(s)
        prev, out = self.gu[self.evals & 1], self.gu[1 - (self.evals & 1)]
        call("mo_mlp_tc_bwd", ptr(a), float(ca), ptr(prev) if cg else None, float(cg), ptr(u), self.n, ptr(P.buf), P.M,
             ptr(act), int(astride), ptr(self.gz[s * self.size:]), ptr(self.gz[(4 + s) * self.size:]), ptr(dx_in),
             ptr(dx_out), ptr(out), ptr(self.partial), int(self.evals == 0), stream_ptr())
        self.evals += 1

    def weights(self, P, st):
        """The hidden weights' gradients of the step's four evaluations."""
        s = stream_ptr()
        for k, layer in ((0, 2), (1, 3)):
            call("mo_mlp_tc_wgrad", ptr(self.gz[4 * k * self.size:]), ptr(st.array(k)), 4 * self.rows, ptr(P.buf), P.M,
                 layer, ptr(self.wpart[k]), int(self.steps == 0), s)
        self.steps += 1

    def reduce(self, P, grads):
        call("mo_mlp_tc_reduce", ptr(self.partial), self.n, ptr(self.wpart[0]), ptr(self.wpart[1]), 4 * self.rows, P.M,
             P.m, *[ptr(g) for g in grads], stream_ptr())


class ODEFlow(Function):
    """x(1) = RK4^steps(x(0)) under the velocity MLP, with an adjoint
    backward on the fused kernels.  store=False: checkpointed (states at
    step starts kept, each step's stage activations recomputed in the
    backward: one step's activations in memory); store=True: every step's
    activations kept from the forward (no recompute).  Both give the same
    gradients bit for bit (the recompute repeats the same kernels)."""

    @staticmethod
    def forward(ctx, x0, steps, store, W1, b1, W2, b2, W3, b3, W4, b4):
        P = _Packed((W1, b1, W2, b2, W3, b3, W4, b4))
        steps = int(steps)
        h = 1.0 / steps
        x = x0.detach().contiguous().float()
        n = x.shape[0]
        ckpt = torch.empty(steps, n, 3, dtype=torch.float32, device=x.device)
        ctx.stores = [] if store else None
        for k in range(steps):
            ckpt[k].copy_(x)
            st = _StepStore(n, P.M, x.device) if store else None
            x = _rk4_step(P, x, h, st)
            if store:
                ctx.stores.append(st)
        ctx.P = P
        ctx.save_for_backward(ckpt)
        ctx.steps = steps
        return x

    @staticmethod
    def backward(ctx, a_out):
        (ckpt,) = ctx.saved_tensors
        P = ctx.P
        steps = ctx.steps
        h = 1.0 / steps
        n = ckpt.shape[1]
        grads = P.grads()
        a = a_out.contiguous().float()
        if n > 0 and steps > 0:
            B = _Backward(n, P.M, a.device)
            work = None if ctx.stores is not None else _StepStore(n, P.M, a.device)
            for k in reversed(range(steps)):
                xk = ckpt[k]
                if ctx.stores is not None:
                    st = ctx.stores[k]
                    ctx.stores[k] = None
                else:
                    st = work
                    _rk4_step(P, xk, h, st)
                # dk4 = a h/6, dk3 = a h/3 + h g4, dk2 = a h/3 + h/2 g3, dk1 = a h/6 + h/2 g2;
                # dL/dx = a + g4 + g3 + g2 + g1
                dx = B.dx[k & 1]
                B.stage_vjp(P, st, 3, st.u[3], a, h / 6, 0.0, a, dx)
                B.stage_vjp(P, st, 2, st.u[2], a, h / 3, h, dx, dx)
                B.stage_vjp(P, st, 1, st.u[1], a, h / 3, h / 2, dx, dx)
                B.stage_vjp(P, st, 0, xk, a, h / 6, h / 2, dx, dx)
                B.weights(P, st)
                a = dx
            B.reduce(P, grads)
        ctx.stores = None
        ctx.P = None
        return (a, None, None) + tuple(grads)


class FitLossFunction(Function):
    """0.5 sum d(x)^2 + rigidity^2 * 0.5 sum |r|^2 of the deformed source
    (the GraphLoss2Function objective, src/python/layers/graph_loss2_layer.py:
    9-41, with the source faces' half-edges as the edge set)."""

    @staticmethod
    def forward(ctx, X, F, pid, rigidity2):
        lossD, gD = PD.DistanceFieldLoss_fwd_bwd(X, pid)
        lossR = PD.RigidEdgeLoss_forward(X, F, pid)
        gR = PD.RigidEdgeLoss_backward(X, F, pid)
        ctx.save_for_backward(gD, gR)
        ctx.r2 = float(rigidity2)
        return lossD.double().sum() * 0.5 + lossR.double().sum() * 0.5 * ctx.r2

    @staticmethod
    def backward(ctx, grad_h):
        gD, gR = ctx.saved_tensors
        return grad_h.float() * (gD + gR * ctx.r2), None, None, None


class NeuralODEDeformer:
    """The velocity-field fit: source normalised by the target template, the
    MLP parameters are the optimisation variables (torch.optim.Adam)."""

    def __init__(self, src_V, src_F, tar_V, tar_F, grid_resolution=128, rigidity=0.1, hidden=256, steps=20,
                 seed=4, lr=1e-3, store_activations=False):
        L.require_cuda()
        dev = torch.device("cuda", torch.cuda.current_device())
        self.pid = PD.InitializeDeformTemplate(tar_V, tar_F, 0, grid_resolution)
        self.x0 = src_V.detach().to(dev).float().contiguous().clone()
        PD.NormalizeByTemplate(self.x0, self.pid)
        self.F = src_F.detach().to(dev).contiguous()
        PD.StoreRigidityInformation(self.x0, self.F, self.pid)
        self.rigidity2 = float(torch.tensor(rigidity * rigidity, dtype=torch.float32))
        self.steps = int(steps)
        # False: checkpointed adjoint (low memory); True: activations kept (faster)
        self.store_activations = bool(store_activations)
        self.params = [p.requires_grad_(True) for p in init_params(hidden, seed, dev)]
        self.opt = torch.optim.Adam(self.params, lr=lr)

    def deformed(self):
        return ODEFlow.apply(self.x0, self.steps, self.store_activations, *self.params)

    def loss(self):
        return FitLossFunction.apply(self.deformed(), self.F, self.pid, self.rigidity2)

    def step(self):
        self.opt.zero_grad()
        L_ = self.loss()
        L_.backward()
        self.opt.step()
        return L_.detach()
