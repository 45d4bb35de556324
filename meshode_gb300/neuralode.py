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

The evaluations of the MLP are one fused libmeshode kernel (mo_mlp_tc_fwd:
the four layers of 128-vertex tiles with their activations kept on chip, and
the RK4 stage update; a flow's evaluations are one launch of it), its
vector-Jacobian product another (mo_mlp_tc_bwd), and the hidden weights'
gradients a split-K kernel over the four stages of a step (mo_mlp_tc_wgrad); a
flow's evaluations are issued by one call (mo_ode_flow, mo_ode_flow_backward).
Their contractions run on the tensor cores in FP16 pairs that carry 22 bits,
accumulated in FP32; everything else is FP32.
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


def _shapes(m):
    return ((m, 3), (m,), (m, m), (m,), (m, m), (m,), (3, m), (3,))


class _Packed:
    """The parameters as the fused kernels take them (mo_mlp_tc_pack): split
    and laid out for the tensor cores, zero-padded to the kernels' width
    (exact: a padded unit's pre-activation and outgoing weights are 0)."""

    def __init__(self, params):
        params = [p.detach() for p in params]
        dev = params[0].device
        m = params[0].shape[0]
        if m > MLP_WIDTH:
            raise RuntimeError("hidden width %d exceeds the fused kernels' %d" % (m, MLP_WIDTH))
        self.units = m
        if m == 0 or any(tuple(p.shape) != s for p, s in zip(params, _shapes(m))):
            # hidden layers of different widths: all padded to the kernels' width,
            # which a larger or differently shaped parameter does not fit
            m = MLP_WIDTH
            params = [self._pad(p, s, dev) for p, s in zip(params[:7], _shapes(m))] + [self._bias4(params[7])]
        params = [p.to(dev, torch.float32).contiguous() for p in params]
        self.m = m  # as packed
        self.M = int(L.lib().mo_mlp_tc_width(m))
        self.dev = dev
        self.buf = torch.empty(int(L.lib().mo_mlp_tc_pack_bytes(self.M)), dtype=torch.uint8, device=dev)
        call("mo_mlp_tc_pack", *[ptr(p) for p in params], m, ptr(self.buf), stream_ptr())

    @staticmethod
    def _pad(t, shape, dev):
        out = torch.zeros(shape, dtype=torch.float32, device=dev)
        out[tuple(slice(0, k) for k in t.shape)] = t
        return out

    @staticmethod
    def _bias4(t):
        if t.numel() < 3:
            raise RuntimeError("b4 needs 3 values, got shape %s" % (tuple(t.shape),))
        return t.reshape(-1)[:3]

    def grads(self):
        return [torch.zeros(sh, dtype=torch.float32, device=self.dev) for sh in _shapes(self.m)]

    def unpad(self, grads):
        if self.m == self.units:
            return grads
        return [g[tuple(slice(0, k) for k in s)].contiguous() for g, s in zip(grads, _shapes(self.units))]


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
        if steps == 0:
            raise ZeroDivisionError("a flow has at least one step")
        if x0.dim() != 2 or x0.shape[1] != 3:
            raise RuntimeError("x0 must be [n, 3], got %s" % (tuple(x0.shape),))
        x = x0.detach().contiguous().float()
        n = x.shape[0]

        def floats(*shape):
            return torch.empty(shape, dtype=torch.float32, device=x.device)

        ckpt = floats(steps, n, 3)
        act = floats(steps, int(L.lib().mo_ode_act_floats(n, P.M))) if store else None
        u = floats(steps if store else 1, 3, n, 3)
        out = torch.empty_like(x)
        call("mo_ode_flow", ptr(x), n, steps, ptr(P.buf), P.M, ptr(ckpt), ptr(act), ptr(u), ptr(out), stream_ptr())
        ctx.P = P
        ctx.kept = (act, u) if store else None
        ctx.save_for_backward(ckpt)
        ctx.steps = steps
        return out

    @staticmethod
    def backward(ctx, a_out):
        (ckpt,) = ctx.saved_tensors
        P = ctx.P
        steps = ctx.steps
        n = ckpt.shape[1]
        grads = P.grads()
        a = a_out.contiguous().float()
        if n > 0:
            act, u = ctx.kept if ctx.kept is not None else (None, None)
            nb = int(L.lib().mo_ode_backward_floats(n, P.M, int(act is not None)))
            scratch = torch.empty(nb, dtype=torch.float32, device=a.device)
            dx = [torch.empty(n, 3, dtype=torch.float32, device=a.device) for _ in range(2)]
            call("mo_ode_flow_backward", ptr(ckpt), n, steps, ptr(P.buf), P.M, P.m, ptr(act), ptr(u), ptr(a),
                 ptr(scratch), nb, ptr(dx[0]), ptr(dx[1]), *[ptr(g) for g in grads], stream_ptr())
            a = dx[0]
        ctx.kept = None
        ctx.P = None
        return (a, None, None) + tuple(P.unpad(grads))


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
