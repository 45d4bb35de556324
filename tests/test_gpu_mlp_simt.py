"""The row-major FP32 MLP calls of the C ABI (mo_mlp_*: evaluation with its RK4
update, vector-Jacobian product, small gradients, weight gradients) against the
same model in FP64, at row counts around their 64-row tiles.

Tolerance: FP32 sums of 256 products through three layers forward and three
back, a few 1e-7 of each result's scale; 1e-5, the bound of the velocity-field
configuration."""
import pytest
import torch

from meshode_gb300 import _lib as L
from meshode_gb300._lib import call, ptr, stream_ptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 63, 64, 65, 1000, 19_457])
@pytest.mark.parametrize("m", [256, 100])
def test_one_evaluation(cuda, n, m):
    lib, s = L.lib(), stream_ptr()
    M = int(lib.mo_mlp_width())
    g = torch.Generator().manual_seed(n + m)

    def rnd(rows, cols, M_rows, M_cols, scale):  # padded with zeros
        out = torch.zeros(M_rows, M_cols)
        out[:rows, :cols] = (torch.rand(rows, cols, generator=g) * 2 - 1) * scale
        return out.to(cuda)

    W1, W2, W3, W4 = rnd(m, 3, M, 3, 0.15), rnd(m, m, M, M, 0.15), rnd(m, m, M, M, 0.15), rnd(3, m, 3, M, 0.15)
    b1, b2, b3, b4 = [rnd(k, 1, K, 1, 0.1).view(-1) for k, K in ((m, M), (m, M), (m, M), (3, 3))]
    u, x, gk = [torch.rand(n, 3, generator=g).to(cuda) for _ in range(3)]
    a, w = 0.25, 1.0 / 3
    W2T, W3T = torch.empty_like(W2), torch.empty_like(W3)
    call("mo_mlp_transpose", ptr(W2), ptr(W2T), s)
    call("mo_mlp_transpose", ptr(W3), ptr(W3T), s)
    unext, acc = torch.empty(n, 3, device=cuda), torch.ones(n, 3, device=cuda)
    act = torch.empty(6, n, M, device=cuda)
    call("mo_mlp_fwd", ptr(u), ptr(x), n, ptr(W1), ptr(b1), ptr(W2T), ptr(b2), ptr(W3T), ptr(b3), ptr(W4), ptr(b4), a, w,
         0, ptr(unext), ptr(acc), ptr(act), n * M, s)
    gz3, gz2, gu = torch.empty(n, M, device=cuda), torch.empty(n, M, device=cuda), torch.empty(n, 3, device=cuda)
    tiles = int(lib.mo_mlp_tiles(n))
    part = torch.empty(tiles * 8 * int(lib.mo_mlp_partial_floats()), device=cuda)
    call("mo_mlp_bwd", ptr(gk), ptr(u), n, ptr(W1), ptr(W2), ptr(W3), ptr(W4), ptr(act), n * M, ptr(gz3), ptr(gz2), ptr(gu),
         ptr(part), s)
    grads = [torch.zeros(sh, device=cuda) for sh in ((M, 3), (M,), (M, M), (M,), (M, M), (M,), (3, M), (3,))]
    dW1, db1, dW2, db2, dW3, db3, dW4, db4 = grads
    red = torch.empty(int(lib.mo_mlp_partial_reduce_bytes()) // 4, device=cuda)
    call("mo_mlp_partial_reduce", ptr(part), tiles * 8, ptr(red), ptr(dW4), ptr(db4), ptr(db3), ptr(db2), ptr(db1),
         ptr(dW1), s)
    splits = max(1, min(64, n // 256))
    wpart = torch.empty(int(lib.mo_mlp_wgrad_partial_bytes(splits)) // 4, device=cuda)
    call("mo_mlp_wgrad", ptr(gz3), ptr(act[3]), n, splits, ptr(wpart), ptr(dW3), s)
    call("mo_mlp_wgrad", ptr(gz2), ptr(act[1]), n, splits, ptr(wpart), ptr(dW2), s)

    q = [t.double().requires_grad_(True) for t in (W1, b1, W2, b2, W3, b3, W4, b4)]
    ud = u.double().requires_grad_(True)
    h = ud
    hs = []
    for k in (0, 2, 4):
        z = h @ q[k].t() + q[k + 1]
        h = torch.nn.functional.softplus(z, threshold=60)
        hs += [z, h]
    kd = h @ q[6].t() + q[7]
    want = torch.autograd.grad(kd, [ud] + q, gk.double())
    with torch.no_grad():
        pairs = [(unext, x.double() + a * kd), (acc, 1.0 + w * kd)] + [(act[k], hs[k]) for k in range(6)]
    pairs += list(zip([gu] + grads, want))
    for k, (got, ref) in enumerate(pairs):
        assert (got.double() - ref).abs().max() <= 1e-5 * ref.abs().max(), k
