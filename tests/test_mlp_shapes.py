"""The velocity field's parameters are handed to the kernels by bare pointers, so
their shapes are checked before: what the kernels are given has the shapes they
read, hidden layers of different widths run zero-padded, and what does not fit is
refused (as is a state that is not [n, 3])."""
import pytest
import torch

from meshode_gb300 import _lib as L
from meshode_gb300 import neuralode


def _params(m1, m2=None, m3=None, seed=0, device="cpu"):
    m2, m3 = m2 or m1, m3 or m2 or m1
    g = torch.Generator().manual_seed(seed)
    shapes = [(m1, 3), (m1,), (m2, m1), (m2,), (m3, m2), (m3,), (3, m3), (3,)]
    return [((torch.rand(s, generator=g) * 2 - 1) * (6.0 / sum(s)) ** 0.5).to(device) for s in shapes]


@pytest.fixture
def given(monkeypatch):
    """The tensors behind the pointers that mo_mlp_tc_pack would be called with."""
    seen = {}
    keep = []

    def ptr(t):
        keep.append(t)
        return t

    def call(name, *args):
        seen[name] = args

    monkeypatch.setattr(neuralode, "ptr", ptr)
    monkeypatch.setattr(neuralode, "call", call)
    monkeypatch.setattr(neuralode, "stream_ptr", lambda: None)

    class Lib:
        @staticmethod
        def mo_mlp_tc_width(m):
            return 64 if m <= 64 else 128 if m <= 128 else 256

        @staticmethod
        def mo_mlp_tc_pack_bytes(W):
            return 8

    monkeypatch.setattr(neuralode.L, "lib", lambda: Lib)
    return seen


def _check_read(args):
    m = args[8]
    want = ((m, 3), (m,), (m, m), (m,), (m, m), (m,), (3, m), (3,))
    for t, s in zip(args[:8], want):
        assert tuple(t.shape) == s and t.is_contiguous() and t.dtype == torch.float32


@pytest.mark.parametrize("widths", [(64, 64, 64), (16, 16, 16), (64, 128, 128), (128, 64, 64), (100, 256, 7), (1, 2, 3)])
def test_what_the_kernels_read(given, widths):
    p = _params(*widths)
    neuralode._Packed(p)
    args = given["mo_mlp_tc_pack"]
    _check_read(args)
    for t, q in zip(args[:8], p):
        cut = tuple(slice(0, k) for k in q.shape)
        assert torch.equal(t[cut], q)
        assert t.abs().sum() == pytest.approx(q.abs().sum().item(), rel=1e-5)  # the rest is zero


@pytest.mark.parametrize("k,shape", [(6, (64, 3)), (1, (64, 1)), (3, (64, 64)), (2, (64, 300)), (4, (257, 64)),
                                     (5, (300,)), (7, (2,)), (0, (64, 4))])
def test_refused(given, k, shape):
    p = _params(64)
    p[k] = torch.zeros(shape)
    with pytest.raises((RuntimeError, IndexError)):
        neuralode._Packed(p)
    assert "mo_mlp_tc_pack" not in given


@pytest.mark.parametrize("shape", [(5, 2), (5, 4), (5, 1), (3,), (1, 5, 3)])
def test_state_of_another_shape(given, shape):
    with pytest.raises(RuntimeError, match="x0"):
        neuralode.ODEFlow.apply(torch.zeros(shape), 2, False, *_params(64))
    assert "mo_ode_flow" not in given


@pytest.mark.gpu
@pytest.mark.parametrize("widths", [(64, 128, 128), (128, 64, 64), (200, 30, 256), (1, 2, 3)])
def test_uneven_widths_against_fp64(cuda, widths):
    p = _params(*widths, seed=3, device=cuda)
    x0 = torch.rand(300, 3, generator=torch.Generator().manual_seed(1)).to(cuda)
    y = neuralode.ODEFlow.apply(x0, 1, False, *p)

    def f(u):
        for k in (0, 2, 4):
            u = torch.nn.functional.softplus(u @ p[k].double().t() + p[k + 1].double(), threshold=60)
        return u @ p[6].double().t() + p[7].double()

    x = x0.double()
    k1 = f(x)
    k2 = f(x + k1 / 2)
    k3 = f(x + k2 / 2)
    want = x + (k1 + 2 * k2 + 2 * k3 + f(x + k3)) / 6
    # a layer is within a few 1e-7 of its scale (22-bit operands, FP32 sums)
    assert (y.double() - want).abs().max() <= 1e-5 * want.abs().max()


@pytest.mark.gpu
def test_a_bias_on_the_host_and_doubles(cuda):
    p = _params(64, seed=3, device=cuda)
    x0 = torch.rand(40, 3, generator=torch.Generator().manual_seed(1)).to(cuda)
    want = neuralode.ODEFlow.apply(x0, 1, False, *p)
    q = [t.cpu() if k in (1, 5) else t.double() for k, t in enumerate(p)]
    assert torch.equal(neuralode.ODEFlow.apply(x0, 1, False, *q), want)
    assert L.lib().mo_mlp_tc_width(64) == 64
