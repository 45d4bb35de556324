"""Sorts of 2^30 keys and more, which the nearest-point query and the reverse
loss take (up to 2^31 - 1): a digit's count then needs more than the 30 bits that
a look-back word of 32 leaves it.  All keys share a digit here, so the last tile's
count is the number of keys."""
import pytest
import torch

from meshode_gb300 import _lib as L

BIG = (1 << 30) + 1234


def test_room_for_wider_words():
    lib = L.lib()
    a, b = (int(lib.mo_reverse_loss_scratch_bytes(5, n)) for n in ((1 << 30) - 1, 1 << 30))
    assert b - a >= 1 << 31  # 4 passes x 2^19 tiles x 256 words, 4 bytes more each
    a, b = (int(lib.mo_nn_scratch_bytes(2, n)) for n in ((1 << 30) - 1, 1 << 30))
    assert b - a >= 1 << 31


@pytest.mark.gpu
def test_gradient_over_many_targets(cuda):
    ns, used = (1 << 16) + 1, 1 << 16  # 17 bits: the third digit of every key is 0
    idx = torch.arange(BIG, dtype=torch.int32, device=cuda)
    idx %= used
    src, tar = torch.ones(ns, 3, device=cuda), torch.zeros(BIG, 3, device=cuda)
    nb = int(L.lib().mo_reverse_loss_scratch_bytes(ns, BIG))
    scratch = torch.empty(nb, dtype=torch.uint8, device=cuda)
    g = torch.ones(1, device=cuda)
    grad = torch.full((ns, 3), -1.0, device=cuda)
    L.call("mo_reverse_loss_backward", L.ptr(src), ns, L.ptr(tar), BIG, L.ptr(idx), L.ptr(g), L.ptr(grad),
           L.ptr(scratch), nb, None, L.stream_ptr())
    # a sum of ones: the number of targets of each vertex, exactly
    want = torch.zeros(ns, device=cuda)
    want[:used] = float(BIG // used)
    want[:BIG % used] += 1
    assert torch.equal(grad, want[:, None].expand(ns, 3))


@pytest.mark.gpu
def test_many_queries(cuda):
    P = torch.tensor([[0.5, 0.25, 0.125]], device=cuda)
    Q = torch.zeros(BIG, 3, device=cuda)
    idx = torch.full((BIG,), -1, dtype=torch.int32, device=cuda)
    L.call("mo_nn_query", L.ptr(P), 1, L.ptr(Q), BIG, L.ptr(idx), None, None, 0, L.stream_ptr())
    assert int(idx.max()) == 0 and int(idx.min()) == 0
