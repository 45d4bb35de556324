"""The radix sort when its look-back does not wait: a tile whose predecessors have
not published yet counts their keys itself, and the order is the same stable one
(one tile, tiles of both sizes, many; one to four digits; random keys, equal keys
and two runs)."""
import pytest
import torch

from meshode_gb300 import _lib as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["random", "equal", "runs"])
@pytest.mark.parametrize("n,bits", [(2, 8), (512, 30), (513, 32), (20_001, 17), (131_072, 31), (131_073, 30), (700_001, 24),
                                    (2_000_003, 32)])
@pytest.mark.parametrize("wait", [0, 2_000_000_000])
def test_order(cuda, n, bits, kind, wait):
    g = torch.Generator(device=cuda).manual_seed(n)
    if kind == "random":
        keys = torch.randint(0, 1 << bits, (n,), generator=g, device=cuda, dtype=torch.int64)
    elif kind == "equal":
        keys = torch.full((n,), (1 << bits) - 1, dtype=torch.int64, device=cuda)
    else:
        keys = torch.where(torch.arange(n, device=cuda) % 7 < 3, (1 << bits) - 2, 1)
    want, perm = torch.sort(keys, stable=True)
    k = torch.where(keys >= 1 << 31, keys - (1 << 32), keys).to(torch.int32)
    v = torch.arange(n, dtype=torch.int32, device=cuda)
    nb = int(L.lib().mo_sort_pairs_scratch_bytes(n))
    scratch = torch.full((nb,), 0xAB, dtype=torch.uint8, device=cuda)
    L.call("mo_sort_pairs", L.ptr(k), L.ptr(v), n, bits, L.ptr(scratch), nb, wait, L.stream_ptr())
    assert torch.equal(k.long() & 0xFFFFFFFF, want)
    assert torch.equal(v.long(), perm)
