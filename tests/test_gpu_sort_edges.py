"""SortByKey and Find{Lower,Upper}Bounds at the edges of their tile sizes:
counts around one tile of 1024, 2048 and 4096 pairs and around the limits
between those sizes, a digit that all keys share, and bounds over empty cells,
block ends and one long run of equal keys."""
import ctypes as C

import numpy as np
import pytest

from sphpc_b200 import _lib

pytestmark = pytest.mark.gpu
U = C.POINTER(C.c_uint)


def ptr(t):
    return C.cast(t.data_ptr(), U)


@pytest.mark.parametrize("n", [1023, 1024, 1025, 3 << 17, (3 << 17) + 1, 3 << 19, (3 << 19) + 1])
@pytest.mark.parametrize("bits", [7, 20, 32])
def test_sort_edges(n, bits):
    import torch
    rng = np.random.default_rng(n + bits)
    keys = (rng.integers(0, 1 << 32, n, dtype=np.uint64) >> (32 - bits)).astype(np.uint32)
    vals = rng.permutation(n).astype(np.uint32)
    k = torch.from_numpy(keys.view(np.int32)).cuda()
    v = torch.from_numpy(vals.view(np.int32)).cuda()
    _lib.call("SortByKey", ptr(k), ptr(v), n, None)
    order = np.argsort(keys, kind="stable")
    np.testing.assert_array_equal(k.cpu().numpy().view(np.uint32), keys[order])
    np.testing.assert_array_equal(v.cpu().numpy().view(np.uint32), vals[order])


@pytest.mark.parametrize("cells", [1, 2047, 2048, 2049, 100_003])
@pytest.mark.parametrize("kind", ["spread", "run", "beyond"])
def test_bounds_edges(cells, kind):
    import torch
    rng = np.random.default_rng(cells)
    n = 70_001
    if kind == "spread":
        keys = rng.integers(0, cells, n)
    elif kind == "run":    # one cell holds more keys than a block reads at once
        keys = np.concatenate([np.full(60_000, cells // 2), rng.integers(0, cells, n - 60_000)])
    else:                  # keys past the last cell
        keys = rng.integers(cells // 2, 3 * cells + 5, n)
    keys = np.sort(keys).astype(np.uint32)
    k = torch.from_numpy(keys.view(np.int32)).cuda()
    lo = torch.empty(cells, dtype=torch.int32, device="cuda")
    hi = torch.empty(cells, dtype=torch.int32, device="cuda")
    _lib.call("FindLowerBounds", ptr(k), n, cells, ptr(lo), None)
    _lib.call("FindUpperBounds", ptr(k), n, cells, ptr(hi), None)
    c = np.arange(cells)
    np.testing.assert_array_equal(lo.cpu().numpy(), np.searchsorted(keys, c, "left"))
    np.testing.assert_array_equal(hi.cpu().numpy(), np.searchsorted(keys, c, "right"))
