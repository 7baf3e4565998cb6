"""FindLowerBounds and FindUpperBounds of keys that are not in order: the starts
are wrong, but each lies in [0, n], nothing beside the table is written and the
device goes on working."""
import ctypes as C

import numpy as np
import pytest

from sphpc_b200 import _lib

pytestmark = pytest.mark.gpu
U = C.POINTER(C.c_uint)
GUARD = 0x5a5a5a5a


def ptr(t):
    return C.cast(t.data_ptr(), U)


def bounds(name, keys, cells):
    import torch
    k = torch.from_numpy(keys.view(np.int32)).cuda()
    out = torch.full((cells + 64,), GUARD, dtype=torch.int32, device="cuda")
    _lib.call(name, ptr(k), len(keys), cells, ptr(out), None)
    out = out.cpu().numpy()
    assert np.all(out[cells:] == GUARD)
    return out[:cells]


@pytest.mark.parametrize("n,cells", [(1, 1), (5, 2049), (3001, 2048), (70_001, 100_003)])
@pytest.mark.parametrize("order", ["reversed", "random", "one_beyond", "one_below"])
def test_keys_out_of_order(n, cells, order):
    rng = np.random.default_rng(n + cells)
    keys = np.sort(rng.integers(0, cells, n)).astype(np.uint32)
    bad = keys.copy()
    if order == "reversed":
        bad = bad[::-1].copy()
    elif order == "random":
        bad = rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32)
    else:
        bad[n // 2] = 0xffffffff if order == "one_beyond" else 0
    for name, side in (("FindLowerBounds", "left"), ("FindUpperBounds", "right")):
        got = bounds(name, bad, cells)
        assert got.min() >= 0 and got.max() <= n
        np.testing.assert_array_equal(bounds(name, keys, cells),
                                      np.searchsorted(keys, np.arange(cells), side))
