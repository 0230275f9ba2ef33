"""The segment lengths that context creation times (host only): short ones where the resident warps
are not filled without them, and not on grids where each would cost a launch of six rows of
work for two rows of output."""
import ctypes as C

import numpy as np
import pytest

from multiblockmomentsfv_b200 import _abi, blockfile as bf


def _lengths(blocks, warps):
    n = C.c_int()
    out = (C.c_double * 512)()
    _abi.check(_abi.lib().mbm_tune_lengths(_abi.block_descs(blocks), len(blocks), warps, warps, out, 512, C.byref(n)))
    assert n.value <= 512
    return np.array(out[:n.value])


def _items(blocks, rows):
    return sum(-(-(b.nx + 3) // 28) * int(np.ceil((b.ny + 3) / rows - 1e-9)) for b in blocks)


# a B200: 148 SMs, 12 resident warps each in fast arithmetic, 8 bitwise
@pytest.mark.parametrize("warps", [148 * 12, 148 * 8])
@pytest.mark.parametrize("n", [20, 128, 256, 512, 700, 1024, 2000])
def test_short_lengths_where_they_can_pay(warps, n):
    blocks = bf.quadrant_deck(n).blocks
    L = _lengths(blocks, warps)
    waves = _items(blocks, 8) / warps
    lo = 2 if waves < 2 else 6 if waves < 5 else 8
    assert L.min() >= lo - 1e-9 and {float(r) for r in range(lo, 8)} <= set(L)
    assert {float(r) for r in range(8, 65, 2)} <= set(L)
    # besides those, one length for each number of full waves
    extra = len(L) - len(range(8, 65, 2)) - len(range(lo, 8))
    assert 0 <= extra <= max(0, _items(blocks, 2 if waves < 2 else 8) // warps)
    assert all(_items(blocks, r) <= warps * 64 for r in L[-extra:]) if extra else True


def test_the_largest_grid_times_no_more_than_the_long_lengths():
    """4 x 1024^2 cells: 38 candidates fast and 43 bitwise, as many as with a floor of 8 rows (76 and 97
    when lengths from 2 rows were timed on every grid)."""
    blocks = bf.quadrant_deck(1024).blocks
    assert len(_lengths(blocks, 148 * 12)) <= 38 and len(_lengths(blocks, 148 * 8)) <= 43


def test_arguments():
    d = _abi.block_descs(bf.quadrant_deck(8).blocks)
    n = C.c_int()
    assert _abi.lib().mbm_tune_lengths(d, 4, 0, 8, None, 0, C.byref(n)) == _abi.MBM_EINVAL
    assert _abi.lib().mbm_tune_lengths(d, 4, 8, 8, None, 0, C.byref(n)) == _abi.MBM_OK and n.value > 0
