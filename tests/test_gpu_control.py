"""The dt controllers of a batch (control_cases, mbm_step.cuh), one to 32 lanes of a warp for each
case by the cases' mean number of blocks: the row march's graph, whose controller kernel they
run in, against the small grids' step loop, where each is a warp; and what they cost where the
cases are many."""
import ctypes as C
import time

import numpy as np
import pytest

import helpers as H
from multiblockmomentsfv_b200 import _abi, blockfile as bf, scenario as sc, solver as sv

pytestmark = pytest.mark.gpu


def _case(k, nblocks, n):
    d = bf.Deck(Kn=0.01 * (1 + k % 7), limiter=(0, 2, 4)[k % 3], CFL=0.95)
    h = 2.0 / nblocks
    d.blocks = [bf.Block(j + 1, -1.0, 1.0, -1.0 + j * h, -1.0 + (j + 1) * h, n + k % 4, n,
                         (0, 0, j if j > 0 else 0, j + 2 if j < nblocks - 1 else 0)) for j in range(nblocks)]
    return d, sc.Scenario.seeded_quadrant(k)


# 1, 2, 4, 8, 16 and 32 lanes a case, with the cases' numbers of blocks on either side of that
@pytest.mark.parametrize("counts", [[1] * 300, [1] * 99 + [7], [1] * 38 + [9], [1, 4] * 9, [1, 9, 2, 8, 1, 33] * 2,
                                    [1, 9, 2, 8] * 2, [33, 1, 7, 3], [33, 7], [40]])
def test_widths(counts, monkeypatch):
    cases = [_case(k, nb, 6) for k, nb in enumerate(counts)]
    tend = np.array([0.002 * (1 + k % 3) for k in range(len(counts))])
    out = []
    for tiles in ("0", "1"):
        monkeypatch.setenv("MBM_TILES", tiles)
        with sv.BatchSolver(cases) as s:
            s.initialise()
            r = s.steps(0.0, tend, max_steps=40)
            out.append((r, [s.download(0, k, b) for k, nb in enumerate(counts) for b in range(nb)]))
    for x, y in zip(out[0][0], out[1][0]):
        assert np.array_equal(x, y)
    assert (out[0][0][1] > 0).all()
    for x, y in zip(out[0][1], out[1][1]):
        H.assert_bitwise(x, y, "layer")


def test_many_cases_side_by_side(monkeypatch):
    """512 one-block cases: what a step attempt takes beside its stages stays below 120 us (a round of
    dependent loads and divisions per eight cases took 200)."""
    monkeypatch.setenv("MBM_TILES", "0")
    with sv.BatchSolver([_case(0, 1, 24) for _ in range(512)], mode="fast") as s:
        s.initialise()
        s.steps(0.0, 1e3, max_steps=3)
        step = np.inf
        for _ in range(5):
            t = time.perf_counter()
            s.steps(0.0, 1e3, max_steps=60)
            step = min(step, (time.perf_counter() - t) / 60 * 1e6)
        stages, ms = 0.0, C.c_double()
        for heun in (0, 1):
            _abi.check(s.L.mbm_time_stage(s.ctx, heun, 1e-6, 20, C.byref(ms)), s.ctx)
            stages += ms.value * 1e3
    assert step - stages < 120, (step, stages)
