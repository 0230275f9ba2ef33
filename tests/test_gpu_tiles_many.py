"""The small grids' step loop with several tiles on a thread block (mbm_tile.cuh; 296 blocks on a B200):
2 to 26 of them against the row march, every layer bit for bit; one more than a block may
keep; and batches whose cases share blocks, end at different steps or stop."""
import numpy as np
import pytest

import helpers as H
from multiblockmomentsfv_b200 import _abi, blockfile as bf, scenario as sc, solver as sv

pytestmark = pytest.mark.gpu


def _both(monkeypatch, fn):
    out = []
    for v in ("1", "0"):
        monkeypatch.setenv("MBM_TILES", v)
        out.append(fn())
    return out


def _tiles(blocks):
    return sum(-(-(b.nx + 3) // 28) * -(-(b.ny + 3) // 4) for b in blocks)


# n: tiles of 4 n^2 cells on 296 blocks
@pytest.mark.parametrize("mode", ["exact", "fast"])
@pytest.mark.parametrize("n,limiter,F,per_block", [(90, 4, 0.0, 2), (97, 3, 0.2, 2), (165, 2, 0.0, 4), (224, 4, 0.0, 7),
                                                   (311, 1, 0.1, 13), (448, 0, 0.0, 26),
                                                   (457, 4, 0.0, 27)])
def test_square(monkeypatch, mode, n, limiter, F, per_block):
    d = bf.quadrant_deck(n)
    d.Kn, d.limiter, d.F = 0.03, limiter, F
    assert -(-_tiles(d.blocks) // 296) == per_block

    def run():
        with sv.Solver(d, sc.Scenario.seeded_quadrant(n), mode=mode, show_every=2) as s:
            s.initialise()
            r = s.steps(0.0, 1.0, max_steps=5)
            r2 = s.steps(r[0], r[0] + 1e-5)
            return (r, r2), s.trace(), [s.download(l, b) for l in (0, 1, 2) for b in range(4)]

    a, b = _both(monkeypatch, run)
    assert a[0] == b[0] and a[0][0][1] == 5 and np.array_equal(a[1], b[1])
    for x, y in zip(a[2], b[2]):
        H.assert_bitwise(x, y, "layer")


@pytest.mark.parametrize("mode", ["exact", "fast"])
def test_cases_that_share_blocks(monkeypatch, mode):
    """70 cases of two ragged blocks and all limiters, more than 1,800 tiles: a block's tiles are of up to
    seven cases.  One holds an infinity and stops, some are over at once, the others end at
    different steps."""
    cases = []
    for k in range(70):
        d = bf.Deck(Kn=0.01 * (1 + k % 9), limiter=k % 5, F=0.1 * (k % 2), CFL=0.95)
        nx, ny = 20 + 7 * (k % 6), 22 + 3 * (k % 5)
        d.blocks = [bf.Block(1, -1.0, 0.0, -0.5, 0.5, nx, ny, (-2, 2, -1, 0)),
                    bf.Block(2, 0.0, 1.0, -0.5, 0.5, nx + 3, ny, (1, 0, 0, -1))]
        cases.append((d, sc.Scenario.seeded_quadrant(k)))
    total = sum(_tiles(d.blocks) for d, _ in cases)
    assert 6 * 296 < total <= 26 * 296
    tend = np.array([0.0 if k % 11 == 5 else 0.002 * (1 + k % 4) for k in range(70)])

    def run():
        with sv.BatchSolver(cases, mode=mode) as s:
            s.initialise()
            U = s.download(0, 31, 1)
            U[8, 9, 7] = np.inf
            s.upload(0, 31, 1, U)
            r = s.steps(0.0, tend, check=False)
            first = [s.download(0, k, b) for k in range(70) for b in range(2) if k != 31]
            status = s.case_status()
            r2 = s.steps(r[0], r[0] + 0.001, max_steps=3, check=False)
            return r, r2, status, first, [s.download(l, k, b) for l in (0, 1, 2) for k in range(70) for b in range(2)
                                          if k != 31]

    a, b = _both(monkeypatch, run)
    for i in (0, 1):
        for x, y in zip(a[i], b[i]):
            assert np.array_equal(x, y)
    assert list(a[2]) == list(b[2]) == [_abi.MBM_ENONFINITE if k == 31 else 0 for k in range(70)]
    assert len(set(a[0][1])) > 3
    for i in (3, 4):
        for x, y in zip(a[i], b[i]):
            H.assert_bitwise(x, y, "layer")
