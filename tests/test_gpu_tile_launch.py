"""The step loop as one cooperative grid (mbm_tile.cuh) beside what else a process does: where the
device refuses the grid the steps go through the graph, with the same result; and contexts
on streams and threads of their own run at the same time."""
import threading

import pytest

import helpers as H
from multiblockmomentsfv_b200 import blockfile as bf, scenario as sc, solver as sv

pytestmark = pytest.mark.gpu


def _run(s):
    s.initialise()
    r = s.steps(0.0, 1.0, max_steps=9)
    r2 = s.steps(r[0], 1.0, max_steps=4)
    return (r, r2), [s.download(l, b) for l in range(3) for b in range(4)]


def _deck(n):
    d = bf.quadrant_deck(n)
    d.Kn, d.limiter = 0.02, 4
    return d


@pytest.mark.parametrize("mode", ["exact", "fast"])
def test_a_grid_that_does_not_fit(monkeypatch, mode):
    """4 x 96^2 cells, 400 tiles: a grid of 400 CTAs is more than are resident."""
    d, scn = _deck(96), sc.Scenario.seeded_quadrant(2)
    monkeypatch.setenv("MBM_TILES", "1")
    with sv.Solver(d, scn, mode=mode) as s:
        want = _run(s)
    monkeypatch.setenv("MBM_TILE_TEST_CTAS", "64")
    with sv.Solver(d, scn, mode=mode) as s:
        got = _run(s)
    assert got[0] == want[0]
    for x, y in zip(got[1], want[1]):
        H.assert_bitwise(x, y, "layer")


def test_contexts_side_by_side(monkeypatch):
    """Four threads, each with a context and stream of its own whose grid fills the device."""
    monkeypatch.setenv("MBM_TILES", "1")
    decks = [(_deck(90 + 6 * k), sc.Scenario.seeded_quadrant(k), ("exact", "fast")[k % 2]) for k in range(4)]
    want = []
    for d, scn, mode in decks:
        with sv.Solver(d, scn, mode=mode) as s:
            want.append(_run(s))
    got = [[] for _ in decks]

    def work(k):
        with sv.Solver(*decks[k][:2], mode=decks[k][2]) as s:
            for _ in range(6):
                got[k].append(_run(s))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(4):
        assert len(got[k]) == 6
        for g in got[k]:
            assert g[0] == want[k][0]
            for x, y in zip(g[1], want[k][1]):
                H.assert_bitwise(x, y, f"context {k}")
