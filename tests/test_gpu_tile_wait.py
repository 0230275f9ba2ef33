"""Failure detection of the step loop's grid barrier (mbm_tile.cuh): every wait is bounded.  A test
hook (MBM_TILE_TEST_DROP=1 at creation, the first loop only) makes one CTA leave before the
first barrier and shortens the bound to 20 ms: the call reports MBM_ETIMEOUT, and so does each
case that was to run; the next call starts from a clean flag."""
import numpy as np
import pytest

import helpers as H
from multiblockmomentsfv_b200 import _abi, blockfile as bf, scenario as sc, solver as sv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["exact", "fast"])
def test_wait_that_runs_out(monkeypatch, mode):
    cases = []
    for k in range(3):
        d = bf.Deck(Kn=0.02, limiter=4)
        d.blocks = [bf.Block(1, -1.0, 1.0, -1.0, 1.0, 40 + 9 * k, 30, (0, 0, 0, 0))]
        cases.append((d, sc.Scenario.seeded_quadrant(k)))
    tend = np.array([1.0, 0.0, 1.0])                 # the second case has nothing to do
    monkeypatch.setenv("MBM_TILES", "1")

    def run(s):
        s.initialise()
        r = s.steps(0.0, tend, max_steps=4)
        return r, [s.download(l, k, 0) for l in range(3) for k in range(3)]

    with sv.BatchSolver(cases, mode=mode) as s:
        want = run(s)
    monkeypatch.setenv("MBM_TILE_TEST_DROP", "1")
    with sv.BatchSolver(cases, mode=mode) as s:
        s.initialise()
        with pytest.raises(_abi.MBMError) as e:
            s.steps(0.0, tend, max_steps=4)
        assert e.value.status == _abi.MBM_ETIMEOUT
        assert list(s.case_status()) == [_abi.MBM_ETIMEOUT, 0, _abi.MBM_ETIMEOUT]
        t, n, _ = s.steps(2.0, tend)                 # nothing to do for any case: no loop runs
        assert list(n) == [0, 0, 0] and list(t) == [2.0, 2.0, 2.0] and not s.case_status().any()
        got = run(s)
    for x, y in zip(got[0], want[0]):
        assert np.array_equal(x, y)
    for x, y in zip(got[1], want[1]):
        H.assert_bitwise(x, y, "layer")
