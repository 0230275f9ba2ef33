"""The stages in tiles and the step loop in one kernel (mbm_tile.cuh; MBM_TILES=1) against the
row march and its graph (MBM_TILES=0): every layer, ghost cells included, bit for bit in both
arithmetic modes, at sizes on and beside the edges of the tiles, with every kind of edge,
every limiter and a body force; in a batch whose cases end at different steps; with ghost
values a caller has set; when a state stops being finite; and mbm_stage_noalloc across its
choices of work items."""
import ctypes as C
import os

import numpy as np
import pytest

import helpers as H
from multiblockmomentsfv_b200 import _abi, blockfile as bf, scenario as sc, solver as sv

pytestmark = pytest.mark.gpu


def _both(fn):
    out = []
    for v in ("1", "0"):
        old = os.environ.get("MBM_TILES")
        os.environ["MBM_TILES"] = v
        try:
            out.append(fn())
        finally:
            if old is None:
                del os.environ["MBM_TILES"]
            else:
                os.environ["MBM_TILES"] = old
    return out


def _same(a, b):
    for x, y in zip(a, b):
        H.assert_bitwise(x, y, "layer")


def _deck(nx, ny, limiter, F=0.0):
    """Two blocks side by side: Dirichlet, wall and open edges and an interface."""
    d = bf.Deck(Kn=0.02, R13=1.0, F=F, limiter=limiter, CFL=0.95)
    d.blocks = [bf.Block(1, -1.0, 0.0, -0.5, 0.5, nx, ny, (-2, 2, -1, 0)),
                bf.Block(2, 0.0, 1.0, -0.5, 0.5, nx + 3, ny, (1, 0, 0, -1))]
    return d


# nx + 3 columns of faces in strips of 28, ny + 3 rows in tiles of 4
@pytest.mark.parametrize("mode", ["exact", "fast"])
@pytest.mark.parametrize("nx,ny,limiter,F", [(3, 3, 4, 0.0), (25, 9, 4, 0.3), (26, 10, 3, 0.0), (24, 5, 2, 0.0),
                                             (54, 29, 1, 0.2), (97, 41, 0, 0.0), (53, 200, 4, 0.0)])
def test_steps(mode, nx, ny, limiter, F):
    d, scn = _deck(nx, ny, limiter, F), sc.Scenario.seeded_quadrant(nx + ny)

    def run():
        with sv.Solver(d, scn, mode=mode, show_every=2) as s:
            s.initialise()
            r = s.steps(0.0, 1.0, max_steps=17)
            r2 = s.steps(r[0], r[0] + 1e-5)          # ends by time, after one step
            return (r, r2), s.trace(), [s.download(l, b) for l in (0, 1, 2) for b in range(2)]

    a, b = _both(run)
    assert a[0] == b[0] and a[0][0][1] == 17 and a[0][1][1] >= 1
    assert np.array_equal(a[1], b[1])
    _same(a[2], b[2])


@pytest.mark.parametrize("mode", ["exact", "fast"])
def test_batch_of_all_limiters(mode):
    cases = []
    for k in range(10):
        d = _deck(7 + 9 * k, 11 + 5 * (k % 4), k % 5, F=0.1 * (k % 2))
        d.Kn = 0.01 * (1 + k)
        cases.append((d, sc.Scenario.seeded_quadrant(50 + k)))
    tend = np.array([0.0 if k == 3 else 0.004 * (1 + k % 4) for k in range(10)])     # case 3 never starts

    def run():
        with sv.BatchSolver(cases, mode=mode) as s:
            s.initialise()
            r = s.steps(0.0, tend)
            return r, [s.download(l, k, b) for l in (0, 1, 2) for k in range(10) for b in range(2)]

    a, b = _both(run)
    for x, y in zip(a[0], b[0]):
        assert np.array_equal(x, y)
    assert a[0][1][3] == 0 and len(set(a[0][1])) > 2
    _same(a[1], b[1])


def test_callers_ghosts_hold_until_the_first_step():
    """steps() on a layer whose ghosts were uploaded, not filled: the first attempts read them."""
    d, scn = _deck(30, 14, 4), sc.Scenario.seeded_quadrant(3)
    rng = np.random.default_rng(3)
    layers = []
    for blk in d.blocks:
        U = sc.initial_state(scn, *blk.centres())
        layers.append(U * (1 + 0.05 * rng.random(U.shape[:2] + (1,))))

    def run():
        with sv.Solver(d, scn) as s:
            for b, U in enumerate(layers):
                s.upload(0, b, U)
            r = s.steps(0.0, 1.0, max_steps=1)
            one = [s.download(l, b) for l in (0, 1, 2) for b in range(2)]
            return r, one, s.steps(r[0], 1.0, max_steps=4), [s.download(l, b) for l in (0, 1, 2) for b in range(2)]

    a, b = _both(run)
    assert a[0] == b[0] and a[2] == b[2]
    _same(a[1], b[1])
    _same(a[3], b[3])


@pytest.mark.parametrize("mode", ["exact", "fast"])
def test_non_finite_case_stops_alone(mode):
    cases = [(_deck(20 + 8 * k, 12, 4), sc.Scenario.seeded_quadrant(k)) for k in range(3)]

    def run():
        with sv.BatchSolver(cases, mode=mode) as s:
            s.initialise()
            U = s.download(0, 1, 0)
            U[8, 9, 7] = np.inf
            s.upload(0, 1, 0, U)
            r = s.steps(0.0, 1.0, max_steps=9, check=False)
            return r, s.case_status(), [s.download(0, k, b) for k in range(3) for b in range(2)]

    a, b = _both(run)
    assert list(a[1]) == list(b[1]) == [0, _abi.MBM_ENONFINITE, 0]
    for x, y in zip(a[0], b[0]):
        assert np.array_equal(x, y)
    for x, y in zip(a[2], b[2]):
        assert np.array_equal(x, y, equal_nan=True)


def test_attempt_limit():
    d = _deck(40, 20, 4)

    def run():
        with sv.Solver(d, sc.Scenario.seeded_quadrant(1), max_attempts=5) as s:
            s.initialise()
            with pytest.raises(_abi.MBMError) as e:
                s.steps(0.0, 10.0)
            return e.value.status, [s.download(l, b) for l in (0, 1, 2) for b in range(2)]

    a, b = _both(run)
    assert a[0] == b[0] == _abi.MBM_ESTEPLIMIT
    _same(a[1], b[1])


@pytest.mark.parametrize("nx,ny", [(3, 3), (25, 5), (53, 122), (700, 331), (1500, 40)])
def test_noalloc_work_items(nx, ny):
    """Tiles, short and long segments of mbm_stage_noalloc give what mbm_update's row march does."""
    import torch
    d = bf.Deck(Kn=0.02, limiter=4)
    d.blocks = [bf.Block(1, -1.0, 1.0, -1.0, 1.0, nx, ny, (0, 0, 0, 0))]
    blk = d.blocks[0]
    rng = np.random.default_rng(nx)
    U = sc.initial_state(sc.Scenario.seeded_quadrant(nx), *blk.centres())
    T = U * (1 + 0.03 * rng.random(U.shape[:2] + (1,)))
    os.environ["MBM_TILES"] = "0"
    try:
        with sv.Solver(d) as s:
            s.upload(0, 0, U)
            s.upload(1, 0, T)
            cfl = [s.update(2, l, 0, 1e-4, 0.0, h)[0] for h, l in ((0, 0), (1, 1))]
            s.update(2, 0, 0, 1e-4, 0.0, 0)
            want = [s.download(2, 0)]
            s.update(2, 1, 0, 1e-4, 0.0, 1)
            want.append(s.download(2, 0))
    finally:
        del os.environ["MBM_TILES"]
    pitch = (blk.nxp + 4) & ~3
    plane = (pitch * blk.nyp + 31) & ~31

    def planes(A):
        t = torch.zeros(9 * plane, dtype=torch.float64)
        torch.as_strided(t, (9, blk.nyp, blk.nxp), (plane, pitch, 1), 1).copy_(torch.from_numpy(A).permute(2, 0, 1))
        return t.cuda()

    u, t = planes(U), planes(T)
    descs, inner = _abi.block_descs([blk]), (slice(3, -3), slice(3, -3))
    for h, x in ((0, u), (1, t)):
        out, c = torch.zeros_like(u), C.c_double(0.0)
        _abi.check(_abi.lib().mbm_stage_noalloc(descs, 1, x.data_ptr(), u.data_ptr(), out.data_ptr(), 0.02, 0.0, 4, 1e-4,
                                                h, C.byref(c), None))
        got = torch.as_strided(out.cpu(), (9, blk.nyp, blk.nxp), (plane, pitch, 1), 1).permute(1, 2, 0).numpy()
        H.assert_bitwise(np.ascontiguousarray(got[inner]), np.ascontiguousarray(want[h][inner]), "stage")
        assert c.value == cfl[h]
