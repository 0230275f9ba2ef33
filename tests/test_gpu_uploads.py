"""Uploads that pass through the context's page-locked ring: the caller's buffer is its own again
when the call returns, more of them than the ring holds are no fewer, sizes on both sides of
what goes through it, and restart payloads."""
import numpy as np
import pytest

import helpers as H
from multiblockmomentsfv_b200 import blockfile as bf, solver as sv

pytestmark = pytest.mark.gpu


def test_buffer_reuse_and_ring_wrap():
    """30 blocks of 20 x 34 cells (37 KB) and one of 120 x 130 (1.2 MB), uploaded three times over
    from one buffer that is overwritten at once: each block holds its own values."""
    sizes = [(20, 34)] * 30 + [(120, 130)]
    d = bf.Deck()
    d.blocks = [bf.Block(k + 1, 0.0, 1.0, 0.0, 1.0, nx, ny, (0, 0, 0, 0)) for k, (nx, ny) in enumerate(sizes)]
    rng = np.random.default_rng(0)
    with sv.Solver(d) as s:
        for _ in range(3):
            want = [rng.standard_normal((b.nyp, b.nxp, 9)) for b in d.blocks]
            buf = {sz: np.empty((sz[1] + 6, sz[0] + 6, 9)) for sz in set(sizes)}
            for b, U in enumerate(want):
                a = buf[sizes[b]]
                a[...] = U
                s.upload(0, b, a)
                a[...] = np.nan
            for b, U in enumerate(want):
                H.assert_bitwise(s.download(0, b), U, f"block {b}")


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_payload_buffer_reuse(dtype):
    d = bf.Deck()
    d.blocks = [bf.Block(k + 1, 0.0, 1.0, 0.0, 1.0, 9 + 60 * (k % 2), 8, (0, 0, 0, 0)) for k in range(4)]
    rng = np.random.default_rng(1)
    with sv.Solver(d) as s:
        want = []
        for b, blk in enumerate(d.blocks):
            p = (1 + rng.random(((blk.nx + 2) * (blk.ny + 2), 10))).astype(dtype)
            s.load_fields(b, p, faithful=True)
            want.append(s.download(0, b))
            s.load_fields(b, p, faithful=True)
            p[...] = 0
        for b in range(4):
            H.assert_bitwise(s.download(0, b), want[b], f"block {b}")


@pytest.mark.parametrize("ncase", [1, 600])
def test_a_wait_for_room_that_runs_out_is_reported(monkeypatch, ncase):
    """The ring is full and the stream busy for longer than MBM_WAIT_TIMEOUT_S: the call that
    needs room returns MBM_ETIMEOUT, as it does where the records of many cases do not fit the
    ring, and the context works again once the stream has caught up."""
    import torch
    from multiblockmomentsfv_b200 import _abi, scenario as sc
    st = torch.cuda.Stream()
    d = bf.Deck(Kn=0.02, limiter=4)
    d.blocks = [bf.Block(1, 0.0, 1.0, 0.0, 1.0, 8, 8, (0, 0, 0, 0))]
    cases = [(d, sc.Scenario.seeded_quadrant(k)) for k in range(ncase)]
    with sv.BatchSolver(cases, stream=st.cuda_stream) as s:
        s.initialise()
        monkeypatch.setenv("MBM_WAIT_TIMEOUT_S", "0.02")
        with torch.cuda.stream(st):
            torch.cuda._sleep(1_500_000_000)                # about 0.8 s
        with pytest.raises(_abi.MBMError) as e:
            for _ in range(4000):
                _abi.check(s.L.mbm_set_physics(s.ctx, 0.02, 0.0), s.ctx)
        assert e.value.status == _abi.MBM_ETIMEOUT
        monkeypatch.setenv("MBM_WAIT_TIMEOUT_S", "60")
        _abi.check(s.L.mbm_set_physics(s.ctx, 0.02, 0.0), s.ctx)
        t, n, _ = s.steps(0.0, 1.0, max_steps=2)
        assert np.all(n == 2)


@pytest.mark.parametrize("mode", ["exact", "fast"])
def test_replayed_steps_on_both_sides_of_the_ring(mode):
    """mbm_replay with more time steps than go through the ring, from page-locked memory, against the
    same steps a part at a time: the same layers, and the same dt however they reach the device."""
    import ctypes as C

    import torch
    from multiblockmomentsfv_b200 import scenario as sc
    d = bf.Deck(Kn=0.05, limiter=4)
    d.blocks = [bf.Block(1, -1.0, 1.0, -1.0, 1.0, 9, 8, (0, 0, 0, 0))]
    n = 14500                                     # 116,000 bytes; the ring takes 114,688
    dts = torch.from_numpy(np.random.default_rng(4).uniform(1e-6, 4e-6, n)).pin_memory()
    out = []
    for parts in ([n], [5000, 1, 9499]):
        with sv.Solver(d, sc.Scenario.seeded_quadrant(6), mode=mode) as s:
            s.initialise()
            at = 0
            for k in parts:
                p = C.cast(dts.data_ptr() + 8 * at, C.POINTER(C.c_double))
                s._check(s.L.mbm_replay(s.ctx, p, k, None))
                at += k
            assert at == n
            out.append(s.download(0, 0))
    H.assert_bitwise(out[0], out[1], "layer")
    assert np.isfinite(out[0]).all()
