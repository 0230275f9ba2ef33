"""What a thread that waits for a long call costs its host."""
import resource
import time

import pytest

from multiblockmomentsfv_b200 import blockfile as bf, scenario as sc, solver as sv

pytestmark = pytest.mark.gpu


def test_a_long_wait_sleeps():
    """A call of a second or more wakes its thread some 2,000 times a second, not 14,000 times."""
    import torch
    st = torch.cuda.Stream()
    d = bf.Deck(Kn=0.02, limiter=4)
    d.blocks = [bf.Block(1, 0.0, 1.0, 0.0, 1.0, 8, 8, (0, 0, 0, 0))]
    with sv.Solver(d, sc.Scenario.seeded_quadrant(1), stream=st.cuda_stream) as s:
        s.initialise()
        with torch.cuda.stream(st):
            torch.cuda._sleep(2_800_000_000)                # 1.4 s or more
        a, t = resource.getrusage(resource.RUSAGE_THREAD).ru_nvcsw, time.perf_counter()
        s.set_boundary(sv.L_DATA, 0.0)
        el = time.perf_counter() - t
        woken = resource.getrusage(resource.RUSAGE_THREAD).ru_nvcsw - a
    assert el > 0.7
    # sleeps of 20 us for a tenth of a second, 5,000 at the most, then of 500 us
    assert woken < 2000 * el + 5000, (woken, el)
