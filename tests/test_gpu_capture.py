"""Calls that take host data on a stream that is being captured into a graph are refused: the graph
would read the context's page-locked ring when it is launched, after the bytes there have
changed.  The capture itself stays valid, and the context works on afterwards."""
import ctypes as C
import glob
import os

import numpy as np
import pytest

import helpers as H
from multiblockmomentsfv_b200 import _abi, blockfile as bf, scenario as sc, solver as sv

pytestmark = pytest.mark.gpu


def _runtime():
    """torch's own CUDA runtime."""
    import torch
    for pat in ("nvidia/cuda_runtime/lib/libcudart.so.12", "torch/lib/libcudart*.so*"):
        for f in glob.glob(os.path.join(os.path.dirname(os.path.dirname(torch.__file__)), pat)):
            return C.CDLL(f)
    return C.CDLL("libcudart.so.12")


CALLS = {
    "upload": lambda s, U, p: s.upload(sv.L_DATA, 0, U),
    "load_fields": lambda s, U, p: s.load_fields(0, p),
    "set_physics": lambda s, U, p: s._check(s.L.mbm_set_physics(s.ctx, C.c_double(0.1), C.c_double(0.0))),
    "steps_async": lambda s, U, p: s._check(s.L.mbm_steps_batch_async(
        s.ctx, (C.c_double * 1)(0.0), (C.c_double * 1)(1.0), C.c_double(1.0), C.c_double(0.9), 3)),
    "replay": lambda s, U, p: s._check(s.L.mbm_replay(s.ctx, (C.c_double * 1)(1e-4), 1, None)),
}


@pytest.mark.parametrize("what", sorted(CALLS))
def test_refused_under_capture(what):
    import torch
    rt, st = _runtime(), torch.cuda.Stream()
    d = bf.Deck(Kn=0.02, limiter=4)
    d.blocks = [bf.Block(1, 0.0, 1.0, 0.0, 1.0, 20, 18, (0, 0, 0, 0))]
    blk, scn = d.blocks[0], sc.Scenario.seeded_quadrant(1)
    U = sc.initial_block(scn, blk)
    payload = np.ones(((blk.nx + 2) * (blk.ny + 2), 10))
    with sv.Solver(d, scn, stream=st.cuda_stream) as s:
        s.initialise()
        before = s.download(0, 0)
        assert rt.cudaStreamBeginCapture(C.c_void_p(st.cuda_stream), 2) == 0        # relaxed
        try:
            with pytest.raises(_abi.MBMError):
                CALLS[what](s, U, payload)
        finally:
            g = C.c_void_p()
            ended = rt.cudaStreamEndCapture(C.c_void_p(st.cuda_stream), C.byref(g))
        assert ended == 0
        rt.cudaGraphDestroy(g)
        H.assert_bitwise(s.download(0, 0), before, "layer")
        t, n, _ = s.steps(0.0, 1.0, max_steps=2)
        assert n == 2 and t > 0
