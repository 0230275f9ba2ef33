"""The adjoint's gather as a march of warps up 28-column strips (the default) against the whole
cell pass, which gathers a thread per cell (MBM_ADJ_SPLIT=0): the same gradient at block sizes
on and beside the edges of the strips and of the 16-row segments, with wall and open edges and an
interface, for every limiter.  A cell's terms are the same in both and are added in another order, so the
gradients differ by roundings: 2^-53 of the largest entry, a few hundred terms and steps deep,
with the cancellation of the reverse sweep on top -- 1e-12 of it, the bound that the split of
the cell pass is held to elsewhere."""
import os

import numpy as np
import pytest

from multiblockmomentsfv_b200 import adjoint as adj
from multiblockmomentsfv_b200 import blockfile as bf

pytestmark = pytest.mark.gpu


# nx + 2 columns in strips of 28, ny + 2 rows in segments of 16
@pytest.mark.parametrize("nx,ny,limiter", [(3, 3, 4), (26, 14, 4), (27, 15, 3), (25, 13, 2), (54, 30, 1),
                                           (55, 31, 4), (61, 47, 0)])
def test_gather_equals_cell_pass(nx, ny, limiter):
    d = bf.Deck(Kn=0.02, R13=1.0, F=0.1, limiter=limiter, CFL=0.95)
    d.blocks = [bf.Block(1, -1.0, 0.0, -0.5, 0.5, nx, ny, (0, 2, -1, 0)),
                bf.Block(2, 0.0, 1.0, -0.5, 0.5, nx + 3, ny, (1, 0, 0, -1))]
    base = adj.smooth_base(d, 31)
    rng = np.random.default_rng(31)
    th0 = [1.0 + 0.2 * np.sin(np.linspace(0, 3, b.nx)[None, :] + np.linspace(0, 2, b.ny)[:, None])
           * rng.uniform(0.5, 1.0) for b in d.blocks]
    layers = adj.state_from_theta(d, base, th0)
    out = {}
    for split in ("1", "0"):
        os.environ["MBM_ADJ_SPLIT"] = split
        try:
            with adj.Sensitivity(d, base) as S:
                S.load(layers)
                J, g, gK, dts, ms = S.run(6, 4)
                out[split] = (J, np.concatenate([x.ravel() for x in g]), gK)
        finally:
            del os.environ["MBM_ADJ_SPLIT"]
    (J1, g1, k1), (J0, g0, k0) = out["1"], out["0"]
    assert J1 == J0
    scale = np.abs(g0).max()
    assert scale > 0 and np.isfinite(g0).all()
    assert np.abs(g1 - g0).max() <= 1e-12 * scale, np.abs(g1 - g0).max() / scale
    assert abs(k1 - k0) <= 1e-12 * abs(k0)
