"""The bitwise kernels' divisions as they run (mbm_div.cuh, quotients and slopes of mbm_math.cuh)
against IEEE division, bit for bit: every quotient a correctly rounded one whatever its
operands, zeros' signs included."""
import numpy as np
import pytest

from multiblockmomentsfv_b200 import _abi

pytestmark = pytest.mark.gpu

N = 400_000


def _mag(rng, n, lo, hi):
    return np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(lo, hi + 1, n))


def _ones(rng, n, lo, hi):
    """Significands a few last places below 2."""
    return np.ldexp(2.0 - rng.integers(1, 4, n) * 2.0 ** -52, rng.integers(lo, hi + 1, n))


def _sign(rng, v):
    return v * rng.choice([-1.0, 1.0], len(v))


def _special(rng, n):
    return rng.choice([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -5e-324, 1e-310, 1.0, -1.0, 1e308,
                       np.ldexp(1.0, 481), np.nextafter(np.ldexp(1.0, 481), 0), np.ldexp(1.0, -480),
                       np.nextafter(np.ldexp(1.0, -480), 0), np.ldexp(1.0, 400), np.ldexp(1.0, -400), 1e-10], n)


SETS = {
    "everyday": lambda r: (_sign(r, _mag(r, N, -4, 4)), _mag(r, N, -8, 3)),
    "wide": lambda r: (_sign(r, _mag(r, N, -470, 470)), _mag(r, N, -470, 470)),
    "whole range": lambda r: (_sign(r, _mag(r, N, -1074, 1022)), _sign(r, _mag(r, N, -1074, 1022))),
    "zeros among others": lambda r: (np.where(r.random(N) < 0.5, r.choice([0.0, -0.0], N), _sign(r, _mag(r, N, -4, 4))),
                                     _mag(r, N, -30, 30)),
    "zeros": lambda r: (r.choice([0.0, -0.0], N), _mag(r, N, -470, 470)),
    "significands of all ones": lambda r: (_sign(r, _ones(r, N, -40, 40)), _ones(r, N, -40, 40)),
    "special": lambda r: (_special(r, N), _special(r, N)),
}


@pytest.mark.parametrize("what", sorted(SETS) + ["near ties"])
def test_divisions_are_ieee(what):
    import torch
    rng = np.random.default_rng(len(what))
    if what == "near ties":
        y = np.where(rng.random(N) < 0.3, _ones(rng, N, -20, 20), _mag(rng, N, -20, 20))
        x = _sign(rng, _mag(rng, N, -20, 20)) * y
        x = np.where(rng.random(N) < 0.5, np.nextafter(x, np.where(rng.random(N) < 0.5, np.inf, -np.inf)), x)
    else:
        x, y = SETS[what](rng)
    xd, yd = torch.tensor(x, device="cuda"), torch.tensor(y, device="cuda")
    out = torch.empty(3 * N, dtype=torch.float64, device="cuda")
    _abi.check(_abi.lib().mbm_division_check(xd.data_ptr(), yd.data_ptr(), N, out.data_ptr()))
    got = out.cpu().numpy().reshape(N, 3)
    with np.errstate(all="ignore"):
        d2 = np.roll(x, -1)
        w1, w2 = np.abs(x) + 1e-10, np.abs(d2) + 1e-10
        want = np.stack([x / y, x / y, (w1 * d2 + w2 * x) / (w1 + w2) / y], axis=1)
    nan = np.isnan(want)
    assert np.array_equal(np.isnan(got), nan)
    same = (got.view(np.int64) == want.view(np.int64)) | nan
    assert same.all(), (what, (~same).sum(axis=0), x[~same.all(axis=1)][:4], y[~same.all(axis=1)][:4])
