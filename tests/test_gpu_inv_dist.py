"""GPU: the pair energy's reciprocal distance 1 / sqrt(d) over the whole exponent range.

Bar, relative to the exact value: in [2^-960, 2^960] the hardware's approximation y (error
below 2^-19, so e = 1 - d y^2 is below 2^-18) is followed by y (1 + e / 2 + 3 e^2 / 8), whose
truncation is 5 e^3 / 16 < 2^-55; the rounding of d y moves e by 2^-53, which counts half; the
last operation rounds by 2^-53: together below 2^-52.  Outside that range a square root and a
division round by 2^-53 each, the root's error counting once: 2^-52.  Zeros, infinities and
NaN are a division's."""
import numpy as np
import pytest

from quantizer_b200 import core, ics

pytestmark = pytest.mark.gpu


def _inv(d):
    d = np.ascontiguousarray(d, dtype=np.float64)
    out = np.empty_like(d)
    with core.Simulation(ics.plummer(10, a=0.05, seed=1), 3) as sim:
        core._check(sim.lib.qz_test_inv_dist(sim.h, core._p(d), core._p(out), d.size))
    return out


def test_every_exponent():
    rng = np.random.default_rng(3)
    e = np.repeat(np.arange(-1022, 1024), 64)
    d = np.ldexp(rng.uniform(1.0, 2.0, e.size), e)
    for g in (2.0 ** -960, 2.0 ** 960, 2.0 ** -961, 2.0 ** 961, 1.0, 4.0):
        d = np.concatenate([d, [np.nextafter(g, 0.0), g, np.nextafter(g, np.inf)]])
    d = np.concatenate([d, np.ldexp(1.0, np.arange(-1074, -1022)), [np.finfo(float).max]])
    want = 1 / np.sqrt(d.astype(np.longdouble))
    assert np.finfo(np.longdouble).nmant >= 63
    err = np.abs(_inv(d).astype(np.longdouble) - want) / want
    assert err.max() <= np.longdouble(2.0) ** -52, d[np.argmax(err)]


def test_special_values():
    got = _inv([0.0, -0.0, np.inf, np.nan, -1.0, -np.inf])
    assert got[0] == np.inf and got[1] == -np.inf and got[2] == 0.0
    assert np.isnan(got[3:]).all()
