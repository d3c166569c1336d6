"""GPU: the exact pair potential energy against a 64-bit sum on the host, at the edges of its
256-particle tiles, and for coincident and very distant particles.

Every term is exact to a few units in the last place and the terms have one sign, so the
sum's relative error is at most about (terms a thread adds in a row) eps = 256 * 2.2e-16;
the bar is 1e-12 as for the sums against the reference."""
import numpy as np
import pytest

from quantizer_b200 import core, ics

pytestmark = pytest.mark.gpu


def _energy(ic, lmin=3):
    with core.Simulation(ic, lmin) as sim:
        return sim.observables(0)["potential"]


def _exact(ic):
    x = np.stack([ic[k] for k in "xyz"]).astype(np.longdouble)
    m = ic["m"].astype(np.longdouble)
    tot = np.longdouble(0)
    for i in range(1, m.size):
        d = x[:, :i] - x[:, i:i + 1]
        tot += m[i] * (m[:i] / np.sqrt((d * d).sum(axis=0))).sum()
    return float(-tot)


@pytest.mark.parametrize("n", [1, 2, 127, 128, 129, 255, 256, 257, 511, 512, 513, 3000])
def test_pair_energy_at_tile_edges(n):
    ic = ics.plummer(n, a=0.05, seed=n)
    ic["m"] = np.random.default_rng(n).uniform(0.1, 1.0, n)
    want = _exact(ic)
    assert abs(_energy(ic) - want) <= 1e-12 * abs(want)


def test_pair_energy_of_extreme_distances():
    ic = ics.plummer(64, a=0.05, seed=3)
    ic["x"][10] = ic["x"][9] + 2e-16
    ic["y"][10], ic["z"][10] = ic["y"][9], ic["z"][9]
    want = _exact(ic)
    assert abs(_energy(ic) - want) <= 1e-12 * abs(want)
    ic["x"][10] = ic["x"][9]  # coincident: the reference divides by zero
    assert _energy(ic) == -np.inf
