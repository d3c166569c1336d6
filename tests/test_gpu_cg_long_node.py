"""GPU: a node longer than the on-chip order's brick coordinates hold (2^16 bricks of four
points) is solved from device memory (cg_variant 3), bit for bit.  Its two groups of points
lie 2^18 points apart, so that coordinates cut to 16 bits would make them one group."""
import ctypes as C

import numpy as np
import pytest

from quantizer_b200 import core, ics

pytestmark = pytest.mark.gpu

P = C.POINTER(C.c_double)


def _solve(variant, far):
    nx = far + 20
    mask = np.zeros((4, 4, nx), dtype=bool)
    mask[1:3, 1:3, 1:10] = mask[1:3, 1:3, far + 1:far + 10] = True
    intr = np.flatnonzero(mask.ravel()).astype(np.int32)
    rng = np.random.default_rng(7)
    d = rng.normal(0.0, 4.0 * np.pi, mask.size)
    pot = rng.normal(0.0, 1e-4, mask.size) + 1e-2
    old = pot.copy()
    with core.Simulation(ics.plummer(100, a=0.05, seed=1), 4, cg_variant=variant, tol=1e-12,
                         tol2=1e-9) as sim:
        core._check(sim.lib.qz_node_conjugate_gradient(
            sim.h, 6, nx - 1, 3, 3, intr.size, intr.ctypes.data_as(C.POINTER(C.c_int)),
            intr.size / 2.0 ** 18, intr.size, d.ctypes.data_as(P), pot.ctypes.data_as(P),
            old.ctypes.data_as(P)))
        return pot, old, sim.stats().cg_iterations


def test_a_node_longer_than_the_order_holds():
    a, b = _solve(0, 1 << 18), _solve(3, 1 << 18)
    assert a[2] == b[2] > 0
    for x, y in zip(a[:2], b[:2]):
        np.testing.assert_array_equal(x, y)


def test_the_longest_node_of_the_order():
    # |A^-1| <= 1 / (12 / H^2 sin^2(pi / 6)) on points two deep; both stop at |r| <= tol rm
    # sqrt(n), rm = 4 pi here: 2 tol 4 pi sqrt(72) H^2 / 3 and rounding, below 1e-10 of |pot|
    a, b = _solve(0, (1 << 18) - 40), _solve(3, (1 << 18) - 40)
    assert np.abs(a[0] - b[0]).max() <= 1e-10 * np.abs(b[0]).max()
