"""GPU: the on-chip node conjugate gradient in units far from one.  Every operation of the
solve is linear in the density, the potential and the node's mass, or a quotient, so a problem
scaled by a power of two gives the scaled potential bit for bit and the same iterations, as
long as r.r itself (here 2^-640 to 2^640 and its 10^-24 at the end) is in range."""
import ctypes as C

import numpy as np
import pytest

from quantizer_b200 import core, ics

pytestmark = pytest.mark.gpu

P = C.POINTER(C.c_double)


def _solve(n, scale):
    mask = np.zeros((n + 2,) * 3, dtype=bool)
    mask[1:-1, 1:-1, 1:-1] = True
    intr = np.flatnonzero(mask.ravel()).astype(np.int32)
    rng = np.random.default_rng(7)
    d = rng.normal(0.0, 4.0 * np.pi, mask.size) * scale
    pot = (rng.normal(0.0, 1e-4, mask.size) + 1e-2) * scale
    old = pot.copy()
    with core.Simulation(ics.plummer(100, a=0.05, seed=1), 4, tol=1e-12, tol2=1e-9) as sim:
        core._check(sim.lib.qz_node_conjugate_gradient(
            sim.h, 6, n + 1, n + 1, n + 1, intr.size, intr.ctypes.data_as(C.POINTER(C.c_int)),
            scale * intr.size / 2.0 ** 18, intr.size, d.ctypes.data_as(P), pot.ctypes.data_as(P),
            old.ctypes.data_as(P)))
        return pot, sim.stats().cg_iterations


@pytest.mark.parametrize("n", [5, 30])  # one block, and many
@pytest.mark.parametrize("e", [-320, -250, 250, 320])
def test_scaled_problem_scales_the_solution(n, e):
    a, ia = _solve(n, 1.0)
    b, ib = _solve(n, 2.0 ** e)
    assert ia == ib
    np.testing.assert_array_equal(b, a * 2.0 ** e)
