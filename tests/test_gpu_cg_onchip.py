"""GPU: the node conjugate gradient with its vectors on chip (cg_variant 0) against
the kernels that keep them in device memory (cg_variant 2: the same iterates by the
pipelined arrangement), on node shapes where the on-chip layout has its edges: single
points, rows of one to nine points at every alignment, chunk remainders, one block and
many, the sizes at which a block's threads and rows a thread change, random masks (most
neighbours in other blocks, ghost rows past the shared memory) and ghost rows forced
into device memory.

Both stop at |r| <= tol rm sqrt(n), so their potentials differ by at most the operator's
inverse times that: |A^-1| <= 1 / (3 pi^2) box units, times 2 tol rm; with tol = 1e-12
and |d| of the order of rm the potentials agree to 1e-11 of their scale; the bar
is 1e-10, and the iteration counts may differ by one check interval."""
import ctypes as C

import numpy as np
import pytest

from quantizer_b200 import core, ics

pytestmark = pytest.mark.gpu

P = C.POINTER(C.c_double)


def _box(nx, ny, nz, at=(1, 1, 1), pad=(1, 1, 1)):
    m = np.zeros((nz + at[2] + pad[2], ny + at[1] + pad[1], nx + at[0] + pad[0]), dtype=bool)
    m[at[2]:at[2] + nz, at[1]:at[1] + ny, at[0]:at[0] + nx] = True
    return m


def _random(n, p, seed):
    rng = np.random.default_rng(seed)
    m = np.zeros((n + 2,) * 3, dtype=bool)
    m[1:-1, 1:-1, 1:-1] = rng.random((n, n, n)) < p
    return m


SHAPES = {
    **{f"row{k}": _box(k, 1, 1, at=(1 + k % 4, 2, 1)) for k in (2, 3, 4, 5, 9)},
    "column": _box(1, 1, 33),
    "odd": _box(7, 5, 3, at=(3, 1, 2)),
    "rows127": _box(4, 127, 1, at=(4, 1, 1)),
    "rows129": _box(4, 43, 3, at=(4, 1, 1)),
    "cube20": _box(20, 20, 20, at=(2, 3, 1)),
    "slab": _box(90, 60, 5),
    "random": _random(40, 0.5, 3),
    "sparse": _random(48, 0.15, 4),
    "cube67": _box(67, 67, 67),     # 608 threads of one row
    "cube76": _box(76, 76, 75),     # two rows a thread
    "cube90": _box(91, 89, 90),     # the most rows a block
}


def _solve(mask, variant, ghosts=0):
    nz, ny, nx = mask.shape
    intr = np.flatnonzero(mask.ravel()).astype(np.int32)
    rng = np.random.default_rng(7)
    d = rng.normal(0.0, 4.0 * np.pi, mask.size)
    pot = rng.normal(0.0, 1e-4, mask.size) + 1e-2
    old = pot.copy()
    H3 = (1.0 / 2 ** 6) ** 3
    with core.Simulation(ics.plummer(100, a=0.05, seed=1), 4, cg_variant=variant, tol=1e-12,
                         tol2=1e-9) as sim:
        core._check(sim.lib.qz_test_cg_ghosts(sim.h, ghosts))
        core._check(sim.lib.qz_node_conjugate_gradient(
            sim.h, 6, nx - 1, ny - 1, nz - 1, intr.size, intr.ctypes.data_as(C.POINTER(C.c_int)),
            H3 * intr.size, intr.size, d.ctypes.data_as(P), pot.ctypes.data_as(P),
            old.ctypes.data_as(P)))
        return pot, old, sim.stats().cg_iterations


@pytest.mark.parametrize("name", sorted(SHAPES))
def test_on_chip_equals_in_memory(name):
    mask = SHAPES[name]
    a, ao, ia = _solve(mask, 0)
    b, bo, ib = _solve(mask, 2)
    scale = np.abs(b).max()
    assert abs(ia - ib) <= 5
    assert np.abs(a - b).max() <= 1e-10 * scale
    if ia == ib:
        assert np.abs(ao - bo).max() <= 1e-8 * scale  # pot at the last failed check


def test_single_point():
    # (the in-memory pipelined form divides 0 by 0 after the first iteration)
    mask = _box(1, 1, 1)
    a, _, _ = _solve(mask, 0)
    rng = np.random.default_rng(7)
    d = rng.normal(0.0, 4.0 * np.pi, mask.size).reshape(mask.shape)
    p0 = rng.normal(0.0, 1e-4, mask.size).reshape(mask.shape) + 1e-2
    nbr = p0[0, 1, 1] + p0[2, 1, 1] + p0[1, 0, 1] + p0[1, 2, 1] + p0[1, 1, 0] + p0[1, 1, 2]
    want = (nbr - d[1, 1, 1] / 2.0 ** 12) / 6.0
    assert abs(a.reshape(mask.shape)[1, 1, 1] - want) <= 1e-10 * abs(want)


@pytest.mark.parametrize("name", ["cube20", "random", "cube76"])
def test_ghost_rows_in_device_memory_change_nothing(name):
    a, ao, ia = _solve(SHAPES[name], 0)
    b, bo, ib = _solve(SHAPES[name], 0, ghosts=16)
    assert ia == ib
    np.testing.assert_array_equal(a, b)
    np.testing.assert_array_equal(ao, bo)


def test_points_on_the_faces_are_solved_in_memory():
    m = np.ones((6, 6, 6), dtype=bool)
    m[0] = m[-1] = m[:, 0] = m[:, -1] = False  # x faces stay
    m[:, :, 1:-1] = False
    m[2:4, 2:4, :] = True
    a, _, ia = _solve(m, 0)
    b, _, ib = _solve(m, 2)
    assert abs(ia - ib) <= 5
    assert np.abs(a - b).max() <= 1e-10 * np.abs(b).max()
