"""GPU: the on-chip conjugate gradient on levels of several nodes, against the two-reduction
kernel in device memory (cg_variant 3): more one-chunk nodes than blocks (a block takes
several), nodes of different sizes in one round with one-chunk nodes beside them, nodes too
large to share a round, and launches across the wrap of the exchange's 31-bit tags.

Bar of a node: both kernels stop at |r| <= tol rm sqrt(n) (2-norms of the n interior points),
so their potentials differ by 2 tol rm sqrt(n) / lambda, lambda = (12 / H^2) sin^2(pi H / 2w)
the smallest eigenvalue on a cube of the node's largest width w; the residual that either
carries differs from its potential's by rounding, at most k 2^-53 (12 / H^2) max |pot| sqrt(n)
after k iterations, which the inverse turns into that over lambda, for each."""
import math

import numpy as np
import pytest

from quantizer_b200 import core

pytestmark = pytest.mark.gpu

TOL = 1e-10


def _cube(lo, size):
    g = np.arange(size)
    z, y, x = np.meshgrid(g, g, g, indexing="ij")
    return np.stack([x.ravel(), y.ravel(), z.ravel()], 1) + np.array(lo)


def _singles(cells, step):
    return np.array([(i, j, k) for k in range(2, cells - 2, step) for j in range(2, cells - 2, step)
                     for i in range(2, cells - 2, step)])


def _cells(name):
    """(head level, cells that hold one particle, and so are refined with their neighbours)"""
    if name == "many":  # 1,728 nodes of 125 points
        return 6, _singles(64, 5)
    if name == "mixed":
        big = np.concatenate([_cube((6, 6, 6), 12), _cube((30, 8, 8), 6), _cube((8, 30, 30), 9),
                              _cube((44, 44, 44), 2)])
        far = _singles(64, 6)
        d = np.abs(far[:, None, :] - big[None, :, :]).max(2).min(1)
        return 6, np.concatenate([big, far[d > 4][:60]])
    big = np.concatenate([_cube((10, 10, 10), 40), _cube((70, 70, 70), 40)])
    far = _singles(128, 15)
    d = np.minimum(np.abs(far - 30).max(1), np.abs(far - 90).max(1))
    return 7, np.concatenate([big, far[d > 26]])


def _solve(name, variant, tag=None):
    lmin, cells = _cells(name)
    n = len(cells)
    rng = np.random.default_rng(4)
    pos = (cells + rng.uniform(0.05, 0.95, (n, 3))) / 2.0 ** lmin
    ic = {k: np.ascontiguousarray(pos[:, q]) for q, k in enumerate("xyz")}
    ic.update({k: np.zeros(n) for k in ("vx", "vy", "vz")})
    ic["m"] = rng.uniform(0.5, 1.5, n) / n
    with core.Simulation(ic, lmin, lmax=lmin + 1, ref_ptcl=1, tol=TOL, cg_variant=variant) as sim:
        sim.init_forces()
        if tag is not None:
            if tag:
                core._check(sim.lib.qz_test_cg_tag(sim.h, tag))
            sim.init_forces()
        nodes = [(sim.node_info(1, q), sim.node_list(1, q, "intr"), sim.node_field(1, q, "pot"))
                 for q in range(sim.num_nodes(1))]
        return nodes, sim.stats().cg_iterations, sim.lib.qz_test_cg_scratch(sim.h), sim.cfg.G, lmin + 1


@pytest.mark.parametrize("name,least", [("many", 1000), ("mixed", 30), ("rounds", 100)])
def test_levels_of_several_nodes(name, least):
    got, ig, scratch, G, lv = _solve(name, 0)
    want, iw, _, _, _ = _solve(name, 3)
    assert len(got) == len(want) >= least
    if name == "many":
        assert scratch == 0  # one-chunk nodes exchange nothing
    H = 0.5 ** lv
    for (info, pts, a), (_, _, b) in zip(got, want):
        w = (max(q - p for p, q in zip(info["bmin"], info["bmax"])) + 1) * H
        lam = 12.0 / H ** 2 * math.sin(math.pi * H / (2.0 * w)) ** 2
        rm = 4.0 * math.pi * G * info["mass"] / (info["ncells"] * H ** 3)
        root, top = math.sqrt(len(pts)), np.abs(b[pts]).max()
        bar = 2.0 * TOL * rm * root / lam + (ig + iw) * 2.0 ** -53 * 12.0 / H ** 2 * top * root / lam
        assert np.abs(a[pts] - b[pts]).max() <= bar


def test_tags_wrap():
    """The tags start again, on cleared words, when the 31 bits run out: nothing changes."""
    want = _solve("mixed", 0, tag=0)
    got = _solve("mixed", 0, tag=2 ** 31 - 2)
    assert got[1] == want[1]
    for (_, _, a), (_, _, b) in zip(got[0], want[0]):
        np.testing.assert_array_equal(a, b)
