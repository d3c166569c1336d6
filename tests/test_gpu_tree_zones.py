"""GPU: the refinement tree and the levels' densities against a plain numpy construction,
on zone shapes at which the union-find, the ordered selections and the segment sums have
their edges: one cell, long chains that turn back (their parents lead far), staircases in
both directions, 1,728 small zones (of more cells than the sort has room for particles), one
large one, zones on the simulation's boundary, and particle numbers at the
edges of the sort's tiles and of the cells' segments.

The construction: a cell with ref_ptcl particles or more and its neighbours in the node
are refined; zones are 6-connected (scipy.ndimage.label); cells, nodes and point lists in
the order that qz_amr.cu states.  Whole numbers compare equal.  A density is a sum of K
products at most, K the particles of the node, added in another order on either side: the
two differ by less than (K + 8) 2^-52 of the sum of the products' absolute values, here
the density itself (every product is positive)."""
import numpy as np
import pytest
from scipy import ndimage

from quantizer_b200 import core

pytestmark = pytest.mark.gpu

REF = 3


def _snake():
    cells = []
    for z in range(4, 28, 6):
        for y in range(4, 28, 5):
            xs = list(range(4, 28))
            cells += [(x, y, z) for x in (xs if (y // 5) % 2 else xs[::-1])]
        cells += [(4 if (z // 6) % 2 else 27, 24, z + k) for k in range(6) if z + k < 28]
    return cells


def _seeds(name):
    rng = np.random.default_rng(11)
    if name == "one":
        return [(9, 14, 20)]
    if name == "many":  # 1,728 zones on a head of 64
        return [(4 * i + 2, 4 * j + 2, 4 * k + 2) for k in range(12) for j in range(12)
                for i in range(12)]
    if name == "corners":
        return [(0, 0, 0), (31, 31, 31), (0, 31, 16)]
    if name == "snake":
        return _snake()
    if name == "stairs":
        return [(k, k, k) for k in range(3, 14)] + [(28 - k, 3 + k, 18 + k // 2) for k in range(12)]
    if name == "ball":
        g = np.argwhere(((np.indices((32,) * 3) - 15.7) ** 2).sum(0) < 9.3 ** 2)
        return [tuple(c) for c in g]
    if name == "sparse":
        return [tuple(c) for c in rng.integers(0, 32, (60, 3))]
    return [tuple(c) for c in rng.integers(1, 31, (420, 3))]  # "dense": one ragged zone


def _particles(name, extra, cells):
    """REF particles in every seed cell, some of them close enough together to refine
    a level further; `extra` more in one cell (a long segment)."""
    rng = np.random.default_rng(5)
    pos = []
    for k, c in enumerate(dict.fromkeys(_seeds(name))):
        w = 0.5 if k % 3 == 0 else 1.0
        pos.append((np.array(c) + w * rng.uniform(0.02, 0.98, (REF, 3))) / cells)
    c = np.array(_seeds(name)[0])
    pos.append((c + rng.uniform(0.02, 0.98, (extra, 3))) / cells)
    pos = np.concatenate(pos)
    return pos[rng.permutation(len(pos))]


def _classify(inside):
    """Category of every grid point of a node box from its 8 cells (True: the node's)."""
    p = np.pad(inside, 1)
    v = {(a, b, c): p[1 - c:p.shape[0] - c, 1 - b:p.shape[1] - b, 1 - a:p.shape[2] - a]
         for a in (0, 1) for b in (0, 1) for c in (0, 1)}
    n = {k: ~w for k, w in v.items()}
    all_ = lambda *ks: np.logical_and.reduce([n[k] for k in ks])
    x4 = all_((1, 0, 0), (1, 1, 0), (1, 0, 1), (1, 1, 1))
    y4 = all_((0, 1, 0), (1, 1, 0), (0, 1, 1), (1, 1, 1))
    z4 = all_((0, 0, 1), (1, 0, 1), (0, 1, 1), (1, 1, 1))
    b0 = x4 | y4 | z4
    b1 = all_((0, 1, 0), (0, 0, 1), (0, 1, 1)) | y4 | z4
    b2 = all_((1, 1, 0), (1, 0, 1), (1, 1, 1)) | all_((0, 0, 1), (1, 0, 1)) | z4
    b3 = all_((0, 0, 1), (0, 1, 1)) | all_((0, 0, 1), (1, 0, 1)) | z4
    rest = v[0, 0, 1] | v[1, 0, 1] | v[0, 1, 1] | v[1, 1, 1]
    border = np.select([v[0, 0, 0], v[1, 0, 0], v[0, 1, 0], v[1, 1, 0]], [b0, b1, b2, b3], True)
    any_ = rest | v[0, 0, 0] | v[1, 0, 0] | v[0, 1, 0] | v[1, 1, 0]
    return np.where(any_, np.where(border, 2, 1), 0)


def _zones(cells, pos, lv):
    """Refined cells of one node (cells: its (n, 3) list in order): per zone, in the order
    of the zones' first cells, the indices of its cells."""
    lo = cells.min(0) - 1
    dim = cells.max(0) - lo + 2
    at = tuple((cells - lo).T)
    inside = np.zeros(dim, dtype=bool)
    inside[at] = True
    cnt = np.zeros(dim, dtype=int)
    c = np.floor(pos * (1 << lv)).astype(int) - lo
    np.add.at(cnt, tuple(c.T), 1)
    flag = ndimage.binary_dilation(inside & (cnt >= REF), np.ones((3, 3, 3))) & inside
    lab = ndimage.label(flag)[0][at]
    first = [k for k in dict.fromkeys(lab.tolist()) if k]
    return [np.flatnonzero(lab == k) for k in first]


CASES = [("one", 0), ("one", 253), ("one", 254), ("corners", 300), ("snake", 2), ("stairs", 2500),
         ("ball", 0), ("sparse", 3916), ("dense", 70), ("many", 0)]


@pytest.mark.parametrize("name,extra", CASES)
def test_tree_and_density(name, extra):
    lmin = 6 if name == "many" else 5
    pos = _particles(name, extra, 1 << lmin)
    n = len(pos)
    rng = np.random.default_rng(1)
    ic = {k: np.ascontiguousarray(pos[:, q]) for q, k in enumerate("xyz")}
    ic.update({k: np.zeros(n) for k in ("vx", "vy", "vz")})
    ic["m"] = rng.uniform(0.5, 1.5, n) / n
    seen = 0
    with core.Simulation(ic, lmin, lmax=lmin + 2, ref_ptcl=REF) as sim:
        sim.tree_adaptation()
        sim.grid_density()
        g = np.arange(1 << lmin)
        z, y, x = np.meshgrid(g, g, g, indexing="ij")
        nodes = [(np.stack([x.ravel(), y.ravel(), z.ravel()], 1), np.arange(n))]
        for level in (1, 2):
            lv, children = lmin + level, []
            for parent, (cells, ptcl) in enumerate(nodes):
                for zone in _zones(cells, pos[ptcl], lv - 1):
                    zc = cells[zone]
                    sub = np.array([(s & 1, s >> 1 & 1, s >> 2) for s in range(8)])
                    mine = (2 * zc[:, None, :] + sub[None]).reshape(-1, 3)
                    pc = np.floor(pos[ptcl] * (1 << (lv - 1))).astype(int)
                    place = 1 << 10 * np.arange(3)
                    here = np.isin(pc @ place, zc @ place)
                    children.append((mine, ptcl[here], parent))
            assert (sim.num_nodes(level) if level < sim.levels() else 0) == len(children)
            for q, (cells, ptcl, parent) in enumerate(children):
                info = sim.node_info(level, q)
                np.testing.assert_array_equal(sim.node_cells(level, q), cells)
                assert info["parent"] == parent and info["nptcl"] == len(ptcl)
                assert info["bmin"] == tuple(cells.min(0)) and info["bmax"] == tuple(cells.max(0))
                rd, ts = np.array(info["rd"]), np.array(info["ts"])
                inside = np.zeros(rd[::-1], dtype=bool)
                inside[tuple((cells - ts).T[::-1])] = True
                cat = _classify(inside)
                if info["contact"]:
                    kk, jj, ii = np.indices(cat.shape)
                    for c, o in ((ii, 0), (jj, 1), (kk, 2)):
                        wall = (c + ts[o] == 0) | (c + ts[o] == 1 << lv)
                        cat = np.where((cat >= 2) & wall, 3, cat)
                for w, c in (("intr", 1), ("bdry", 2), ("simb", 3)):
                    np.testing.assert_array_equal(sim.node_list(level, q, w),
                                                  np.flatnonzero(cat.ravel() == c))
                H = 1.0 / (1 << lv)
                d = np.zeros(cat.shape)
                f = np.floor(pos[ptcl] * (1 << lv)).astype(int)
                w1 = pos[ptcl] - H * f
                cm = 4.0 * np.pi * sim.cfg.G / H ** 6 * ic["m"][ptcl]
                for s in range(8):
                    o = np.array([s & 1, s >> 1 & 1, s >> 2])
                    w = np.where(o, w1, H - w1).prod(1) * cm
                    np.add.at(d, tuple((f + o - ts).T[::-1]), w)
                got = sim.node_field(level, q, "d").reshape(d.shape)
                k = len(ptcl) + 8
                assert (np.abs(got - d) <= k * 2.0 ** -52 * d).all()
                mass = ic["m"][ptcl].sum()
                assert abs(info["mass"] - mass) <= k * 2.0 ** -52 * mass
                seen += len(cells)
            nodes = [c[:2] for c in children]
    assert seen > 0
