"""Performance cases: the calls a program makes of this framework, over the sizes
it is used at.

A case is a dict of plain values; its "kind" says which call it times:

* host_step   one leapfrog step on host-resident page-locked state
              (qz_step_host): what a main loop that keeps its particles on the
              host pays per step.
* run         `steps` leapfrog steps on device-resident state (qz_step, with a
              fixed dt or, cfl = 1, the CFL step before every step), then the
              state read back into page-locked arrays: a run between two outputs.
* ensemble    one step of independent members of mixed sizes (qz_ensemble_step),
              then all their states read back.
* vjp         the pull-back of an accelerations' adjoint through one force
              evaluation (qz_force_vjp): a backward pass through one step.
* gradient    the gradient of a final-state loss through `steps` steps with
              checkpoints (qz_adjoint_final_loss) on a frozen refinement tree.
* energies    kinetic and exact pair potential energy and momentum
              (qz_observables), taken at every output.

Initial conditions are the Plummer spheres of quantizer_b200.ics or a merger of
two Hernquist spheres in its geometry; dt is 1e-3 of the crossing time.
"""
import ctypes
import math
import random

import numpy as np
import torch

from quantizer_b200 import core, ics

STATE = ("x", "y", "z", "vx", "vy", "vz", "ax", "ay", "az")
VJP = ("gx", "gy", "gz", "gm")
GRAD = ("gx", "gy", "gz", "gvx", "gvy", "gvz", "gm", "loss")


def listed():
    return [
        # the smallest call: a small sphere on a 32^3 head, stepped from a host main loop
        dict(name="small_head32", kind="host_step", n=10000, a=0.05, lmin=5, levels=0, ref=4,
             bdry=1, stencil=0, mixed=0),
        # periodic box with the 5-point force stencil, an odd particle count, head only
        dict(name="periodic_head64", kind="run", n=100003, a=0.05, lmin=6, levels=0, ref=4,
             bdry=0, stencil=1, mixed=0, steps=10, cfl=0),
        # no refinement, a large head: 128^3
        dict(name="head128", kind="run", n=262144, a=0.04, lmin=7, levels=0, ref=4, bdry=1,
             stencil=0, mixed=0, steps=10, cfl=0),
        # a middle-sized refined run at the CFL step, ragged particle count
        dict(name="sphere200k_amr2_cfl", kind="run", n=200003, a=0.05, lmin=6, levels=2, ref=9,
             bdry=1, stencil=0, mixed=0, steps=5, cfl=1),
        # the main workload: a million particles, 128^3 head, three levels, FP64, host main loop
        dict(name="sphere1m_amr3_host", kind="host_step", n=1048576, a=0.02, lmin=7, levels=3,
             ref=9, bdry=1, stencil=0, mixed=0),
        # the same sphere in the mixed-precision form, device-resident between outputs
        dict(name="sphere1m_amr3_mixed", kind="run", n=1048576, a=0.02, lmin=7, levels=3, ref=9,
             bdry=1, stencil=0, mixed=1, steps=5, cfl=0),
        # the largest: two colliding spheres, 4.2 million particles, 256^3 head, four levels
        dict(name="merger4m_amr4_host", kind="host_step", n=4194304, a=0.03, lmin=8, levels=4,
             ref=9, bdry=1, stencil=0, mixed=0, merger=1),
        # many small systems side by side
        dict(name="ensemble24", kind="ensemble", members=24, nmin=2048, nmax=65536, levels=2,
             ref=9, mixed=1, threads=16),
        # backward through one force evaluation, head only
        dict(name="vjp_head128", kind="vjp", n=262144, a=0.04, lmin=7),
        # a training step of the initial state through a short refined trajectory
        dict(name="gradient_amr2", kind="gradient", n=262144, a=0.04, lmin=7, levels=2, ref=9,
             steps=4, every=2),
        # the output stage's exact energies
        dict(name="energies65k", kind="energies", n=65536, a=0.05, lmin=6),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("head", "head", "refined", "refined", "refined", "ensemble", "vjp",
                       "gradient", "energies"))
    a = round(rng.uniform(0.02, 0.08), 4)
    if kind == "head":
        c = dict(n=_log(rng, 2048, 400000), a=a, lmin=rng.choice((4, 5, 6, 7)), levels=0, ref=4,
                 bdry=rng.choice((0, 1, 1)), stencil=rng.choice((0, 0, 1)),
                 mixed=rng.choice((0, 0, 1)))
        if rng.random() < 0.5:
            return dict(kind="host_step", **c)
        return dict(kind="run", steps=rng.randint(2, 10), cfl=0, **c)
    if kind == "refined":
        c = dict(n=_log(rng, 8000, 1200000), a=a, lmin=rng.choice((5, 6, 7)),
                 levels=rng.choice((1, 2, 3)), ref=9, bdry=1, stencil=rng.choice((0, 0, 0, 1)),
                 mixed=rng.choice((0, 0, 1)))
        if rng.random() < 0.5:
            return dict(kind="host_step", **c)
        return dict(kind="run", steps=rng.randint(1, 4), cfl=rng.choice((0, 0, 1)), **c)
    if kind == "ensemble":
        return dict(kind="ensemble", members=rng.randint(3, 24), nmin=2048,
                    nmax=_log(rng, 8192, 65536), levels=rng.choice((0, 1, 2)), ref=9,
                    mixed=rng.choice((0, 1)), threads=rng.choice((4, 8, 16)))
    if kind == "vjp":
        return dict(kind="vjp", n=_log(rng, 4096, 400000), a=a, lmin=rng.choice((5, 6, 7)))
    if kind == "gradient":
        return dict(kind="gradient", n=_log(rng, 16384, 300000), a=a, lmin=rng.choice((5, 6, 7)),
                    levels=rng.choice((0, 1, 2)), ref=9, steps=rng.randint(2, 4),
                    every=rng.choice((1, 2)))
    return dict(kind="energies", n=_log(rng, 2048, 100000), a=a, lmin=rng.choice((5, 6)))


# -- inputs -----------------------------------------------------------------------------

def _pinned(n):
    return torch.empty(n, dtype=torch.float64, pin_memory=True).numpy()


def _ptr(a):
    return a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))


def _merger(n_each, a, seed, rmax=0.14, sep=0.3):
    """Two Hernquist spheres truncated at rmax, sep apart on x, approaching at half the
    mutual escape speed (the geometry of ics.merger); speeds inside a sphere are the
    Plummer fractions q of the local escape speed, q^2 (1 - q^2)^(7/2), which are drawn in
    a fraction of the time of the Hernquist distribution function's rejection."""
    rng = np.random.default_rng(seed)
    parts = []
    for side in (-1.0, 1.0):
        su = np.sqrt(rng.uniform(0.0, (rmax / (rmax + a)) ** 2, n_each))
        r = a * su / (1.0 - su)
        q = np.empty(0)
        while q.size < n_each:
            t, y = rng.uniform(0.0, 1.0, 3 * n_each), rng.uniform(0.0, 0.1, 3 * n_each)
            q = np.concatenate([q, t[y < t * t * (1.0 - t * t) ** 3.5]])
        v = q[:n_each] * np.sqrt(2.0 / (r + a))
        cols = []
        for length in (r, v):
            ct, ph = rng.uniform(-1.0, 1.0, n_each), rng.uniform(0.0, 2.0 * math.pi, n_each)
            st = np.sqrt(1.0 - ct * ct)
            cols += [length * st * np.cos(ph), length * st * np.sin(ph), length * ct]
        cols[0] += 0.5 + side * sep / 2
        cols[1] += 0.5
        cols[2] += 0.5
        cols[3] -= side * 0.25 * math.sqrt(4.0 / sep)
        parts.append(cols)
    ic = {k: np.concatenate([p[i] for p in parts]) for i, k in enumerate(STATE[:6])}
    ic["m"] = np.full(2 * n_each, 1.0 / n_each)
    return ic


def _ic(case, seed):
    if case.get("merger"):
        return _merger(case["n"] // 2, case["a"], seed)
    return ics.plummer(case["n"], a=case["a"], seed=seed)


def _dt(case):
    return 1e-3 * ics.crossing_time(case["a"])


def _members(case, seed):
    """(n, a, head level) of each ensemble member: n log-uniform, head 32^3 below 16384
    particles, else 64^3.  The sizes are the case's, the particles the seed's."""
    rng = random.Random(case["members"] * 1000003 + case["nmax"])
    out = []
    for _ in range(case["members"]):
        n = _log(rng, case["nmin"], case["nmax"])
        out.append((n, rng.uniform(0.02, 0.08), 5 if n < 16384 else 6))
    return out


def _sim(case, ic):
    return core.Simulation(ic, case["lmin"], lmax=case["lmin"] + case["levels"],
                           ref_ptcl=case["ref"], bdry=case["bdry"],
                           force_stencil=case["stencil"], precision=case["mixed"])


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind == "ensemble":
        st["sims"], st["dts"], total = [], [], 0
        for k, (n, a, lmin) in enumerate(_members(case, seed)):
            s = core.Simulation(ics.plummer(n, a=a, seed=1000 * (seed % 100000) + k), lmin,
                                lmax=lmin + case["levels"], ref_ptcl=case["ref"],
                                precision=case["mixed"], cg_chunk_min=2048)
            s.init_forces()
            st["sims"].append(s)
            st["dts"].append(1e-3 * ics.crossing_time(a))
            total += n
        st["out"] = {k: _pinned(total) for k in STATE}
        at = np.cumsum([0] + [s.n for s in st["sims"]])
        st["ptrs"] = [[_ptr(st["out"][k][at[i]:at[i + 1]]) for k in STATE]
                      for i in range(len(st["sims"]))]
        return st
    ic = _ic(case, seed)
    if kind in ("host_step", "run"):
        sim = st["sim"] = _sim(case, ic)
        sim.init_forces()
        st["out"] = {k: _pinned(case["n"]) for k in STATE}
        if kind == "host_step":
            st["out"]["m"] = _pinned(case["n"])
            st["out"]["m"][:] = ic["m"]
        st["ptrs"] = [_ptr(st["out"][k]) for k in STATE]
        core._check(sim.lib.qz_get_particles(sim.h, *st["ptrs"]))
        st["dt"] = _dt(case)
        return st
    rng = np.random.default_rng(seed)
    if kind == "energies":
        st["sim"] = core.Simulation(ic, case["lmin"])
        st["sim"].init_forces()
        return st
    tight = dict(tol=1e-11, tol2=1e-11, adjoint_tol=1e-11)
    if kind == "vjp":
        st["sim"] = core.Simulation(ic, case["lmin"], **tight)
        st["sim"].init_forces()
        st["abar"] = [rng.normal(0.0, 1.0, case["n"]) for _ in range(3)]
        return st
    if case["levels"] > 0:
        tight.update(lmax=case["lmin"] + case["levels"], ref_ptcl=case["ref"], freeze_tree=1)
    st["sim"] = core.Simulation(ic, case["lmin"], **tight)
    st["sim"].init_forces()
    st["targets"] = {k: ic[k] + rng.normal(0.0, 1e-3, case["n"]) for k in ("x", "y", "z")}
    st["dt"] = _dt(case)
    return st


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "host_step":
        state["sim"].step_host(state["out"], state["dt"])
        return {k: state["out"][k] for k in STATE}
    if kind == "run":
        sim = state["sim"]
        sim.step(0.0 if case["cfl"] else state["dt"], case["steps"])
        core._check(sim.lib.qz_get_particles(sim.h, *state["ptrs"]))
        return state["out"]
    if kind == "ensemble":
        core.ensemble_step(state["sims"], state["dts"], 1, threads=case["threads"])
        for s, p in zip(state["sims"], state["ptrs"]):
            core._check(s.lib.qz_get_particles(s.h, *p))
        return state["out"]
    if kind == "vjp":
        return state["sim"].force_vjp(*state["abar"])
    if kind == "gradient":
        g = state["sim"].adjoint_final_loss(case["steps"], state["dt"], state["targets"],
                                            checkpoint_every=case["every"])
        return {k: g[k] for k in GRAD}
    e = state["sim"].observables(0)
    return {k: e[k] for k in ("kinetic", "potential", "total", "momentum")}


def work(case):
    """State in (x, v, a, m) and out (x, v, a) once per force evaluation, the head grid's
    unknowns, and the arithmetic of the particle stages and of one pass over the grid."""
    kind = case["kind"]
    if kind == "ensemble":
        n = sum(m[0] for m in _members(case, 0))
        return {"bytes": 152.0 * n, "flops": 400.0 * n}
    n = case["n"]
    if kind == "energies":
        return {"bytes": 56.0 * n, "flops": 10.0 * n * (n - 1) / 2}
    g = float(2 ** case["lmin"]) ** 3
    if kind == "vjp":
        return {"bytes": 88.0 * n + 24.0 * g, "flops": 600.0 * n + 60.0 * g}
    evals = case.get("steps", 1)
    if kind == "gradient":
        evals *= 2
    return {"bytes": evals * (152.0 * n + 24.0 * g), "flops": evals * (400.0 * n + 60.0 * g)}


# -- 64-bit answers of the head-only cases, by a direct solve ----------------------------

def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


class _Head:
    """Force on every particle of the head-only path (deposit, Poisson solve with the
    analytic -GM/r shell, 3-point gradient, gather) with the discrete Poisson problem
    solved directly by sine transforms, in FP64."""

    def __init__(self, lmin, dev):
        self.nc = nc = 2 ** lmin
        self.H = 1.0 / nc
        k = torch.arange(1, nc, dtype=torch.float64, device=dev)
        self.S = torch.sin(math.pi * k[:, None] * k[None, :] / nc) * math.sqrt(2.0 / nc)
        lam = -4.0 * torch.sin(math.pi * k / (2 * nc)) ** 2
        self.lam = lam[:, None, None] + lam[None, :, None] + lam[None, None, :]
        c = torch.arange(nc + 1, dtype=torch.float64, device=dev) * self.H - 0.5
        self.c = c
        z, y, x = torch.meshgrid(c, c, c, indexing="ij")
        r = torch.sqrt(x * x + y * y + z * z)
        r[nc // 2, nc // 2, nc // 2] = 1.0
        shell = torch.ones_like(r, dtype=torch.bool)
        shell[1:-1, 1:-1, 1:-1] = False
        self.pot1 = torch.where(shell, -1.0 / r, torch.zeros_like(r))
        self.acc1 = [torch.where(shell, -q / r ** 3, torch.zeros_like(r)) for q in (x, y, z)]

    def _dst(self, f):
        for _ in range(3):
            f = torch.tensordot(f, self.S, dims=([0], [0]))
        return f

    def force(self, pos, m):
        nc, n1 = self.nc, self.nc + 1
        M = m.sum()
        p = [q * nc for q in pos]
        i0 = [torch.clamp(torch.floor(q.detach()), 0, nc - 1) for q in p]
        w = [(1.0 - (q - i), q - i) for q, i in zip(p, i0)]
        base = (i0[0] + n1 * i0[1] + n1 * n1 * i0[2]).long()
        corners = [(base + (i + n1 * j + n1 * n1 * k), w[0][i] * w[1][j] * w[2][k])
                   for k in (0, 1) for j in (0, 1) for i in (0, 1)]
        rho = torch.zeros(n1 ** 3, dtype=torch.float64, device=m.device)
        for g, ww in corners:
            rho = rho.index_add(0, g, m * ww)
        rho = rho.view(n1, n1, n1) * (4.0 * math.pi / self.H ** 3)
        b = self.pot1 * M
        rhs = self.H ** 2 * rho[1:-1, 1:-1, 1:-1] - (
            b[2:, 1:-1, 1:-1] + b[:-2, 1:-1, 1:-1] + b[1:-1, 2:, 1:-1] + b[1:-1, :-2, 1:-1] +
            b[1:-1, 1:-1, 2:] + b[1:-1, 1:-1, :-2])
        phi = b + torch.nn.functional.pad(self._dst(self._dst(rhs) / self.lam), (1,) * 6)
        acc = []
        for ax, a1 in zip((2, 1, 0), self.acc1):
            d = (phi.narrow(ax, 0, nc - 1) - phi.narrow(ax, 2, nc - 1)) / (2.0 * self.H)
            for other in (0, 1, 2):
                if other != ax:
                    d = d.narrow(other, 1, nc - 1)
            ga = (a1 * M + torch.nn.functional.pad(d, (1,) * 6)).reshape(-1)
            acc.append(sum(ga[g] * ww for g, ww in corners))
        return acc


def exact(case, seed):
    kind = case["kind"]
    dev = _device()
    if kind == "energies":
        ic = _ic(case, seed)
        x, y, z, vx, vy, vz, m = [torch.as_tensor(ic[k], device=dev) for k in
                                  ("x", "y", "z", "vx", "vy", "vz", "m")]
        kin = 0.5 * (m * (vx * vx + vy * vy + vz * vz)).sum()
        pot = torch.zeros((), dtype=torch.float64, device=dev)
        n = x.numel()
        for a in range(0, n, 2048):
            s = slice(a, min(n, a + 2048))
            r2 = ((x[s, None] - x[None, :]) ** 2 + (y[s, None] - y[None, :]) ** 2 +
                  (z[s, None] - z[None, :]) ** 2)
            q = torch.arange(a, s.stop, device=dev)
            r2[q - a, q] = math.inf
            pot -= 0.5 * (m[s, None] * m[None, :] / torch.sqrt(r2)).sum()
        mom = torch.stack([(m * v).sum() for v in (vx, vy, vz)])
        return {"kinetic": np.float64(kin.item()), "potential": np.float64(pot.item()),
                "total": np.float64((kin + pot).item()), "momentum": mom.cpu().numpy()}
    head = case.get("levels", 0) == 0 and case.get("bdry", 1) == 1 and not case.get("stencil", 0)
    if kind not in ("host_step", "run", "vjp") or not head:
        return None
    ic = _ic(case, seed)
    t = {k: torch.as_tensor(ic[k], device=dev) for k in ic}
    H = _Head(case["lmin"], dev)
    pos, m = [t[k] for k in ("x", "y", "z")], t["m"]
    if kind == "vjp":
        rng = np.random.default_rng(seed)
        abar = [torch.as_tensor(rng.normal(0.0, 1.0, case["n"]), device=dev) for _ in range(3)]
        leaf = [v.clone().requires_grad_(True) for v in pos + [m]]
        loss = sum((f * b).sum() for f, b in zip(H.force(leaf[:3], leaf[3]), abar))
        return {k: g.cpu().numpy() for k, g in zip(VJP, torch.autograd.grad(loss, leaf))}
    if case.get("cfl"):
        return None
    dt, vel = _dt(case), [t[k] for k in ("vx", "vy", "vz")]
    acc = H.force(pos, m)
    for _ in range(case.get("steps", 1)):
        vel = [v + a * dt * 0.5 for v, a in zip(vel, acc)]
        pos = [x + v * dt for x, v in zip(pos, vel)]
        for c in range(3):
            out = (pos[c] < 0.0) | (pos[c] >= 1.0)
            back = torch.where(pos[c] >= 1.0, 2.0 - pos[c], -pos[c])
            pos[c] = torch.where(out, back, pos[c])
            vel[c] = torch.where(out, -vel[c], vel[c])
        acc = H.force(pos, m)
        vel = [v + a * dt * 0.5 for v, a in zip(vel, acc)]
    return {k: v.cpu().numpy() for k, v in zip(STATE, pos + vel + acc)}
