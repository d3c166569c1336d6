"""GPU: what a step leaves whose Poisson solve does not reach its tolerance (a cap of five
cycles, which the direct solve does not stand in for): the drifted positions, the velocities
of the first kick, no accelerations, and, through qz_step_host, the caller's velocities and
accelerations untouched.  The expected values are the kick and the drift in numpy, in the
order of the kernels' operations, so they compare equal."""
import numpy as np
import pytest
import torch

from quantizer_b200 import core

pytestmark = pytest.mark.gpu

KEYS = ("x", "y", "z", "vx", "vy", "vz", "m", "ax", "ay", "az")
DT = 1e-4


def _state(n):
    rng = np.random.default_rng(n)
    st = {k: 0.5 + rng.normal(0.0, 0.05, n).clip(-0.3, 0.3) for k in "xyz"}
    st.update({k: rng.normal(0.0, 0.1, n) for k in ("vx", "vy", "vz", "ax", "ay", "az")})
    st["m"] = rng.uniform(0.5, 1.5, n) / n
    return st


def _expect(st):
    v = {k: st["v" + k] + st["a" + k] * DT * 0.5 for k in "xyz"}
    return {**{k: st[k] + v[k] * DT for k in "xyz"}, **{"v" + k: v[k] for k in "xyz"},
            **{"a" + k: np.zeros_like(st["x"]) for k in "xyz"}}


def _check(sim, st):
    want, got = _expect(st), sim.particles()
    for k in want:
        np.testing.assert_array_equal(got[k], want[k], err_msg=k)


# head only, queued and (mixed form) queued; refined with its stages one after another
@pytest.mark.parametrize("kw", [dict(), dict(precision=1), dict(lmax=6, tree_overlap=0)], ids=str)
def test_failed_step(kw):
    st = _state(3000)
    with core.Simulation(st, 5, max_iter=5, **kw) as sim:
        sim.set_accelerations(st["ax"], st["ay"], st["az"])
        with pytest.raises(core.QZError, match="after 5 multigrid cycles"):
            sim.step(DT, 2)
        _check(sim, st)


@pytest.mark.parametrize("n", [3000, 40000])  # arrays moved by loads, and by transfers
def test_failed_host_step(n):
    st = _state(n)
    host = {}
    for k in KEYS:
        host[k] = torch.empty(n, dtype=torch.float64, pin_memory=True).numpy()
        host[k][:] = st[k]
    with core.Simulation(st, 5, max_iter=5) as sim:
        with pytest.raises(core.QZError, match="after 5 multigrid cycles"):
            sim.step_host(host, DT)
        _check(sim, st)
    want = _expect(st)
    for k in KEYS:
        np.testing.assert_array_equal(host[k], want[k] if k in "xyz" else st[k], err_msg=k)
