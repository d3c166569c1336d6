"""GPU: the direct head solve (sine transforms) against the multigrid cycles it stands
in for, on every head size from 4^3 up, every boundary kind, FP64 and mixed, and the
rules around it.

Both paths end at the discrete solution of one problem: the cycles to the residual
tolerance 1e-10 of 4 pi G rho_mean (errors below 1e-10 of the potential's scale, whose
Laplacian's inverse is at most 1 / (3 pi^2)), the direct solve to rounding, so the
potentials are held to 1e-9 of their largest value and forces to 1e-8.  An iteration cap
below 100 keeps the cycles."""
import os
import subprocess
import sys

import numpy as np
import pytest

from quantizer_b200 import core, ics

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _run(L, steps=2, **kw):
    ic = ics.plummer(3000, a=0.05, seed=5)
    with core.Simulation(ic, L, **kw) as sim:
        sim.init_forces()
        sim.step(2e-4, steps)
        return sim.field("pot"), sim.field("pot_old"), sim.particles(), sim.stats()


@pytest.mark.parametrize("kw", [dict(), dict(precision=1), dict(bdry=0), dict(check_method=1),
                                dict(check_method=2)], ids=str)
@pytest.mark.parametrize("L", [2, 3, 4, 5, 6, 7])
def test_direct_equals_cycles(L, kw):
    # the point-wise test (method 1) holds the residual where the potential is rounded:
    # 6 |pot| eps / H^2 at the dense centre, above 1e-10 of the mean on the finer heads
    tol = dict(tol=1e-7) if kw.get("check_method") == 1 else {}
    pot, old, p, st = _run(L, **kw, **tol)
    ref, _, q, rt = _run(L, max_iter=99, **kw, **tol)
    bar = 1e-6 if tol else 1e-9
    assert st.last_converged == 1 and st.last_vcycles == 0 and rt.last_vcycles > 0
    assert np.abs(pot - ref).max() <= bar * np.abs(ref).max()
    np.testing.assert_array_equal(pot, old)
    for k in ("ax", "ay", "az"):
        assert np.abs(p[k] - q[k]).max() <= 10 * bar * np.abs(q[k]).max()


@pytest.mark.parametrize("L", [8, 9])
def test_large_heads_meet_the_test(L):
    ic = ics.plummer(3000, a=0.05, seed=5)
    with core.Simulation(ic, L) as sim:
        sim.init_forces()
        st = sim.stats()
        assert st.last_converged == 1
        if L == 8:
            assert st.last_vcycles == 0


def test_cycles_go_on_where_the_test_does_not_hold():
    """A tolerance below rounding: the direct result fails the test, cycles run from it to
    the cap, and the call fails with the cap's message, the potential at the solution."""
    ic = ics.plummer(3000, a=0.05, seed=5)
    for kw in (dict(), dict(precision=1)):
        with core.Simulation(ic, 5, **kw) as sim:
            sim.init_forces()
            ref = sim.field("pot")
        with core.Simulation(ic, 5, tol=1e-300, max_iter=100, **kw) as sim:
            with pytest.raises(core.QZError, match="after 100 multigrid cycles"):
                sim.init_forces()
            assert np.abs(sim.field("pot") - ref).max() <= 1e-12 * np.abs(ref).max()


def test_cap_near_the_cycles_needs_decides_as_before():
    ic = ics.plummer(3000, a=0.05, seed=5)
    with core.Simulation(ic, 5, max_iter=5) as sim:
        with pytest.raises(core.QZError, match="after 5 multigrid cycles"):
            sim.init_forces()


CHILD = r"""
import sys
import numpy as np
from quantizer_b200 import core, ics
L, prec, out, tile = int(sys.argv[1]), int(sys.argv[2]), sys.argv[3], int(sys.argv[4])
ic = ics.plummer(20000, a=0.05, seed=3)
with core.Simulation(ic, L, precision=prec, mg_tile=tile, max_iter=99) as sim:
    sim.init_forces()
    sim.step(2e-4, 2)
    np.savez(out, pot=sim.field("pot"), n=np.array([sim.stats().vcycles_total]))
"""


@pytest.mark.parametrize("L,prec", [(5, 0), (7, 0), (7, 1)])
def test_persistent_cycles_match_launch_per_phase(tmp_path, L, prec):
    """The cycles themselves (tests/test_gpu_mg_paths.py), which the direct solve leaves to
    runs with a low cap."""
    got = {}
    for launches, tile in ((1, 0), (0, 0), (0, 6), (0, -1)):
        out = str(tmp_path / f"{launches}_{tile}.npz")
        env = dict(os.environ, PYTHONPATH=ROOT)
        env.pop("QZ_MG_LAUNCHES", None)
        if launches:
            env["QZ_MG_LAUNCHES"] = "1"
        subprocess.run([sys.executable, "-c", CHILD, str(L), str(prec), out, str(tile)], check=True,
                       env=env, cwd=ROOT, timeout=300)
        with np.load(out) as z:
            got[launches, tile] = z["pot"], int(z["n"][0])
    want, n = got.pop((1, 0))
    assert n > 0
    for key, (pot, m) in got.items():
        assert m == n, key
        np.testing.assert_array_equal(pot, want, err_msg=str(key))
