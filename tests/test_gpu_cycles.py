"""GPU: the multigrid cycles themselves, which the direct head solve leaves to its failures,
to low caps and to solver schedules.  The cases of tests/test_gpu_mg_paths.py (which now end
in the direct solve) and the mixed form's force bar of tests/test_gpu_head.py, with a cap of
99 cycles, below which the direct solve does not stand in; every run has to count cycles."""
import os
import subprocess
import sys

import numpy as np
import pytest

from oracle import oracle as O
from quantizer_b200 import core, ics

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import sys
import numpy as np
from quantizer_b200 import core, ics
L, prec, out, tiles = int(sys.argv[1]), int(sys.argv[2]), sys.argv[3], sys.argv[4].split(",")
ic = ics.plummer(20000, a=0.05, seed=3)
got = {}
for t in tiles:
    with core.Simulation(ic, L, precision=prec, mg_tile=int(t), max_iter=99) as sim:
        sim.init_forces()
        sim.step(2e-4, 3)
        p = sim.particles()
        got.update({"pot" + t: sim.field("pot"), "x" + t: p["x"], "ax" + t: p["ax"],
                    "n" + t: np.array([sim.stats().vcycles_total])})
np.savez(out, **got)
"""


def _run(tmp_path, L, prec, launches, tiles):
    out = str(tmp_path / f"{launches}.npz")
    env = dict(os.environ, PYTHONPATH=ROOT)
    env.pop("QZ_MG_LAUNCHES", None)  # (read once a process)
    if launches:
        env["QZ_MG_LAUNCHES"] = "1"
    subprocess.run([sys.executable, "-c", CHILD, str(L), str(prec), out,
                    ",".join(map(str, tiles))], check=True, env=env, cwd=ROOT, timeout=300)
    with np.load(out) as z:
        return {k: z[k] for k in z.files}


@pytest.mark.parametrize("L", [5, 6, 7])
@pytest.mark.parametrize("prec", [0, 1])
def test_persistent_cycles_match_launch_per_phase(tmp_path, L, prec):
    tiles = (0, 1, 2, 3, 4, 5, 6, 7, -1) if L == 7 else (0, 6, -1)
    want = _run(tmp_path, L, prec, 1, [0])
    got = _run(tmp_path, L, prec, 0, tiles)
    assert want["n0"][0] > 0
    for t in tiles:
        for k in ("n", "pot", "x", "ax"):
            np.testing.assert_array_equal(got[f"{k}{t}"], want[k + "0"], err_msg=f"{k} tile {t}")


def test_mixed_precision_force_error_of_the_cycles():
    ic = ics.plummer(10000, a=0.05, seed=1)
    dt = 1e-3 * ics.crossing_time(0.05)
    M = core.sequential_mass(ic["m"])
    ref = O.OracleSim(ic, O.params(5, total_mass=M))
    for _ in range(5):
        ref.step(dt)
    rp = ref.particles()
    ref.close()
    with core.Simulation(ic, 5, total_mass=M, precision=core.QZ_PREC_MIXED, max_iter=99) as sim:
        sim.init_forces()
        sim.step(dt, 5)
        p, st = sim.particles(), sim.stats()
    amag = np.sqrt(rp["ax"] ** 2 + rp["ay"] ** 2 + rp["az"] ** 2)
    err = np.sqrt(sum((p[k] - rp[k]) ** 2 for k in ("ax", "ay", "az")))
    assert (err / amag).max() < 1e-5
    assert st.last_converged == 1 and st.vcycles_total > 0 and st.last_vcycles > 0
