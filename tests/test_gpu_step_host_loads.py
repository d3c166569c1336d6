"""GPU: qz_step_host on few particles (one kernel each way moves the page-locked arrays)
gives the state of separate calls bit for bit: one particle, the edges of a block, the
largest number that takes this way and the next one, which does not; head only and refined;
arrays that start at an odd multiple of eight bytes."""
import numpy as np
import pytest
import torch

from quantizer_b200 import core

pytestmark = pytest.mark.gpu

KEYS = ("x", "y", "z", "vx", "vy", "vz", "m", "ax", "ay", "az")


@pytest.mark.parametrize("n", [1, 255, 257, 32768, 32769])
@pytest.mark.parametrize("levels", [0, 1])
def test_few_particles(n, levels):
    rng = np.random.default_rng(n)
    ic = {k: 0.5 + rng.normal(0.0, 0.05, n).clip(-0.3, 0.3) for k in "xyz"}
    ic.update({k: rng.normal(0.0, 0.1, n) for k in ("vx", "vy", "vz")})
    ic["m"] = rng.uniform(0.5, 1.5, n) / n
    with core.Simulation(ic, 4, lmax=4 + levels, ref_ptcl=9) as a, \
            core.Simulation(ic, 4, lmax=4 + levels, ref_ptcl=9) as b:
        a.init_forces()
        b.init_forces()
        p = a.particles()
        state = {}
        for q, k in enumerate(KEYS):
            buf = torch.empty(n + 1, dtype=torch.float64, pin_memory=True).numpy()
            state[k] = buf[q % 2:q % 2 + n]
            state[k][:] = ic["m"] if k == "m" else p[k]
        ref = {k: v.copy() for k, v in state.items()}
        for _ in range(2):
            a.step_host(state, 1e-4)
            b.set_particles(ref)
            b.set_accelerations(ref["ax"], ref["ay"], ref["az"])
            b.step(1e-4, 1)
            got = b.particles()
            for k in KEYS:
                if k != "m":
                    ref[k][:] = got[k]
        for k in KEYS:
            np.testing.assert_array_equal(state[k], ref[k], err_msg=k)
