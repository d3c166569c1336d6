"""GPU: the on-chip conjugate gradient's waits, for a ghost's words and for a block's sums, on
words that nothing publishes: each ends at its poll limit, the call fails with the wait's
message, and the simulation keeps working."""
import pytest

from quantizer_b200 import core, ics

pytestmark = pytest.mark.gpu


def test_waits_give_up():
    with core.Simulation(ics.plummer(20000, a=0.04, seed=9), 5, lmax=6, ref_ptcl=9) as sim:
        res = (core.C.c_int * 2)(7, 7)
        assert sim.lib.qz_test_wait_gives_up(sim.h, 2, res) == 1
        assert "another block's words" in sim.lib.qz_last_error().decode()
        assert list(res) == [0, 0]
        sim.init_forces()
        sim.step(1e-5, 1)
        assert sim.stats().steps == 1
