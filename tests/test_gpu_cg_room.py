"""GPU: where the on-chip conjugate gradient finds no room for a level's order (more bricks
than it takes) or for the exchange between its blocks, the level is solved from device memory
by the two-reduction kernel (cg_variant 3): same state, bit for bit, and same iterations."""
import numpy as np
import pytest

from quantizer_b200 import core, ics

pytestmark = pytest.mark.gpu


def _run(limits=(0, 0), **kw):
    ic = ics.plummer(20000, a=0.04, seed=9)
    with core.Simulation(ic, 5, lmax=7, ref_ptcl=9, **kw) as sim:
        core._check(sim.lib.qz_test_cg_limits(sim.h, *limits))
        sim.init_forces()
        sim.step(1e-4, 2)
        assert sim.stats().levels == 3
        return sim.particles(), sim.stats().cg_iterations, sim.lib.qz_test_cg_scratch(sim.h)


@pytest.mark.parametrize("limits", [(1, 0), (0, 1)], ids=["bricks", "exchange"])
def test_no_room_leaves_a_level_to_the_kernel_in_memory(limits):
    got, it, scratch = _run(limits)
    want, iw, _ = _run(cg_variant=3)
    assert it == iw and scratch == 0
    for k in want:
        np.testing.assert_array_equal(got[k], want[k], err_msg=k)


def test_a_list_of_one_node_too():
    ic = ics.plummer(3000, a=0.05, seed=2)
    pots = []
    for bricks, kw in ((1, dict()), (0, dict(cg_variant=3))):
        with core.Simulation(ic, 4, head_pot_method=1, **kw) as sim:
            core._check(sim.lib.qz_test_cg_limits(sim.h, bricks, 0))
            sim.init_forces()
            pots.append(sim.field("pot"))
    np.testing.assert_array_equal(pots[0], pots[1])
