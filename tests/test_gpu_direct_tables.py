"""GPU: the direct head solve's tables are in place when a simulation exists.  The passes run
on the simulation's streams, which nothing on the default stream precedes, so no copy there
may belong to the first solve: it is done while the default stream is still busy, and gives
what later solves of the same state give, bit for bit."""
import numpy as np
import pytest
import torch

from quantizer_b200 import core, ics

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lmin", [4, 6])  # (the cycles behind a 128^3 solve want every SM)
def test_first_solve_leaves_the_default_stream_alone(lmin):
    ic = ics.plummer(3000, a=0.05, seed=5)
    pots = []
    for _ in range(3):  # the first simulation also loads the kernels
        with core.Simulation(ic, lmin) as sim:
            busy = torch.cuda.Event()
            torch.cuda.synchronize()
            torch.cuda._sleep(600_000_000)  # some 0.3 s
            busy.record()
            sim.init_forces()
            waited = busy.query()
            torch.cuda.synchronize()
            pots.append(sim.field("pot"))
    assert not waited
    for p in pots[1:]:
        np.testing.assert_array_equal(p, pots[0])
