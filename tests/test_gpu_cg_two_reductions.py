"""GPU: cg_variant 3, the reference's two-reduction conjugate gradient from device memory,
on the fixture and with the bars of tests/test_gpu_node_cg.py."""
import ctypes as C

import numpy as np
import pytest

from conftest import golden
from quantizer_b200 import core, ics

pytestmark = pytest.mark.gpu

P = C.POINTER(C.c_double)


def test_two_reductions_match_the_reference():
    z = golden("node_cg.npz")
    pot, old, d = z["pot_in"].copy(), z["pot_in"].copy(), z["d"].copy()
    intr = z["intr"].astype(np.int32)
    rd = [int(v) for v in z["rd"]]
    with core.Simulation(ics.plummer(100, a=0.05, seed=1), 4, cg_variant=3) as sim:
        rc = sim.lib.qz_node_conjugate_gradient(
            sim.h, int(z["lv"][0]), rd[0], rd[1], rd[2], intr.size,
            intr.ctypes.data_as(C.POINTER(C.c_int)), float(z["mass"][0]), int(z["cells"][0]),
            d.ctypes.data_as(P), pot.ctypes.data_as(P), old.ctypes.data_as(P))
        assert rc == int(z["rc"][0]), sim.lib.qz_last_error().decode()
        assert sim.stats().cg_iterations > 0
    scale = np.abs(z["pot_out"]).max()
    assert np.abs(pot - z["pot_out"]).max() < 1e-9 * scale
    assert np.abs(old - z["pot_old_out"]).max() < 1e-9 * scale
