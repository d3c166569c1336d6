"""GPU: qz_ensemble_autotune picks between settings of the multigrid cycles only where cycles
run.  With heads that the direct solve does, whichever combination the clock favours, the
first points-per-thread and tile options are taken; with a cap of 99 cycles, which the direct
solve does not stand in for, every combination is tried, so repeated picks stay among them."""
import pytest

from quantizer_b200 import core, ics

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", [dict(), dict(max_iter=99)], ids=str)
def test_cycle_settings_are_tuned_where_cycles_run(kw):
    sims = []
    for k in range(3):
        sims.append(core.Simulation(ics.plummer(2000 + 500 * k, a=0.05, seed=k), 4, **kw))
        sims[-1].init_forces()
    ppt, tiles = (8, 2, 4, 16, 1), (6, -1, 1, 5)
    for _ in range(3):
        t, p, g, ms = core.ensemble_autotune(sims, 1e-4, thread_opts=(1, 2), ppt_opts=ppt,
                                             tile_opts=tiles)
        assert t in (1, 2) and p in ppt and g in tiles and ms > 0
        if not kw:
            assert (p, g) == (8, 6)
    assert all((s.stats().vcycles_total > 0) == bool(kw) for s in sims)
    for s in sims:
        s.close()
