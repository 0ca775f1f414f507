"""The reposition's resample when its blocks stop waiting for one another: the
stuck particles that the rounds leave are resampled all the same, in the
reference's order, so the velocities are the oracle's bit for bit however early
the waits end, the call succeeds, and the solve's status stays clear of it.

Two or three blocks share the 448 stuck particles. With a limit of 0 every
block but the last to arrive leaves at the first barrier; 5 us and 50 us let it
end in a later round."""
import numpy as np
import pytest

from flip3d_gb300 import scenes
from test_gpu_parity import _forced_reposition_state, make_sim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wait", [0.0, 5e-6, 5e-5, 2.0])
@pytest.mark.parametrize("wide", [False, True])
def test_a_wait_that_ends_early_changes_nothing(wide, wait):
    from flip3d_gb300 import gpu
    from oracle import pyoracle as orc
    sc = scenes.pool_sphere(16, seed=4)
    o, pos, vel, dens, typ, u, A, zeros = _forced_reposition_state(orc, sc, 7, wide)
    o.stage(3)
    opos, ovel, _, _ = o.get()
    g = make_sim(gpu, sc.n, sc.count, seed=7)
    g.reposition_wait(wait)
    for _ in range(3):
        g.set_particles(pos, typ, vel, sc.nrm, dens)
        g.set_grid(u, A, zeros, zeros, zeros)
        g.set_step(5)
        assert g.advect() == o.stuck == 448
        gpos, gvel, _, _ = g.get_particles()
        assert np.array_equal(gpos, opos)
        fl = typ == 1
        assert np.array_equal(gvel[fl], ovel[fl])
    assert g.last_solve_stats().status == 0
    g.close()


def test_steps_do_not_depend_on_the_wait():
    """Whole steps, plain and as a replayed graph, whose statistics are read
    after the reposition."""
    from flip3d_gb300 import gpu
    sc = scenes.dam_break(32, seed=2)
    out = []
    for wait in (2.0, 0.0):
        for graph in (False, True):
            sim = gpu.Simulation(gpu.default_params(
                sc.n, sc.count, rel_tol=1e-6, seed=3, solve_mode=gpu.SOLVE_FAST,
                precond=gpu.PRECOND_MG, arith=gpu.ARITH_FAST))
            sim.set_scene(sc)
            sim.calibrate_max_density()
            sim.reposition_wait(wait)
            if graph:
                sim.capture_step()
            for _ in range(6):
                sim.step_graph() if graph else sim.step()
                assert sim.last_solve_stats().status == 0
            out.append(sim.get_particles())
            sim.close()
    for other in out[1:]:
        for x, y in zip(out[0], other):
            assert np.array_equal(x, y)
