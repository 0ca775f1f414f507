"""The reposition's resample with fewer blocks than the device holds, as on a
context with fewer SMs: one (an ordinary launch, as on a device without
cooperative launches), two, and as many as fit give the oracle's velocities."""
import numpy as np
import pytest

from flip3d_gb300 import scenes
from test_gpu_parity import _forced_reposition_state, make_sim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wide", [False, True])
def test_blocks_do_not_change_the_resample(wide):
    from flip3d_gb300 import gpu
    from oracle import pyoracle as orc
    sc = scenes.pool_sphere(16, seed=4)
    o, pos, vel, dens, typ, u, A, zeros = _forced_reposition_state(orc, sc, 9, wide)
    o.stage(3)
    opos, ovel, _, _ = o.get()
    g = make_sim(gpu, sc.n, sc.count, seed=9)
    for blocks in (1, 2, 0):
        g.reposition_blocks(blocks)
        g.set_particles(pos, typ, vel, sc.nrm, dens)
        g.set_grid(u, A, zeros, zeros, zeros)
        g.set_step(5)
        assert g.advect() == o.stuck > 400
        gpos, gvel, _, _ = g.get_particles()
        assert np.array_equal(gpos, opos)
        fl = typ == 1
        assert np.array_equal(gvel[fl], ovel[fl])
    g.close()
