"""The mesher's field at grids where the slab-bound blocks loop over their
cells (n^3 above 304 blocks of 256 cells) and where one line of cells is
shorter than the five-cell window, on lists older than the positions: bit
for bit the oracle's."""
import numpy as np
import pytest

from flip3d_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4, 47])
def test_field_on_stale_lists(n):
    from flip3d_gb300 import gpu
    from oracle import pyoracle as orc
    sc = scenes.pool_sphere(n, seed=2)
    sim = gpu.Simulation(gpu.default_params(n, sc.count))
    sim.set_scene(sc)
    sim.sort()
    cs, perm = sim.get_cells()
    rng = np.random.default_rng(n)
    moved = sc.pos.copy()
    fl = sc.type == scenes.FLUID
    moved[fl] += rng.uniform(-1.2 / n, 1.2 / n, size=(int(fl.sum()), 3)).astype(np.float32)
    sim.put_state(moved, np.zeros_like(moved))
    pts = rng.uniform(-0.05, 1.05, size=(3000, 3)).astype(np.float32)
    assert np.array_equal(sim.implicit(pts), orc.implicit(n, moved, sc.type, cs, perm, pts))
    m = sim.mesh(field=True)
    om = orc.mesh(n, moved, sc.type, cs, perm)
    assert np.array_equal(m["field"], om["phi"])
    assert np.array_equal(m["vertices"].ravel(), om["vertices"])
    assert np.array_equal(m["normals"].ravel(), om["normals"])
    sim.close()
