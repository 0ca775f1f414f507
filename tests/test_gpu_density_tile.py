"""The FAST density's tile kernel (from n = 64) against the kernel with a
particle a thread (FLIPGPU_GATHER=particle): bit for bit on grids that are and
are not multiples of its 4 x 4 x 8 tiles, with single particles and pairs, empty
and crowded cells, wall and liquid particles sharing a cell, particles outside
the grid (listed in its edge cells), and positions that are not finite."""
import os

import numpy as np
import pytest

from flip3d_gb300 import scenes

pytestmark = pytest.mark.gpu


def density(gpu, n, pos, typ, mode=None):
    if mode:
        os.environ["FLIPGPU_GATHER"] = mode
    try:
        sim = gpu.Simulation(gpu.default_params(n, len(pos), arith=gpu.ARITH_FAST))
        sim.set_particles(pos, typ)
        sim.set_max_density(31.0)
        sim.sort()
        sim.compute_density()
        d = sim.get_particles()[2]
        sim.mark_water()
        _, A, L, _, _ = sim.get_grid()
        sim.close()
        return d, A, L
    finally:
        os.environ.pop("FLIPGPU_GATHER", None)


@pytest.mark.parametrize("n", [64, 65, 70, 75, 96])
def test_tile_density(n):
    from flip3d_gb300 import gpu
    rng = np.random.default_rng(n)
    sc = scenes.pool_sphere(n, seed=n)
    pos, typ = sc.pos.copy(), sc.type.copy()
    fl = np.flatnonzero(typ == scenes.FLUID)
    crowd = rng.choice(fl, 900, replace=False)
    pos[crowd] = (rng.uniform(0, 1, (900, 3)) * (2.0 / n) + 0.4).astype(np.float32)
    out = rng.choice(fl, 60, replace=False)
    pos[out] = rng.uniform(-2, 3, (60, 3)).astype(np.float32)
    pos[out[:3]] = [[np.nan, 0.5, 0.5], [np.inf, 0.2, 0.2], [0.3, -np.inf, 0.7]]
    pos[out[3:5]] = 1e9
    typ[rng.choice(fl, 200, replace=False)] = scenes.WALL
    a, b = density(gpu, n, pos, typ), density(gpu, n, pos, typ, "particle")
    for x, y in zip(a, b):
        assert np.array_equal(x, y, equal_nan=True)
