"""The FAST corrector's row lists against the kernels that visit every cell
(FLIPGPU_GATHER=particle), bit for bit: scattered single particles, crowded
cells (near lists of several fills), pairs closer than the kick distance, wall
and liquid particles sharing a cell, particles in the grid's edge cells and
outside it, coincident particles, and counts that leave a partial warp."""
import os

import numpy as np
import pytest

from flip3d_gb300 import scenes

pytestmark = pytest.mark.gpu


def correct(gpu, n, pos, vel, typ, nrm, mode=None):
    if mode:
        os.environ["FLIPGPU_GATHER"] = mode
    try:
        sim = gpu.Simulation(gpu.default_params(n, len(pos), seed=5, arith=gpu.ARITH_FAST))
        sim.set_particles(pos, typ, vel, nrm)
        sim.set_step(2)
        sim.sort()
        sim.correct()
        p, v, _, _ = sim.get_particles()
        sim.close()
        return p, v
    finally:
        os.environ.pop("FLIPGPU_GATHER", None)


@pytest.mark.parametrize("n,m,crowd", [(8, 1, 0), (8, 33, 0), (9, 2500, 700), (24, 4097, 1500),
                                       (50, 30011, 900), (109, 60000, 5000)])
def test_rows_against_every_cell(n, m, crowd):
    from flip3d_gb300 import gpu
    rng = np.random.default_rng(n + m)
    pos = rng.uniform(0, 1, (m, 3)) * min(1.0, (m / 8.0) ** (1 / 3) / n)
    pos[:crowd] = 0.3 / n + rng.uniform(0, 1.5 / n, (crowd, 3))
    k = m // 10
    pos[rng.choice(m, k, replace=False)] = pos[rng.choice(m, k, replace=False)]
    i = rng.choice(m, k, replace=False)
    pos[i] = pos[rng.choice(m, k)] + rng.normal(0, 0.02 / n, (k, 3))
    i = rng.choice(m, k, replace=False)
    pos[i] = 1.0 - pos[i]
    pos[rng.choice(m, m // 50, replace=False)] = rng.uniform(-0.5, 1.5, (m // 50, 3))
    pos = pos.astype(np.float32)
    vel = rng.normal(0, 1, pos.shape).astype(np.float32)
    typ = np.where(rng.uniform(size=m) < 0.1, scenes.WALL, scenes.FLUID).astype(np.uint8)
    nrm = rng.normal(0, 1, pos.shape).astype(np.float32)
    a = correct(gpu, n, pos, vel, typ, nrm)
    b = correct(gpu, n, pos, vel, typ, nrm, "particle")
    for x, y in zip(a, b):
        assert np.array_equal(x, y, equal_nan=True)
