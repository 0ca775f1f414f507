"""P2G on both sides of the sizes where its kernel changes (n = 39, 40 in FAST
and 63, 64 in REF arithmetic; 9 for the smallest, 112 for a large grid), FAST
arithmetic against the per-particle kernels (FLIPGPU_GATHER=particle) and REF
arithmetic against the oracle: bit for bit."""
import os

import numpy as np
import pytest

from flip3d_gb300 import scenes

pytestmark = pytest.mark.gpu


def faces(gpu, sc, vel, arith, mode=None):
    if mode:
        os.environ["FLIPGPU_GATHER"] = mode
    try:
        sim = gpu.Simulation(gpu.default_params(sc.n, sc.count, arith=arith))
        sim.set_particles(sc.pos, sc.type, vel, sc.nrm)
        sim.sort()
        sim.p2g()
        u = sim.get_grid()[0]
        sim.close()
        return u
    finally:
        os.environ.pop("FLIPGPU_GATHER", None)


@pytest.mark.parametrize("n", [9, 39, 40, 63, 64, 112])
def test_p2g_kernels_agree(n):
    from flip3d_gb300 import gpu
    from oracle import pyoracle as orc
    sc = scenes.pool_sphere(n, seed=n)
    vel = np.random.default_rng(n).normal(0, 1, sc.pos.shape).astype(np.float32)
    vel[sc.type != scenes.FLUID] = 0
    a, b = faces(gpu, sc, vel, gpu.ARITH_FAST), faces(gpu, sc, vel, gpu.ARITH_FAST, "particle")
    assert all(np.array_equal(x, y) for x, y in zip(a, b))
    r = faces(gpu, sc, vel, gpu.ARITH_REF)
    cs, perm = orc.sort(n, sc.pos)
    want = orc.p2g(n, sc.pos, vel, sc.type, cs, perm)
    assert all(np.array_equal(x, np.asarray(y).ravel()) for x, y in zip(r, want))
