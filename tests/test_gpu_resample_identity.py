"""The corrector around the grid size from which its resample's weights are
all zero (N = 159 at the default spacing): 158 still resamples, 159 and above
leave every velocity as it is. Positions and velocities against the oracle,
bit for bit in REF arithmetic; in FAST arithmetic the velocities of 159 and
above are unchanged exactly."""
import numpy as np
import pytest

from flip3d_gb300 import scenes

pytestmark = pytest.mark.gpu


def cloud(n, seed):
    """A block of liquid of 14^3 cells, eight particles a cell, and its step-3 state."""
    rng = np.random.default_rng(seed)
    i = np.stack(np.meshgrid(*[np.arange(28)] * 3, indexing="ij"), -1).reshape(-1, 3)
    pos = ((i + 0.5 + rng.uniform(-0.45, 0.45, i.shape)) * (0.5 / n) + 20.0 / n).astype(np.float32)
    vel = rng.normal(0, 1, pos.shape).astype(np.float32)
    return pos, vel, np.full(len(pos), scenes.FLUID, np.uint8)


@pytest.mark.parametrize("n", [158, 159, 200])
@pytest.mark.parametrize("fast", [False, True])
def test_correct_around_the_identity(n, fast):
    from flip3d_gb300 import gpu
    from oracle import pyoracle as orc
    pos, vel, typ = cloud(n, n)
    nrm = np.zeros_like(pos)
    sim = gpu.Simulation(gpu.default_params(n, len(pos), seed=9,
                                            arith=gpu.ARITH_FAST if fast else gpu.ARITH_REF))
    sim.set_particles(pos, typ, vel, nrm)
    sim.set_step(3)
    sim.correct()
    p, v, _, _ = sim.get_particles()
    sim.close()
    cs, perm = orc.sort(n, pos)
    dt, re = np.float32(0.006), np.float32(0.5 / n)
    op, ov = orc.correct(n, pos, vel, typ, nrm, cs, perm, dt, re, 9, 3)
    if n > 158:
        assert np.array_equal(v, vel)
    if fast:  # native FP32: the FAST step test's tolerance
        assert np.abs(p - op).max() <= 2e-5
    else:
        assert np.array_equal(p, op)
        assert np.array_equal(v, ov)
