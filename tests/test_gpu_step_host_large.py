"""flipgpu_step_host on both sides of the grid size from which the corrector leaves
the velocities as they are (N = 159 at the default spacing), where they are copied
out beside the spring: steps on host arrays, in place and into other arrays, and
without one of the outputs, against the same steps with the transfers apart."""
import numpy as np
import pytest

from flip3d_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [156, 160])
@pytest.mark.parametrize("fast", [True, False])
def test_steps(n, fast):
    from flip3d_gb300 import gpu
    rng = np.random.default_rng(n)
    g = np.stack(np.meshgrid(*[np.arange(24)] * 3, indexing="ij"), -1).reshape(-1, 3)
    pos = ((g + 0.5 + rng.uniform(-0.4, 0.4, g.shape)) * (0.5 / n) + 20.0 / n).astype(np.float32)
    vel = rng.normal(0, 0.3, pos.shape).astype(np.float32)
    typ = np.full(len(pos), scenes.FLUID, np.uint8)

    def make():
        sim = gpu.Simulation(gpu.default_params(
            n, len(pos), seed=3, solve_mode=gpu.SOLVE_FAST, precond=gpu.PRECOND_JACOBI,
            rel_tol=1e-6, arith=gpu.ARITH_FAST if fast else gpu.ARITH_REF))
        sim.set_particles(pos, typ, vel)
        sim.set_max_density(31.0)
        return sim
    a, b = make(), make()
    pb, vb = pos.copy(), vel.copy()
    for k in range(3):
        assert a.step().status == 0
        po, vo = (pb, vb) if k == 0 else (np.zeros_like(pb), np.zeros_like(vb))
        assert b.step_host(pb, vb, po, vo if k < 2 else None).status == 0
        p, v, _, _ = a.get_particles()
        assert np.array_equal(po, p)
        if k < 2:
            assert np.array_equal(vo, v)
            pb, vb = po, vo
        assert np.array_equal(b.get_particles()[1], v)
    a.close()
    b.close()
