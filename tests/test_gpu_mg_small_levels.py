"""The multigrid levels of at most eight cells an axis, whose cells are split
among four threads a line segment: grids whose first block level is such a level
itself (12, 16) and grids whose levels end in every small size (36: 36, 18, 9, 5,
3; 44: 44, 22, 11, 6, 3; 56: 56, 28, 14, 7, 4; 60: 60, 30, 15, 8, 4; 64: 64, 32,
16, 8, 4), with one to three sweeps.

The V-cycle is a fixed operator, so it shows in the iterations: on pool scenes the
refined solve with levels of powers of two takes 8 to 16 iterations to 1e-6; a
level that reads or skips a wrong cell costs a multiple. The bound is 24, and 36
for one sweep. The residual is checked in FP64 on the host, and a repeated solve
gives the same bits."""
import numpy as np
import pytest

from flip3d_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [12, 16, 36, 44, 56, 60, 64])
@pytest.mark.parametrize("sweeps", [1, 2, 3])
def test_small_levels(n, sweeps):
    from flip3d_gb300 import gpu
    from oracle import pyoracle as orc
    sc = scenes.pool_sphere(n, seed=4)
    sim = gpu.Simulation(gpu.default_params(n, sc.count, rel_tol=1e-6, solve_mode=gpu.SOLVE_FAST,
                                            precond=gpu.PRECOND_MG, arith=gpu.ARITH_FAST,
                                            mg_sweeps=sweeps))
    sim.set_scene(sc)
    sim.calibrate_max_density()
    sim.set_capture(True)
    assert sim.step().status == 0
    A, L, b, x0, _, _ = sim.solve_system()
    got = []
    for _ in range(2):
        sim.set_grid(A=A, L=L, press=x0, div=-b)
        st = sim.solve()
        got.append(sim.get_pressure())
    sim.close()
    assert st.status == 0 and st.iterations <= (36 if sweeps == 1 else 24), st.iterations
    assert np.array_equal(got[0], got[1])
    r = orc.fast_residual_fp64(n, A, L, b, got[0])
    rel = np.linalg.norm(r) / np.linalg.norm(b[A == 1].astype(np.float64))
    assert rel <= 1.05e-6, rel  # the device's own norm carries about 48 bits
