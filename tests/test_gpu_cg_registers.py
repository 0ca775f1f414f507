"""The solver with its cells in registers (grids of up to four cells a thread
on one block an SM: n up to 67) against the kernel that reads them from memory
in every phase, which a cap of a few blocks selects: REF arithmetic and the
Jacobi-preconditioned FAST solver on odd grids, with one, two and four cells
a thread, and n = 68, which takes the latter either way.

Both evaluate the same expressions cell by cell and sum the dots, to about 48
bits, in other orders, so the iterates differ by the rounding of the scalars:
the solver's stated 1e-5 of the largest pressure bounds it, and the iteration
counts agree to one per hundred."""
import numpy as np
import pytest

from flip3d_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [9, 41, 43, 53, 55, 67, 68])
@pytest.mark.parametrize("ref", [True, False])
def test_register_solver_matches_the_general_one(n, ref):
    from flip3d_gb300 import gpu
    if not ref and n % 4 == 0:
        n += 2
    sc = scenes.pool_sphere(n, seed=n)
    kw = {} if ref else {"solve_mode": gpu.SOLVE_FAST, "precond": gpu.PRECOND_JACOBI}
    sim = gpu.Simulation(gpu.default_params(n, sc.count, rel_tol=1e-6 if not ref else 1e-5, **kw))
    sim.set_scene(sc)
    sim.calibrate_max_density()
    sim.set_capture(True)
    assert sim.step().status == 0
    A, L, b, x0, _, _ = sim.solve_system()
    got = {}
    for blocks in (0, 3, 0):
        sim.solve_blocks(blocks)
        sim.set_grid(A=A, L=L, press=x0, div=-b)
        st = sim.solve()
        assert st.status == 0
        p = sim.get_pressure()
        if blocks in got:
            assert np.array_equal(got[blocks][0], p)  # deterministic
        got[blocks] = (p, st.iterations)
    (p, it), (q, jt) = got[0], got[3]
    assert np.abs(p - q).max() <= 1e-5 * np.abs(q).max()
    assert abs(it - jt) <= 1 + jt // 100, (it, jt)
    sim.close()
