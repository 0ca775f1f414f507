"""The solver with its cells in registers on the smallest grids, where a cap
cannot select the general kernel, against the oracle: a block that is partly
filled (n = 6, 7), just filled (n = 8) and followed by a partly filled one (n = 9,
10, 12), and the same grids in one block with two and four cells a thread.

REF arithmetic: the oracle evaluates the same expressions and sums the dots in
another order, so the solver's stated 1e-5 of the largest pressure bounds the
difference and the iteration counts agree to one. FAST (not at multiples of four,
which take another kernel): the true residual in FP64 on the host meets the
tolerance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def system(n, seed):
    rng = np.random.default_rng(seed)
    A = (rng.random((n, n, n)) < 0.7).astype(np.uint8)
    for d in range(3):
        for e in (0, n - 1):
            A[(slice(None),) * d + (e,)] = 2
    L = np.where(A == 1, rng.uniform(-1.5, -0.2, A.shape), rng.uniform(0.1, 1.0, A.shape))
    b = np.where(A == 1, rng.standard_normal(A.shape), 0.0)
    return A.ravel(), L.ravel().astype(np.float32), b.ravel().astype(np.float32)


@pytest.mark.parametrize("n,ref", [(n, True) for n in (6, 7, 8, 9, 10, 12)] +
                         [(n, False) for n in (6, 7, 9, 10)])
def test_small_grids(n, ref):
    from flip3d_gb300 import gpu
    from oracle import pyoracle as orc
    A, L, b = system(n, n)
    zero = np.zeros(n ** 3, np.float32)
    kw = {} if ref else {"solve_mode": gpu.SOLVE_FAST, "precond": gpu.PRECOND_JACOBI}
    sim = gpu.Simulation(gpu.default_params(n, 1, rel_tol=1e-6, **kw))
    for blocks in (0, 1, 2):
        sim.solve_blocks(blocks)
        sim.set_grid(A=A, L=L, press=zero, div=b)
        st = sim.solve()
        assert st.status == 0
        p = sim.get_pressure()
        if ref:
            prm = orc.params(n, orc.PRECOND_REF, rel_tol=1e-6)
            x, _, it, _, _ = orc.solve(prm, A, L, zero, b)
            assert abs(st.iterations - it) <= 1, (st.iterations, it)
            assert np.abs(p - x).max() <= 1e-5 * np.abs(x).max()
        else:
            r = orc.fast_residual_fp64(n, A, L, -b, p)
            rel = np.linalg.norm(r) / np.linalg.norm(b.astype(np.float64))
            assert rel <= 1.05e-6, rel
    sim.close()
