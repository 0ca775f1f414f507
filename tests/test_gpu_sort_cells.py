"""The cell lists' order at every size of cell where the sort changes its method
(networks of 8 and 16 keys, insertion up to 32, heapsort above): cells of exactly
0 to 40 particles and some large ones, the particles' indices shuffled, half of
them above the cell's mid-plane. FAST lists put the lower half first, each half in
particle order; REF lists are in particle order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [list(range(41)), [200, 1, 33, 0, 1500, 16, 17, 8, 9]])
@pytest.mark.parametrize("fast", [False, True])
def test_cells_of_every_size(sizes, fast):
    from flip3d_gb300 import gpu
    n = 8
    rng = np.random.default_rng(len(sizes))
    ids = rng.choice(n ** 3, len(sizes), replace=False)
    cell = np.repeat(ids, sizes)
    rng.shuffle(cell)
    base = np.stack([cell // (n * n), cell // n % n, cell % n], -1)
    pos = ((base + rng.uniform(0.05, 0.95, base.shape)) / n).astype(np.float32)
    sim = gpu.Simulation(gpu.default_params(n, len(pos),
                                            arith=gpu.ARITH_FAST if fast else gpu.ARITH_REF))
    sim.set_particles(pos, np.ones(len(pos), np.uint8))
    sim.sort()
    cs, perm = sim.get_cells()
    sim.close()
    assert np.array_equal(np.diff(cs.astype(np.int64)), np.bincount(cell, minlength=n ** 3))
    up = pos[:, 2] >= ((base[:, 2] + 0.5) / n).astype(np.float32)  # n = 8: exact
    want = np.lexsort((np.arange(len(pos)), up if fast else np.zeros(len(pos)), cell))
    assert np.array_equal(perm, want)
