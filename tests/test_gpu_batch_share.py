"""The batch tuner's caps are shares of the grid that a member's solve takes
without a cap. Small odd grids run the solver with its cells in registers, one
block an SM, unless a cap leaves it too few blocks: then the general kernel
runs, with more blocks an SM. The caps that tuning leaves have to be the chosen
share of the former, whichever kernel the last trial ran: with 48 members of
67^3 cells the trial without caps runs the former, and every other the latter."""
import numpy as np
import pytest

from flip3d_gb300 import scenes

pytestmark = pytest.mark.gpu


def test_caps_are_the_share_that_was_timed():
    torch = pytest.importorskip("torch")
    from flip3d_gb300 import gpu
    n, members = 67, 48
    w = 1.0 / n
    sc = scenes.build(n, [scenes.Box((w, w, w), (0.3, 0.3, 0.3))], 3)
    sims = []
    for m in range(members):
        sim = gpu.Simulation(gpu.default_params(n, sc.count, rel_tol=1e-6, seed=m,
                                                solve_mode=gpu.SOLVE_FAST,
                                                precond=gpu.PRECOND_JACOBI, arith=gpu.ARITH_FAST))
        sim.set_scene(sc)
        sim.calibrate_max_density()
        sims.append(sim)
    batch = gpu.Batch(sims)
    batch.step()
    batch.sync()
    before = [s.get_pressure() for s in sims]
    share = batch.tune()
    caps = [s.solve_blocks() for s in sims]
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    want = 0 if share == 0.0 else max(1, int(np.floor(share * sms / members + 0.5)))
    print(f"share {share}, caps {set(caps)}, expected {want}")
    assert set(caps) == {want}
    for s, p in zip(sims, before):
        assert np.array_equal(s.get_pressure(), p)
