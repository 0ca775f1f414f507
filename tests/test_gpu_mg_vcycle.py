"""One V-cycle of the multigrid preconditioner against a plain restatement on
the host: the pressure after one CG iteration from zero, alpha z with z the
V-cycle of the right-hand side.

With one or two sweeps the middle levels run in tiles of shared memory, with
three in passes over the grid, and the levels of at most 16 cells an axis in one
block. The restatement knows none of that: whole-grid red-black half sweeps on
every level. Grids with middle levels of 18 to 64 cells (whole, partial and single
tiles, one and two middle levels) and random holes cover tiles at every edge.

The bound is eight times the distance of the restatement's own FP32 evaluation
from its FP64 one (the kernels multiply by an approximate reciprocal, off by a
rounding more): 1 to 3e-6 of the largest value. A half sweep of a middle level
that misses a sixth of one cell's neighbours, at a tile's edge, moves the result by
more than four times that (test_a_planted_mistake_exceeds_the_bound)."""
import numpy as np
import pytest

COARSE_SWEEPS = 2


def system(n, seed):
    """Liquid under a wavy surface with random holes of air and wall."""
    rng = np.random.default_rng(seed)
    x = (np.arange(n) + 0.5) / n
    X, Y, Z = np.meshgrid(x, x, x, indexing="ij")
    A = (Y < 0.55 + 0.15 * np.sin(7 * X) * np.cos(5 * Z)).astype(np.uint8)
    u = rng.random(A.shape)
    A[u < 0.02] = 0
    A[u > 0.99] = 2
    for d in range(3):
        for e in (0, n - 1):
            A[(slice(None),) * d + (e,)] = 2
    # no liquid cell walled in on all sides: its diagonal would be 0
    open_ = sum(np.roll(A != 2, s, d) for d in range(3) for s in (-1, 1)) > 0
    A[(A == 1) & ~open_] = 2
    L = np.where(A == 1, rng.uniform(-1.5, -0.2, A.shape), rng.uniform(0.1, 1.0, A.shape))
    b = np.where(A == 1, rng.standard_normal(A.shape), 0.0)
    return A, L.astype(np.float32), b.astype(np.float32)


def neighbours(x):
    p = np.pad(x, 1)
    return (((((p[:-2, 1:-1, 1:-1] + p[2:, 1:-1, 1:-1]) + p[1:-1, :-2, 1:-1]) +
              p[1:-1, 2:, 1:-1]) + p[1:-1, 1:-1, :-2]) + p[1:-1, 1:-1, 2:])


def pad_even(x):
    return np.pad(x, [(0, s % 2) for s in x.shape])


def children(x):
    m = x.shape[0] // 2
    return x.reshape(m, 2, m, 2, m, 2)


class Level:
    def __init__(self, A, diag, hs):
        self.A, self.hs = A, hs
        self.fl = A == 1
        self.d = np.where(self.fl, diag, 1)
        par = np.indices(A.shape).sum(0) & 1
        self.mask = [self.fl & (par == c) for c in (0, 1)]


def levels(A, diag, hs):
    out = [Level(A, diag, hs)]
    while A.shape[0] > 4:
        f = children(np.pad(A, [(0, s % 2) for s in A.shape], constant_values=2))
        liquid, air = (f == 1).any((1, 3, 5)), (f == 0).any((1, 3, 5))
        A = np.where(liquid, 1, np.where(air, 0, 2)).astype(np.uint8)
        hs = hs / 4
        out.append(Level(A, np.maximum(neighbours((A != 2).astype(np.int64)), 1), hs))
    return out


def vcycle(lv, l, b, nu, t, mistake=None):
    """z = V(b) in arithmetic of type t, mistake(l, color, sum) may change a
    half sweep's neighbour sums"""
    F = lv[l]
    hs, ihs, d = t(F.hs), t(1) / t(F.hs), F.d.astype(t)
    x = np.zeros(F.A.shape, t)

    def half(color):
        s = neighbours(x)
        if mistake:
            mistake(l, color, s)
        x[F.mask[color]] = ((b * ihs + s) / d)[F.mask[color]]

    if l == len(lv) - 1:
        for h in range(4 * COARSE_SWEEPS - 1):
            half(h & 1)
        return x
    for h in range(2 * nu):
        half(h & 1)
    res = np.where(F.fl, b - hs * (d * x - neighbours(x)), t(0))
    rc = children(pad_even(res)).sum((1, 3, 5), dtype=t) * t(0.125)
    e = vcycle(lv, l + 1, rc, nu, t, mistake)
    m = F.A.shape[0]
    up = e.repeat(2, 0).repeat(2, 1).repeat(2, 2)[:m, :m, :m]
    x[F.fl] += up[F.fl]
    for h in range(2 * nu):
        half((h & 1) ^ 1)
    return x


def one_iteration(A, L, b, nu, t, mistake=None):
    from oracle import pyoracle as orc
    n = A.shape[0]
    diag = orc.fast_diag(n, A.ravel(), L.ravel()).reshape(A.shape)
    hs = float(np.float32(1.0 / float(np.float32(1.0 / (float(n) * n)))))
    lv = levels(A, diag, hs)
    r = np.where(A == 1, b, 0).astype(t)
    z = vcycle(lv, 0, r, nu, t, mistake)
    z64, F = z.astype(np.float64), lv[0]
    q = np.where(F.fl, hs * (F.d.astype(np.float64) * z64 - neighbours(z64)), 0)
    return (r.astype(np.float64) * z64).sum() / (z64 * q).sum() * z64


def bound(A, L, b, nu):
    x = one_iteration(A, L, b, nu, np.float64)
    return x, 8 * np.abs(one_iteration(A, L, b, nu, np.float32) - x).max()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [36, 40, 52, 64, 76, 100, 128])
@pytest.mark.parametrize("sweeps", [1, 2, 3])
def test_one_iteration(n, sweeps):
    from flip3d_gb300 import gpu
    A, L, b = system(n, 10 * n + sweeps)
    want, tol = bound(A, L, b, sweeps)
    sim = gpu.Simulation(gpu.default_params(n, 1, rel_tol=1e-9, solve_mode=gpu.SOLVE_FAST,
                                            precond=gpu.PRECOND_MG, mg_sweeps=sweeps,
                                            refine_steps=0, max_iters=1))
    sim.set_grid(A=A.ravel(), L=L.ravel(), press=np.zeros(n ** 3, np.float32), div=-b.ravel())
    with pytest.raises(gpu.FlipGpuError):  # one iteration does not converge
        sim.solve()
    got = sim.get_pressure().reshape(A.shape)
    scale = np.abs(want).max()
    err = np.abs(got - want).max()
    print(f"n {n} sweeps {sweeps}: {err / scale:.2e} of the largest, bound {tol / scale:.2e}")
    assert err <= tol
    sim.close()


@pytest.mark.parametrize("sweeps", [1, 2])
def test_a_planted_mistake_exceeds_the_bound(sweeps):
    """On the host: one cell of a middle level beside a tile's edge misses a sixth
    of its neighbours' sum."""
    n = 52
    A, L, b = system(n, 3)
    want, tol = bound(A, L, b, sweeps)

    def mistake(l, color, s):
        if l == 1:
            s[cell] -= s[cell] / 6

    for cell in [(7, 8, 9), (8, 7, 8), (15, 10, 12), (16, 5, 9)]:
        err = np.abs(one_iteration(A, L, b, sweeps, np.float64, mistake) - want).max()
        assert err > 4 * tol, (cell, err / tol)
