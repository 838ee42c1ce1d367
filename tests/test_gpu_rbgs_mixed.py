"""The mixed-precision red-black Gauss-Seidel solve: its FP32 sweeps on every cut of
the grid equal an FP32 emulation, and it stops after max_iters sweeps at most."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def zero_sum_integers(nx, ny, seed):
    rho = np.random.default_rng(seed).integers(-50, 50, nx * ny).astype(np.float64)
    rho[0] -= rho.sum()  # sums of them are exact: the right-hand side does not depend on their order
    return rho


def solve(pg, nx, ny, lx, ly, rho, mixed, **kw):
    with pg.Context(nx, ny, lx, ly, 1) as c:
        c.set_rho(rho)
        c.set_rbgs_precision(mixed)
        it, res = c.poisson_rbgs(warm_start=False, **kw)
        return it, res, c.fields()[0].reshape(ny, nx)


def emulate(nx, ny, lx, ly, rho, sweeps):
    """FP32 red-black sweeps from zero on the FP64 right-hand side, in the solver's order."""
    dx2, dy2 = (lx / nx) * (lx / nx), (ly / ny) * (ly / ny)
    den = 2.0 * (1.0 / dx2 + 1.0 / dy2)
    ix2, iy2, inv = np.float32(1.0 / dx2), np.float32(1.0 / dy2), np.float32(1.0 / den)
    b = (rho * ((lx / nx) * (ly / ny))).astype(np.float32).reshape(ny, nx)
    e = np.zeros((ny, nx), np.float32)
    colour = np.add.outer(np.arange(ny), np.arange(nx)) % 2
    for _ in range(sweeps):
        for k in (0, 1):
            we = np.roll(e, 1, 1) + np.roll(e, -1, 1)
            sn = np.roll(e, 1, 0) + np.roll(e, -1, 0)
            e = np.where(colour == k, (we * ix2 + sn * iy2 + b) * inv, e)
    phi = e.astype(np.float64)
    return phi - phi.mean()


# one tile; tiles as wide as the halo; sizes that no tile divides; the largest that fit
GRIDS = [(2, 2), (2, 64), (16, 8), (96, 50), (64, 64), (90, 46), (384, 128), (512, 512), (1024, 512)]


@pytest.mark.parametrize("dx,dy", [(1.0, 1.0), (2.0, 3.0)])  # unit cells (the exact power-of-two form), unequal ones
@pytest.mark.parametrize("nx,ny", GRIDS)
def test_fp32_sweeps_equal_the_emulation(pg, nx, ny, dx, dy):
    rho = zero_sum_integers(nx, ny, nx + ny)
    lx, ly = nx * dx, ny * dy
    for sweeps in (4, 8):  # one pass, the residual checked before and after it
        it, _, phi = solve(pg, nx, ny, lx, ly, rho, True, tol=0.0, max_iters=sweeps, check_every=64)
        assert it == sweeps
        want = emulate(nx, ny, lx, ly, rho, sweeps)
        # the same FP32 values; the mean is an FP64 sum of them
        assert np.max(np.abs(phi - want)) <= nx * ny * 2.3e-16 * np.max(np.abs(want))


def test_other_grids_sweep_in_fp64(pg):
    nx, ny = 222, 106  # 5,883 tiles of 2 x 2: too many for the mixed mode
    rho = zero_sum_integers(nx, ny, nx + ny)
    a, b = (solve(pg, nx, ny, 2.0 * nx, 3.0 * ny, rho, mixed, tol=0.0, max_iters=8, check_every=8) for mixed in (True, False))
    assert a[0] == b[0] == 8 and a[1] == b[1] and np.array_equal(a[2], b[2])


@pytest.mark.parametrize("check_every", [1, 16])
@pytest.mark.parametrize("max_iters", [0, 1, 2, 3, 5, 6, 37, 402])
@pytest.mark.parametrize("nx,ny", [(64, 64), (96, 50)])
def test_stops_after_max_iters_sweeps(pg, nx, ny, max_iters, check_every):
    rho = zero_sum_integers(nx, ny, 7)
    it, res, phi = solve(pg, nx, ny, float(nx), float(ny), rho, True, tol=0.0, max_iters=max_iters,
                         check_every=check_every)
    assert it == max_iters
    it64, res64, phi64 = solve(pg, nx, ny, float(nx), float(ny), rho, False, tol=0.0, max_iters=max_iters, check_every=5)
    assert it64 == max_iters
    if max_iters < 4:  # all in FP64
        assert np.array_equal(phi, phi64)


def test_largest_sweep_limit(pg):
    """A limit near the largest int converges as any other that is not reached."""
    rho = zero_sum_integers(64, 64, 3)
    a = solve(pg, 64, 64, 64.0, 64.0, rho, True, tol=1e-8, max_iters=100000, check_every=16)
    b = solve(pg, 64, 64, 64.0, 64.0, rho, True, tol=1e-8, max_iters=2**31 - 1, check_every=16)
    assert a[0] == b[0] and a[0] < 100000 and a[1] == b[1] <= 1e-8 and np.array_equal(a[2], b[2])
