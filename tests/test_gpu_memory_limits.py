"""Solves on a device that has no room for more: the one-launch Gauss-Seidel solve's
buffers are optional, and an FFT solve takes no more memory than its spectrum and one
grid."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("room", [0, 140000])  # none, or for the partial sums alone
@pytest.mark.parametrize("nx,ny", [(64, 96), (256, 128)])
def test_gauss_seidel_without_its_exchange_buffers(pg, nx, ny, room, mixed):
    rho = np.random.default_rng(nx).normal(size=nx * ny)
    with pg.Context(nx, ny, 1.0, 2.0, 1) as c:
        c.set_rho(rho)
        c.set_rbgs_precision(False)
        c.poisson_rbgs(tol=0.0, max_iters=3, warm_start=False, check_every=1)  # the buffers of any solve
        want = c.poisson_rbgs(tol=0.0, max_iters=40, warm_start=False, check_every=5), c.fields()
        c.set_rbgs_precision(mixed)
        with pg.test_alloc_budget(room):
            got = c.poisson_rbgs(tol=0.0, max_iters=40, warm_start=False, check_every=8), c.fields()
        assert got[0][0] == want[0][0] == 40
        assert all(np.array_equal(a, b) for a, b in zip(got[1], want[1]))
        it, _ = c.poisson_rbgs(tol=0.0, max_iters=40, warm_start=False, check_every=8)  # with room again
        assert it == 40


@pytest.mark.parametrize("nx,ny", [(96, 160), (64, 64), (77, 33)])
def test_fft_solve_within_spectrum_and_one_grid(pg, nx, ny):
    rho = np.random.default_rng(nx).normal(size=nx * ny)
    with pg.Context(nx, ny, float(nx), float(ny), 1) as c, pg.Context(nx, ny, float(nx), float(ny), 1) as free:
        for k in (c, free):
            k.set_rho(rho)
            k.fields()  # phi and E
        with pg.test_alloc_budget(16 * (nx // 2 + 1) * ny + 8 * nx * ny):
            c.poisson_fft()
        free.poisson_fft()
        assert all(np.array_equal(a, b) for a, b in zip(c.fields(), free.fields()))


def test_the_budget_fails_with_nomem(pg):
    with pg.test_alloc_budget(1000):
        with pytest.raises(pg.PicError) as e:
            pg.Context(16, 16, 1.0, 1.0, 1000)
    assert e.value.code == -3  # PIC_ERR_NOMEM
    pg.Context(16, 16, 1.0, 1.0, 1000).close()
