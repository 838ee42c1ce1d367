"""The diagnostics' sums of rho and E^2 belong to the grids at hand whoever made them: a
time step's solve leaves them, a solve by itself does not, and each change of rho or E
is seen."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def check(c, nx, ny):
    d = c.diagnostics()
    rho = c.rho()
    _, ex, ey = c.fields()
    # FP64 sums in another order
    assert abs(d["integrated_rho"] - rho.sum()) <= 2.3e-16 * rho.size * np.abs(rho).sum()
    want = 0.5 * (ex**2 + ey**2).sum()
    assert abs(d["field_energy"] - want) <= 2.3e-16 * rho.size * want


@pytest.mark.parametrize("solve", ["poisson_fft", "poisson_rbgs"])
@pytest.mark.parametrize("nx,ny", [(16, 8), (30, 22), (512, 330), (1200, 900)])
def test_sums_follow_the_grids(pg, nx, ny, solve):
    rng = np.random.default_rng(nx)
    n = 4000
    kw = dict(tol=1e-3, max_iters=200) if solve == "poisson_rbgs" else {}
    with pg.Context(nx, ny, float(nx), float(ny), n) as c:
        c.upload(rng.random(n) * nx, rng.random(n) * ny, -np.ones(n), rng.normal(size=n), rng.normal(size=n))
        c.deposit(1, background=1.0, download=False)
        getattr(c, solve)(**kw)
        check(c, nx, ny)
        c.set_rho(rng.normal(size=nx * ny))
        check(c, nx, ny)
        getattr(c, solve)(**kw)
        check(c, nx, ny)
        hist = c.run(3, scheme=1, dt=0.1, background=n / (nx * ny), use_graph=True)
        d = c.diagnostics()
        assert d["field_energy"] == hist[-1][4] and d["integrated_rho"] == hist[-1][2]
        check(c, nx, ny)
        getattr(c, solve)(**kw)
        check(c, nx, ny)
        c.set_fields(ex=rng.normal(size=nx * ny))
        check(c, nx, ny)
