"""The one-launch red-black Gauss-Seidel solve cuts the grid into tiles of any
size, one CTA each; every cut gives the per-colour launches' phi bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# one tile; tiles narrower than their halo would be; sizes that no tile divides;
# a thousand tiles' worth of cells; both halos (check intervals of 2 and of 4)
GRIDS = [(2, 2), (2, 64), (16, 8), (34, 130), (106, 46), (222, 106), (256, 256), (1024, 640)]


@pytest.mark.parametrize("check_every", [2, 8])
@pytest.mark.parametrize("lx,ly", [("nx", "ny"), (1.0, 3.0)])  # unit cells (the exact power-of-two form), unequal ones
@pytest.mark.parametrize("nx,ny", GRIDS)
def test_tiles_equal_per_colour_launches(pg, nx, ny, lx, ly, check_every):
    lx, ly = (float(nx), float(ny)) if lx == "nx" else (lx, ly)
    rho = np.random.default_rng(nx * 1000 + ny).normal(size=nx * ny)
    out = []
    for check in (check_every, 5):
        with pg.Context(nx, ny, lx, ly, 1) as c:
            c.set_rho(rho)
            it, res = c.poisson_rbgs(tol=0.0, max_iters=40, warm_start=False, check_every=check)
            out.append((it, res, *c.fields()))
    a, b = out
    assert a[0] == b[0] == 40
    for u, v in zip(a[2:], b[2:]):
        assert np.array_equal(u, v)
    # the residual's sums are grouped by tile: FP64 rounding of a sum of positive terms
    assert abs(a[1] - b[1]) <= nx * ny * 2.3e-16 * b[1]
