"""Units of cells whose particles are taken in pieces: all lanes of a warp share the cells
that a piece reaches, whatever their number and place in the unit; and tiles so large, or
grids so small, that the launch has few warps. The grids equal the one-particle-per-thread
kernel's bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NGP, CIC, TSC, ESK = 0, 1, 2, 3
ATOMIC, AUTO = 3, 0


def start(pg, nx, ny, dense, per, species, seed):
    """`per` particles in each of the cells `dense` = [(ix, iy), ...], a few anywhere."""
    rng = np.random.default_rng(seed)
    m, few = per * len(dense), nx * ny // 3 + 2
    x, y = rng.random(m + few) * nx, rng.random(m + few) * ny
    x[:m] = np.repeat([c[0] for c in dense], per) + rng.random(m)
    y[:m] = np.repeat([c[1] for c in dense], per) + rng.random(m)
    n = m + few
    q = np.full(n, -1.5) if species == 1 else rng.choice([-1.0, 2.0, 0.25], n)
    vx, vy = np.clip(rng.normal(0, 0.15, (2, n)), -0.9, 0.9)
    c = pg.Context(nx, ny, float(nx), float(ny), n)
    c.upload(x, y, q, vx, vy)
    return c


def compare(c, schemes=(NGP, CIC, TSC, ESK)):
    for scheme in schemes:
        got = []
        for order in (AUTO, ATOMIC):
            c.set_order(order)
            c.deposit(scheme, dt=1.0, download=False)
            got.append(c.rho_fixed()[0])
        c.set_order(AUTO)
        assert np.array_equal(*got), scheme


# neighbours along a row, from one cell to more than half a unit; with gaps; at a unit's
# ends; rows apart
DENSE = {"1": [(7, 3)], "2": [(7, 3), (8, 3)], "3": [(31, 3), (32, 3), (33, 3)], "5": [(k, 5) for k in range(60, 65)],
         "17": [(k, 2) for k in range(40, 57)], "gaps": [(3, 1), (9, 1), (30, 1)], "ends": [(0, 0), (31, 0), (32, 0), (69, 8)],
         "rows": [(20, 0), (20, 1), (21, 1), (20, 8)]}


@pytest.mark.parametrize("species", [1, 2])
@pytest.mark.parametrize("per", [130, 700, 5003])
@pytest.mark.parametrize("dense", list(DENSE))
def test_dense_cells_among_sparse_ones(pg, dense, per, species):
    with start(pg, 70, 9, DENSE[dense], per, species, per) as c:
        c.sort()
        compare(c)
        c.deposit_current(1.0, download=False)
        sorted_j = c.current_fixed()
        c.push(0.3)  # between sorts
        compare(c)
    with start(pg, 70, 9, DENSE[dense], per, species, per) as c:
        if c.is_sorted():
            c.push(0.0)
        c.deposit_current(1.0, download=False)
        for a, b in zip(sorted_j, c.current_fixed()):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("species", [1, 2])
def test_tiles_beyond_their_accumulators(pg, species):
    """More than 2^17 particles in a tile: its pieces go to the grid."""
    with start(pg, 40, 9, [(10, 4), (11, 4), (12, 5)], 60000, species, 3) as c:
        c.sort()
        compare(c)
        c.push(0.3)
        compare(c)


@pytest.mark.parametrize("tile", [(64, 32), (32, 4), (3, 5), (1, 1)])
@pytest.mark.parametrize("nx,ny,n", [(64, 64, 20000), (200, 13, 900), (5, 4, 3000)])
def test_tiles_asked_for(pg, nx, ny, n, tile):
    rng = np.random.default_rng(n)
    with pg.Context(nx, ny, float(nx), float(ny), n) as c:
        c.upload(rng.random(n) * nx, rng.random(n) * ny, np.full(n, 2.0), *rng.normal(0, 0.3, (2, n)))
        c.set_tile(*tile)
        c.sort()
        compare(c)
        c.push(0.4)
        compare(c)
