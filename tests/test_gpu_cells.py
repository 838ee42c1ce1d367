"""The cell kernels (freshly sorted and between sorts) and the sorted current
against the kernels that take one particle per thread, in the int64 grids: sums
of integers, equal bit for bit whatever the units, pieces and lanes per cell."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NGP, CIC, TSC, ESK = 0, 1, 2, 3
ATOMIC, AUTO = 3, 0

# grid and particles per cell: one to 32 lanes per cell, units of 1 to 32 cells, rows
# shorter than a unit or a tile, cells longer than the stage buffer
SHAPES = [(1, 1, 9), (5, 3, 7), (33, 9, 2), (70, 34, 40), (64, 16, 64), (130, 10, 200), (20, 10, 1500)]


def particles(nx, ny, ppc, kind, rng):
    n = nx * ny * ppc
    if kind == "lattice":  # the same number in every cell, corners and edges of cells among them
        c = np.repeat(np.arange(nx * ny), ppc)
        t = np.tile(np.arange(ppc), nx * ny)
        x, y = c % nx + (t % 4) / 4.0, c // nx + (t // 4 % 4) / 4.0
    elif kind == "clump":  # two thirds of them in one cell, many cells empty
        x, y = rng.random(n) * nx, rng.random(n) * ny
        m = 2 * n // 3
        x[:m], y[:m] = nx // 2 + rng.random(m), ny // 2 + rng.random(m)
    else:
        x, y = rng.random(n) * nx, rng.random(n) * ny
    return x, y


def start(pg, nx, ny, ppc, kind, species, vth, seed):
    rng = np.random.default_rng(seed)
    x, y = particles(nx, ny, ppc, kind, rng)
    n = len(x)
    q = np.full(n, -1.5) if species == 1 else rng.choice([-1.0, 2.0, 0.25], n)
    vx, vy = np.clip(rng.normal(0, vth, (2, n)), -0.9, 0.9)
    vx[: n // 8] = 0.0
    c = pg.Context(nx, ny, float(nx), float(ny), n)
    c.upload(x, y, q, vx, vy)
    return c


@pytest.mark.parametrize("species", [1, 2])
@pytest.mark.parametrize("kind", ["uniform", "lattice", "clump"])
@pytest.mark.parametrize("nx,ny,ppc", SHAPES)
def test_cell_kernels_equal_one_particle_per_thread(pg, nx, ny, ppc, kind, species):
    with start(pg, nx, ny, ppc, kind, species, 0.2, 7) as c:
        c.sort()
        for moved in (False, True):
            for scheme in (NGP, CIC, TSC, ESK):
                got = []
                for order in (AUTO, ATOMIC):
                    c.set_order(order)
                    c.deposit(scheme, dt=1.0, download=False)
                    got.append(c.rho_fixed())
                assert got[0][1] == got[1][1]
                assert np.array_equal(got[0][0], got[1][0]), (moved, scheme)
            if not moved:
                c.push(0.3)  # between sorts: some particles have left their cell


@pytest.mark.parametrize("vth", [0.02, 0.3])  # few and many particles leave their cell in the move
@pytest.mark.parametrize("species", [1, 2])
@pytest.mark.parametrize("kind", ["uniform", "lattice", "clump"])
@pytest.mark.parametrize("nx,ny,ppc", SHAPES)
def test_sorted_current_equals_any_order(pg, nx, ny, ppc, kind, species, vth):
    got = []
    for sort in (True, False):
        with start(pg, nx, ny, ppc, kind, species, vth, 11) as c:
            if sort:
                c.sort()
            elif c.is_sorted():
                c.push(0.0)  # the same positions, no longer marked sorted
            c.deposit_current(1.0, download=False)
            got.append(c.current_fixed())
    for a, b in zip(*got):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("vth,dt", [(0.05, 1.0), (0.9, 1.0), (0.5, 0.0), (0.9, 3.0)])
def test_trajectory_charge_light_and_cell_paths(pg, vth, dt):
    """The sample sends the first case down the light path and the others (most
    particles leave their cell, none moves, moves of several cells) to the cells."""
    with start(pg, 70, 34, 40, "uniform", 1, vth, 3) as c:
        c.sort()
        got = []
        for order in (AUTO, ATOMIC):
            c.set_order(order)
            c.deposit(ESK, dt=dt, download=False)
            got.append(c.rho_fixed()[0])
        assert np.array_equal(*got)
