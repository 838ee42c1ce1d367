"""The sorted current evaluates every particle in full where many of them leave their
cell (chosen on the device from a sample, on grids that fill the GPU), and lists the
leaving ones elsewhere. Both give the any-order kernel's grids bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NX, NY = 210, 130  # more than a warp of 32 cells for every scheduler; no tile divides it


def particles(kind, nx, ny, ppc, species, vth, seed):
    rng = np.random.default_rng(seed)
    n = nx * ny * ppc
    x, y = rng.random(n) * nx, rng.random(n) * ny
    if kind == "clump":  # one cell's range takes many runs of 64
        m = n // 2
        x[:m], y[:m] = 32.0 + rng.random(m), 7.0 + rng.random(m)
    vx, vy = np.clip(rng.normal(0, vth, (2, n)), -0.95, 0.95)
    vx[: n // 16] = 0.0
    q = np.full(n, -1.5) if species == 1 else rng.choice([-1.0, 2.0, 0.25], n)
    return x, y, q, vx, vy


def current(pg, nx, ny, p, sort):
    with pg.Context(nx, ny, float(nx), float(ny), len(p[0])) as c:
        c.upload(*p)
        if sort:
            c.sort()
        elif c.is_sorted():
            c.push(0.0)
        c.deposit_current(1.0, download=False)
        return c.current_fixed(), c.test_device_choices()["current_full"]


# fractions that leave their cell: 0.05, 0.28, 0.35, 0.52 and 0.68, each more than three
# standard deviations of a sample of 1,024 off the rule's line
@pytest.mark.parametrize("vth,ppc,full", [(0.03, 8, 0), (0.03, 40, 0), (0.4, 1, 0), (0.2, 40, 1), (0.25, 40, 1), (0.6, 3, 1),
                                          (0.6, 8, 1)])
@pytest.mark.parametrize("species", [1, 2])
@pytest.mark.parametrize("kind", ["uniform", "clump"])
def test_choice_and_grids(pg, kind, species, vth, ppc, full):
    p = particles(kind, NX, NY, ppc, species, vth, 5)
    a, chose = current(pg, NX, NY, p, True)
    b, _ = current(pg, NX, NY, p, False)
    ex, ey = p[0] % 1.0 + p[3], p[1] % 1.0 + p[4]
    leave = np.mean((ex < 0.0) | (ex >= 1.0) | (ey < 0.0) | (ey >= 1.0))
    assert chose == full == (leave >= 0.1 + 0.58 / ppc**0.5)
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1]) and a[2:] == b[2:]


@pytest.mark.parametrize("nx,ny,ppc", [(64, 64, 20), (1, 1, 300), (33, 9, 2)])
def test_small_grids_list(pg, nx, ny, ppc):
    p = particles("uniform", nx, ny, ppc, 1, 0.6, 6)
    a, chose = current(pg, nx, ny, p, True)
    b, _ = current(pg, nx, ny, p, False)
    assert chose == 0
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


def test_a_tile_beyond_its_accumulators(pg):
    """More than 2^22 particles in one cell, all moving the same way: the sums of 64 would
    overflow the tile's words."""
    rng = np.random.default_rng(8)
    n, extra = (1 << 22) + 5000, NX * NY
    x = np.concatenate([40.0 + 0.5 * rng.random(n), rng.random(extra) * NX])
    y = np.concatenate([9.0 + 0.5 * rng.random(n), rng.random(extra) * NY])
    v = np.full(n + extra, 0.9)
    p = x, y, np.full(n + extra, 1.0), v, v
    a, chose = current(pg, NX, NY, p, True)
    b, _ = current(pg, NX, NY, p, False)
    assert chose == 1
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


def test_a_move_of_a_cell_is_refused_either_way(pg):
    for vth in (0.02, 0.6):
        p = particles("uniform", NX, NY, 4, 1, vth, 9)
        p[3][1234] = 1.5
        with pg.Context(NX, NY, float(NX), float(NY), len(p[0])) as c:
            c.upload(*p)
            c.sort()
            with pytest.raises(pg.PicError) as e:
                c.deposit_current(1.0)
            assert e.value.code == -6  # PIC_ERR_COURANT


@pytest.mark.parametrize("nx,ny", [(300, 211), (64, 40)])
def test_sparse_sets(pg, nx, ny):
    """Less than a particle per two cells: the any-order kernel, sorted or not. With
    particles of no charge up to a particle per cell the cell kernels take the same set."""
    rng = np.random.default_rng(4)
    m, n = nx * ny // 3, nx * ny
    x, y = rng.random(n) * nx, rng.random(n) * ny
    q = np.where(np.arange(n) < m, rng.choice([-1.0, 2.0], n), 0.0)
    vx, vy = np.clip(rng.normal(0, 0.4, (2, n)), -0.95, 0.95)
    few, _ = current(pg, nx, ny, (x[:m], y[:m], q[:m], vx[:m], vy[:m]), True)
    all_, _ = current(pg, nx, ny, (x, y, q, vx, vy), True)
    assert np.array_equal(few[0], all_[0]) and np.array_equal(few[1], all_[1])
