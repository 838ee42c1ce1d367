"""The trajectory charge of freshly sorted particles with one charge: which of its two
paths the device takes follows the rule on the fraction that leaves its cell, on either
side of the line, and both give the one-particle-per-thread kernel's grid bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ESK, AUTO, ATOMIC = 3, 0, 3


def stays(r, d):
    e = r + d
    return (np.abs(d) > 0) & (np.abs(d) < 1.0) & np.where(d > 0, e <= 1.0, e >= 0.0)


# every sample (1,024 of the particles) more than three standard deviations off the line
@pytest.mark.parametrize("vth,ppc,light", [(0.05, 40, 1), (0.25, 40, 1), (0.45, 40, 0), (0.9, 40, 0), (0.35, 6, 1),
                                           (0.9, 6, 0), (0.9, 1, 1), (0.0, 40, 0)])
@pytest.mark.parametrize("charge", [1.5, -0.25])
@pytest.mark.parametrize("nx,ny", [(70, 34), (128, 40), (210, 130)])
def test_path_and_grid(pg, nx, ny, charge, vth, ppc, light):
    rng = np.random.default_rng(nx + ppc)
    n = nx * ny * ppc
    x, y = rng.random(n) * nx, rng.random(n) * ny
    vx, vy = np.clip(rng.normal(0, 1, (2, n)), -2, 2) * vth
    line = max(0.45 if nx * ny < 16384 else 0.37, 0.3 + 0.8 / ppc**0.5)
    leave = 1.0 - np.mean(stays(x % 1.0, vx) & stays(y % 1.0, vy))
    assert abs(leave - line) > 3 * 0.5 / 1024**0.5 and light == (leave < line)
    with pg.Context(nx, ny, float(nx), float(ny), n) as c:
        c.upload(x, y, np.full(n, charge), vx, vy)
        c.sort()
        got = []
        for order in (AUTO, ATOMIC):
            c.set_order(order)
            c.deposit(ESK, dt=1.0, download=False)
            got.append(c.rho_fixed())
            if order == AUTO:
                assert c.test_device_choices()["esk_light"] == light
        assert np.array_equal(got[0][0], got[1][0]) and got[0][1] == got[1][1]


@pytest.mark.parametrize("nx,ny,n", [(1, 1, 1), (1, 1, 1025), (3, 2, 7), (5, 5, 1024), (300, 200, 100)])
def test_few_particles_and_empty_cells(pg, nx, ny, n):
    rng = np.random.default_rng(n)
    x, y = rng.random(n) * nx, rng.random(n) * ny
    v = rng.normal(0, 0.3, (2, n))
    with pg.Context(nx, ny, float(nx), float(ny), n) as c:
        c.upload(x, y, np.full(n, -2.0), *v)
        c.sort()
        got = []
        for order in (AUTO, ATOMIC):
            c.set_order(order)
            for _ in range(2):  # a second deposit starts its grid anew
                c.deposit(ESK, dt=1.0, download=False)
            got.append(c.rho_fixed()[0])
        assert np.array_equal(*got)
