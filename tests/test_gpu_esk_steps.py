"""Time steps of the trajectory scheme do not sort: the sort count says so, and the
results and the particles' order are the same whatever sort is asked for."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [True, False])
def test_trajectory_steps_do_not_sort(pg, graph):
    nx, ny, n = 24, 20, 5000
    rng = np.random.default_rng(2)
    p = rng.random(n) * nx, rng.random(n) * ny, np.full(n, -1.0 / n), rng.normal(size=n), rng.normal(size=n)
    out = []
    for kw in (dict(sort_interval=0), dict(sort_interval=2), dict(sort_interval=3, sort_moved_fraction=0.01)):
        with pg.Context(nx, ny, float(nx), float(ny), n) as c:
            c.upload(*p)
            hist = c.run(7, scheme=3, dt=0.1, background=1.0 / (nx * ny), use_graph=graph, **kw)
            assert c.sort_count() == 0
            out.append((hist, c.rho(), *c.device_layout().values()))
    for o in out[1:]:
        for a, b in zip(out[0], o):
            assert np.array_equal(a, b)


def test_the_other_schemes_count_the_sorts_they_do(pg):
    n = 3000
    rng = np.random.default_rng(3)
    with pg.Context(16, 16, 16.0, 16.0, n) as c:
        c.upload(rng.random(n) * 16, rng.random(n) * 16, np.full(n, -1.0 / n), rng.normal(size=n), rng.normal(size=n))
        for scheme in (0, 1, 2):
            before = c.sort_count()
            c.run(7, scheme=scheme, dt=0.1, background=1.0 / 256, use_graph=True, sort_interval=3)
            assert c.sort_count() == before + 3
