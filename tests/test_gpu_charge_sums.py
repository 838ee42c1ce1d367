"""The charge sums of the diagnostics are made once per particle set, not in every
replay of a captured step: a run's first steps after an upload launch no more kernels
per step than those of a later run, and report the same charges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scheme", [1, 3])
@pytest.mark.parametrize("sort_interval", [0, 3])
@pytest.mark.parametrize("graph", [True, False])
def test_steps_after_an_upload_launch_no_more_than_later_ones(pg, graph, sort_interval, scheme):
    nx, ny, n = 32, 48, 6000
    rng = np.random.default_rng(5)
    x, y = rng.random(n) * nx, rng.random(n) * ny
    q = rng.choice([-1.0, 2.0], n) / n
    cfg = dict(scheme=scheme, dt=0.1, background=1.0 / (nx * ny), sort_interval=sort_interval, use_graph=graph)

    def launches(c, steps):
        before = c.launch_count()
        hist = c.run(steps, **cfg)
        return c.launch_count() - before, hist

    with pg.Context(nx, ny, float(nx), float(ny), n) as c:
        c.upload(x, y, q)
        c.run(2, **cfg)  # the context's tables are made
        per_step, charges = [], []
        for fresh in (True, False):
            counts = []
            for steps in (6, 12):
                if fresh:
                    c.upload(x, y, q, 0.1 * rng.normal(size=n), 0.1 * rng.normal(size=n))
                count, hist = launches(c, steps)
                counts.append(count)
                charges.append(hist[:, 1])
            per_step.append(counts[1] - counts[0])
        assert per_step[0] == per_step[1]
        want = np.sum(q.astype(np.float32).astype(np.float64))
        for t in charges:
            assert np.allclose(t, want, rtol=1e-6) and np.all(t == t[0])
