"""Gather, push and both around the counts where a thread takes one particle or two,
odd counts among them: each particle's result does not depend on how many there are."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NX, NY = 48, 40
SM = 152
COUNTS = [1, 2, 3, 255, 257, SM * 256 - 1, SM * 256, SM * 256 + 1, SM * 4096, SM * 4096 + 1, SM * 4096 + 512]


def moved(pg, what, p, m, n):
    with pg.Context(NX, NY, float(NX), float(NY), n) as c:
        c.upload(*(a[:n] for a in p), None if m is None else m[:n])
        rng = np.random.default_rng(4)
        c.set_fields(*(rng.normal(size=NX * NY) for _ in range(3)))
        getattr(c, what)(0.3)
        out = c.device_layout()
    return np.stack([out["cell"].astype(np.float64)] + [out[k].astype(np.float64) for k in ("xr", "yr", "vx", "vy")])


@pytest.mark.parametrize("masses", [False, True])
@pytest.mark.parametrize("what", ["gather", "push", "gather_push"])
def test_result_does_not_depend_on_the_count(pg, what, masses):
    rng = np.random.default_rng(1)
    n = max(COUNTS)
    p = rng.random(n) * NX, rng.random(n) * NY, rng.choice([-1.0, 1.0], n), rng.normal(size=n), rng.normal(size=n)
    p[2][0] = 1.0
    m = rng.choice([0.5, 2.0], n) if masses else None
    whole = moved(pg, what, p, m, n)
    for k in COUNTS[:-1]:
        assert np.array_equal(moved(pg, what, p, m, k), whole[:, :k]), k
