"""Masses of uploads read in place: stored in the conversion's pass where the first one is
not 1 or the context has held masses before, else in a pass of their own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 1537


def mass_sets():
    rng = np.random.default_rng(3)
    ones, first, last, all_ = np.ones(N), np.ones(N), np.ones(N), rng.random(N) + 1.5
    first[0], last[-1] = 2.0, 4.0
    return {"none": None, "ones": ones, "first": first, "last": last, "all": all_}


@pytest.mark.parametrize("before", ["none", "ones", "first", "last", "all"])
@pytest.mark.parametrize("then", ["none", "ones", "first", "last", "all"])
def test_masses_after_masses(pg, before, then):
    rng = np.random.default_rng(1)
    x, y, v = rng.random(N) * 16, rng.random(N) * 16, rng.normal(size=N)
    e = rng.normal(size=256)
    m = mass_sets()
    with pg.Context(16, 16, 16.0, 16.0, N) as c:
        c.upload(x, y, -np.ones(N), v, v, m[before])
        c.upload(y, x, -np.ones(N), v, v, m[then])
        want = np.ones(N) if m[then] is None else m[then].astype(np.float32)
        assert np.array_equal(c.download()["m"], want)
        launches = c.launch_count()
        c.upload(y, x, -np.ones(N), v, v, m[then])
        per_upload = c.launch_count() - launches
        assert per_upload == 2  # conversion, and the charges and keys of all: no pass for the masses
        c.set_fields(ex=e, ey=e)
        c.gather(0.1)
        got = c.device_layout()["vx"]
    with pg.Context(16, 16, 16.0, 16.0, N) as c:
        c.upload(y, x, -np.ones(N), v, v, want)
        c.set_fields(ex=e, ey=e)
        c.gather(0.1)
        assert np.array_equal(got, c.device_layout()["vx"])


def test_first_upload_with_masses_is_one_pass(pg):
    rng = np.random.default_rng(1)
    x, y = rng.random(N) * 16, rng.random(N) * 16
    with pg.Context(16, 16, 16.0, 16.0, N) as c:
        before = c.launch_count()
        c.upload(x, y, -np.ones(N), m=np.full(N, 2.0))
        assert c.launch_count() - before == 2
        assert np.all(c.download()["m"] == 2.0)
