"""Ensemble members against the same runs advanced alone through pic_gpu_run: after
one step (its first gather sees E = 0) positions and rho equal bit for bit, and phi,
whose solves are different transforms and factors, to FP64 rounding."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DT = 0.1


def alone(pg, st0, info):
    n, ppc = info["N"], info["ppc"]
    count = len(st0["x"])
    with pg.Context(n, n, float(n), float(n), count) as c:
        c.upload(st0["x"], st0["y"], np.full(count, -1.0 / ppc), st0["vx"], st0["vy"], np.full(count, 1.0 / ppc))
        c.run(1, scheme=1, dt=DT, background=1.0, sort_interval=0, use_graph=False, poisson=0)
        return c.download(), c.rho().ravel(), c.fields()[0].ravel()


# sizes of the library's own transforms (both radices) and of cuFFT's, one member or several of a size
@pytest.mark.parametrize("members", [
    [(6, 16, 1), (8, 64, 1), (16, 4, 2), (32, 16, 3), (64, 4, 4), (64, 16, 5), (96, 4, 6), (96, 16, 7)],
    [(256, 4, 1), (256, 16, 2), (512, 4, 3)],
    [(1024, 2, 1), (2048, 1, 2)],
])
def test_members_equal_single_runs_to_the_solve(pg, members):
    with pg.Ensemble(members, dt=DT, sort_interval=0, use_graph=False) as e:
        start = [e.download_run(r) for r in range(len(members))]
        infos = [e.info(r) for r in range(len(members))]
        e.run(1)
        after = [e.download_run(r) for r in range(len(members))]
    for a, s, i in zip(after, start, infos):
        p, rho, phi = alone(pg, s, i)
        assert np.array_equal(a["x"], p["x"]) and np.array_equal(a["y"], p["y"])
        assert np.array_equal(a["rho"], rho)
        # both FP64: a few roundings per butterfly level of either
        assert np.linalg.norm(a["phi"] - phi) <= 8 * 2.3e-16 * np.log2(phi.size) * np.linalg.norm(phi)
