"""Energies of an ensemble's runs against FP64 sums of the runs' particles and
fields: runs of less than one block of either sum, and of several."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_energies_match_fp64_sums(pg):
    # 16 particles; 3,600 (chains of unequal length); 1,228,800 (two kinetic blocks, 4,096 field cells)
    runs = [(2, 4, 1), (30, 4, 2), (64, 300, 3), (66, 2, 4)]
    with pg.Ensemble(runs, sort_interval=2) as e:
        fe, ke = e.run(3)
        for r in range(len(runs)):
            n, ppc = e.info(r)["N"], e.info(r)["ppc"]
            d = e.download_run(r)
            phi = d["phi"].reshape(n, n)
            ex, ey = phi - np.roll(phi, -1, 1), phi - np.roll(phi, -1, 0)
            want = 0.5 * np.sum(ex * ex + ey * ey)
            assert abs(fe[2, r] - want) <= 1e-12 * want
            want = 0.5 / ppc * np.sum(d["vx"] ** 2 + d["vy"] ** 2)
            # FP32 chains of at most 4,096 positive terms, three roundings a term, and the FP32 mass
            assert abs(ke[2, r] - want) <= (4096 + 4) * 2.0 ** -24 * want
