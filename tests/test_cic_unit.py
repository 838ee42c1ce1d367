"""The CIC deposit's short form for a particle of charge +-max|q| (cic_unit in
pic-deposition_gb300/csrc/pic_internal.cuh), checked on the CPU with exact float32
emulation against the general rule: A = +-2^24, node (j, i) carries
rint((A * Y[j]) * X[i]), and the node of largest weight A minus the others.
Whole numbers: equality, no tolerance."""
import numpy as np

A = 1 << 24
ONE, HALF = np.float32(1), np.float32(0.5)


def general(x, y, sign):
    X, Y = [ONE - x, x], [ONE - y, y]
    bi, bj = (x > HALF).astype(int), (y > HALF).astype(int)
    q = np.float32(sign * A)
    v = np.array([[np.rint((q * Y[j]) * X[i]).astype(np.int64) for i in (0, 1)] for j in (0, 1)])
    k = np.arange(x.size)
    v[bj, bi, k] = 0
    v[bj, bi, k] = sign * A - v.sum(axis=(0, 1))
    return v


def short(x, y):
    bits = lambda f: f.astype(np.float32).view(np.int32).astype(np.int64)
    bias = 2 * 0x3F000000 + (1 << 23)
    xs, ys = np.minimum(x, ONE - x), np.minimum(y, ONE - y)
    xb, yb = ONE - xs, ONE - ys
    sx, sy = np.where(x > HALF, 1, -1), np.where(y > HALF, 1, -1)
    p, q, s = bits(yb * xs + HALF), bits(ys * xb + HALF), bits(ys * xs + HALF)
    return sy * (q + s - bias), sx * (p + s - bias), -sx * sy * (p + q - bias)


def test_three_sums_equal_the_general_nodes():
    rng = np.random.default_rng(11)
    ulp = np.float32(2.0**-24)
    edge = np.array([0, ulp, 2 * ulp, 3 * ulp, 2.0**-13, 0.25, 0.5 - ulp, 0.5, 0.5 + 2 * ulp, 0.75, 1 - 2 * ulp, 1 - ulp, 1,
                     2.0**-60, 2.0**-149, 1e-30], np.float32)
    ex, ey = [g.ravel() for g in np.meshgrid(edge, edge)]
    n = 400_000
    rx, ry = rng.random(n).astype(np.float32), rng.random(n).astype(np.float32)
    tx, ty = np.float32(2.0) ** -rng.integers(0, 40, n).astype(np.float32) * rx, np.float32(1) - ry * np.float32(1e-5)
    x, y = np.concatenate([ex, rx, tx, ty]), np.concatenate([ey, ry, ty, tx])
    row0, col0, diag = short(x, y)
    for sign in (1, -1):
        v = general(x, y, sign)
        assert np.array_equal(v[0, 0] + v[0, 1], sign * (A // 2 + row0))
        assert np.array_equal(v[0, 0] + v[1, 0], sign * (A // 2 + col0))
        assert np.array_equal(v[0, 0] + v[1, 1], sign * (A // 2 + diag))
