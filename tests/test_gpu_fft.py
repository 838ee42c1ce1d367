"""The FFT Poisson solve against numpy's FP64 transforms: sides that this
library's transforms take (every radix chain, both sides' largest and smallest)
and sides that go to cuFFT."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIDES = [(8, 8), (16, 8), (8, 32), (64, 64), (128, 16), (32, 256), (512, 64), (64, 1024), (2048, 8), (16, 2048),
         (256, 512), (1024, 128), (4, 64), (64, 4), (48, 64), (30, 21), (4096, 8)]


@pytest.mark.parametrize("lx,ly", [(1.0, 3.0), (None, None)])
@pytest.mark.parametrize("nx,ny", SIDES)
def test_solve_matches_numpy(pg, nx, ny, lx, ly):
    lx, ly = (lx, ly) if lx else (float(nx), float(ny))
    rho = np.random.default_rng(nx + ny).normal(size=(ny, nx))
    with pg.Context(nx, ny, lx, ly, 1) as c:
        for _ in range(2):  # the second solve reuses the tables; rho is left as it was
            c.set_rho(rho.reshape(-1))
            c.poisson_fft()
            phi, ex, ey = (f.reshape(ny, nx) for f in c.fields())
            assert np.array_equal(c.rho().reshape(ny, nx), rho)
    dx, dy = lx / nx, ly / ny
    kx = 2 * np.pi * np.fft.rfftfreq(nx, dx)[None, :]
    ky = 2 * np.pi * np.fft.fftfreq(ny, dy)[:, None]
    k2 = kx * kx + ky * ky
    k2[0, 0] = 1.0
    spec = np.fft.rfft2(rho * dx * dy) / k2
    spec[0, 0] = 0.0
    want = np.fft.irfft2(spec, s=(ny, nx))
    # both FP64: a few roundings per butterfly level of either
    tol = 8 * 2.3e-16 * np.log2(nx * ny) * np.linalg.norm(want)
    assert np.linalg.norm(phi - want) <= tol
    assert np.allclose(ex, -(np.roll(phi, -1, 1) - phi) / dx, rtol=0, atol=1e-15 * np.max(np.abs(phi)) / dx)
    assert np.allclose(ey, -(np.roll(phi, -1, 0) - phi) / dy, rtol=0, atol=1e-15 * np.max(np.abs(phi)) / dy)
