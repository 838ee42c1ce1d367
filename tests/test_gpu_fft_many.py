"""The FFT Poisson solve on grids with many transforms along one side or both: each
length there takes the kernels for many transforms, where the same length on a smaller
grid takes those for few. Same comparison and tolerance as test_gpu_fft.py."""
import pytest

from test_gpu_fft import test_solve_matches_numpy as solve_matches_numpy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(32, 2048), (64, 2048), (128, 2048), (256, 2048), (512, 2048), (1024, 2048),
                                   (2048, 16), (2048, 32), (2048, 64), (2048, 256), (2048, 512), (2048, 1024)])
def test_many_transforms(pg, nx, ny):
    solve_matches_numpy(pg, nx, ny, None, None)
