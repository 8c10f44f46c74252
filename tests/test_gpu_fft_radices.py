"""The shared-memory column transform over its radices (24, 16, 12, 9, 8, 7, 5, 4, 3, 2 in first, middle
and last passes), block widths, grids whose row count is no multiple of the bank swizzle's runs, and read columns at odd
starts: the moment planes equal numpy's unnormalised inverse 2-D DFT of the gridded planes on the columns the
recombination reads. FP32 transforms of up to six passes: 2e-6 relative L2, as in test_gpu_fft.py."""
import numpy as np
import pytest

from svdimager_b200 import api
from tests.conftest import snapshot

pytestmark = pytest.mark.gpu

FFT_TOL = 2e-6


@pytest.mark.parametrize("N,sigma,G_expect,K", [
    (28, 1.5, 42, 1), (40, 1.5, 60, 1), (64, 1.5, 96, 2), (80, 1.5, 120, 1), (256, 1.5, 384, 3), (1120, 1.5, 1680, 1),
    (1024, 1.5, 1536, 1), (2048, 1.5, 3072, 1), (1920, 1.5, 2880, 1), (33, 1.5, 50, 3), (84, 1.5, 126, 1),
    (64, 1.75, 112, 2), (180, 1.5, 270, 1), (192, 1.5, 288, 8),
    (101, 1.5, 152, 1), (320, 1.5, 480, 1), (480, 1.5, 720, 1), (500, 1.5, 750, 1), (768, 1.5, 1152, 1),
    (1000, 1.5, 1500, 1), (1080, 1.5, 1620, 1), (1440, 1.5, 2160, 1), (1536, 1.5, 2304, 1), (2100, 1.5, 3150, 1)])
def test_moments_are_the_inverse_dft_of_the_grid(cuda_device, N, sigma, G_expect, K):
    s = snapshot("small", n_rows_limit=3000, nchan=8)
    with api.Engine(keep_grid=1, sigma=sigma, k_rule=api.KRULE_FIXED, fixed_k=K) as e:
        e.image(s, N, 4e-4 * 256 / N)
        G = e.stats()["grid_size"]
        grid = e.buffer(api.BUF_GRID).reshape(K, G, G)
        mom = e.buffer(api.BUF_MOMENTS).reshape(K, G, G)
    assert G == G_expect
    c0 = G // 2 - N // 2
    want = (np.fft.ifft2(grid.astype(np.complex128), axes=(1, 2)) * (G * G))[:, :, c0:c0 + N]
    got = mom[:, :, c0:c0 + N].astype(np.complex128)
    assert np.linalg.norm(got - want) <= FFT_TOL * np.linalg.norm(want)
