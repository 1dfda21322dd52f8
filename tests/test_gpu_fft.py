"""The line transforms of csrc/fft.cu over every line length they are built
for, oblong grids and one-cell axes, against numpy's transforms.  Each length
has its own pass schedule (radix 8, ending 4 4 or 4), so each is run along
both axes.

Tolerance: a transform of N points has a root-mean-square error of about
eps * sqrt(log2 N) / 2 relative to the output's root mean square; the largest
of N errors is below six of those for N <= 2^20, and the twiddle products
double it at most."""
import numpy as np
import pytest

import unstaggered_pic_b200 as up

pytestmark = pytest.mark.gpu

SHAPES = ([(1 << k, 4) for k in range(0, 14)] + [(4, 1 << k) for k in range(0, 14)] +
          [(1, 1), (1, 64), (64, 1), (2, 2), (16, 8), (64, 64), (128, 512), (1024, 256)])


@pytest.mark.parametrize("nx,ny", SHAPES)
def test_transform_lengths(nx, ny):
    rng = np.random.default_rng(nx * 10007 + ny)
    z = rng.standard_normal((nx, ny)) + 1j * rng.standard_normal((nx, ny))
    tol = 6 * np.finfo(float).eps * np.sqrt(np.log2(2 * nx * ny))
    with up.Simulation(up.Config(nx=nx, ny=ny)) as sim:
        for inverse, f in ((False, np.fft.fft2), (True, np.fft.ifft2)):
            re, im = sim.fft2d(z.real, z.imag, inverse=inverse)
            ref = f(z)
            rms = np.sqrt(np.mean(np.abs(ref) ** 2))
            assert np.max(np.abs(re + 1j * im - ref)) <= tol * rms, inverse
