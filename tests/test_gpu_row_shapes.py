"""The row kernels' split of lines among warps, and the gradient's factored sums,
against the forward-mode pass, which evaluates every derivative pixel by pixel.

Both evaluate in FP32 (rounding 6e-8 per pixel, FFT noise a few times that of
the largest pixel): 2e-6 of the statistic, 2e-4 of the largest gradient entry.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PAR = {"Sersic": [30.0, 0.3, 2.0, 20.0, 4.0], "Exponential": [60.0, 0.4, 15.0, 6.0],
       "GaussianRing": [10.0, 0.2, 8.0, 9.0, 2.0], "Moffat": [40.0, 0.1, 200.0, 4.0, 3.0],
       "Gaussian": [70.0, 0.2, 90.0, 2.0], "TiltedSkyPlane": [20.0, 0.05, -0.03]}


# lines that divide the warps and lines that do not, one warp, more warps than
# a line has runs; 9 x 9 PSF: windows of 46 and 37 rows leave a remainder
@pytest.mark.parametrize("shape", [(1, 32), (1, 256), (2, 64), (2, 96), (3, 96), (3, 256), (4, 64), (4, 128), (4, 1024)])
@pytest.mark.parametrize("region", [0, 5])
@pytest.mark.parametrize("cols,rows", [(47, 38), (70, 29)])
def test_shape(gpu, shape, region, cols, rows):
    rng = np.random.default_rng(7)
    m = gpu.ModelObject()
    p = [24.3, 18.8]
    for i, f in enumerate(PAR):
        m.add_function(f, i == 0)
        p += PAR[f]
    m.finish_functions()
    m.set_autotune(False)
    y, x = np.mgrid[-4:5, -4:5]
    m.add_psf(np.exp(-(x ** 2 + 0.7 * y ** 2) / 4.0))
    m.add_image_data(rng.uniform(40.0, 90.0, (rows, cols)))
    m.add_image_characteristics(2.0, 3.0, 1.0, 1, 0.0)
    if region:
        k = region
        yy, xx = np.mgrid[-4 * k:4 * k + 1, -4 * k:4 * k + 1] / k
        m.add_oversampled_psf(np.exp(-(xx ** 2 + 0.7 * yy ** 2) / 4.0), k, (15, 30, 10, 25))
    assert m.final_setup() == 0
    m.set_launch_shape(shape[0], shape[1], 0, 0)
    v = np.array(p)
    S, _, b = m.jtwj(v)
    s, g = m.statistic_and_gradient(v)
    assert abs(S - s) <= 2e-6 * abs(s)
    assert np.max(np.abs(2 * b - g)) <= 2e-4 * np.max(np.abs(g))
    s3, g3 = m.batch_statistic_and_gradient(np.stack([v, 1.02 * v, v]))
    assert abs(s3[0] - s) <= 2e-6 * abs(s) and s3[0] == s3[2] and np.array_equal(g3[0], g3[2])
    assert np.max(np.abs(g3[0] - g)) <= 2e-4 * np.max(np.abs(g))
