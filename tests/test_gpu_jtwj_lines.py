"""The model that the J^T W J pass forms from its derivative images, against the
statistic and the adjoint gradient of the forward pass.

Both evaluate in FP32 (rounding 6e-8 per pixel, FFT noise a few times that of
the largest pixel): 2e-6 of the statistic, 2e-4 of the largest entry of
2 J^T dev against the gradient, as the tests of the two passes allow.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PAR = {"Sersic": [30.0, 0.3, 2.0, 20.0, 4.0], "Exponential": [60.0, 0.4, 15.0, 6.0],
       "GaussianRing": [10.0, 0.2, 8.0, 9.0, 2.0], "Moffat": [40.0, 0.1, 200.0, 4.0, 3.0],
       "Gaussian": [70.0, 0.2, 90.0, 2.0], "FlatSky": [30.0], "TiltedSkyPlane": [20.0, 0.05, -0.03],
       "PointSource": [900.0]}


@pytest.mark.parametrize("functions,zero,region,stat", [
    (["Sersic", "Exponential", "GaussianRing", "Moffat", "Gaussian", "FlatSky"], False, 0, "chi2"),
    (["Sersic", "Exponential", "FlatSky"], True, 0, "model"),      # a zero amplitude
    (["Sersic", "TiltedSkyPlane", "PointSource"], False, 0, "pmlr"),
    (["Sersic", "Exponential", "TiltedSkyPlane", "FlatSky"], False, 5, "chi2"),
    (["Gaussian", "FlatSky"], False, 3, "chi2"),
    (["FlatSky"], False, 0, "chi2"),                               # no derivative line but the centre's
    (["TiltedSkyPlane"] * 31 + ["FlatSky"], False, 0, "chi2"),     # more linear parameters than the list holds
])
def test_statistic_and_gradient(gpu, functions, zero, region, stat):
    rng = np.random.default_rng(3)
    cols, rows = 47, 38
    p = [24.3, 18.8]
    for f in functions:
        q = list(PAR[f])
        if f == "TiltedSkyPlane" and len(functions) > 4:
            q = [2.0, 0.004, -0.003]
        if zero and f == "Exponential":
            q[2] = 0.0
        p += q
    p = np.array(p)
    m = gpu.ModelObject()
    for i, f in enumerate(functions):
        m.add_function(f, i == 0)
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
    if stat == "model":
        m.use_model_errors()
    if stat == "pmlr":
        m.use_pmlr()
    assert m.final_setup() == 0
    for scale in (1.0, 1.03):
        v = p * scale
        S, A, b = m.jtwj(v)
        s, g = m.statistic_and_gradient(v)
        assert abs(S - s) <= 2e-6 * abs(s)
        assert np.max(np.abs(2 * b - g)) <= 2e-4 * np.max(np.abs(g))
        assert np.all(np.isfinite(A)) and np.allclose(A, A.T)
