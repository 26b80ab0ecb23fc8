"""The plain FP64 path's few-instruction profiles, shared subsample lattice,
valid-window regions and batched finite differences against the oracle.

Tolerances.  A profile I = A 2^x is formed from a rounded exponent, so its
relative error is |ln(I/A)| times a few units of 2^-53 plus a few units; the
reference's own expressions have errors of the same form.  Eight units each
are allowed: 1e-15 (8 + 8 |ln(I/A)|).  After an FFT: 1e-10 normwise, as
elsewhere.  Finite differences divide the rounding noise of the statistic's
terms (2^-52 of the image's largest value per pixel after the FFT) by steps of
1.5e-8: 1e-5 of the gradient's norm.
"""
import numpy as np
import pytest

from helpers import normwise

pytestmark = pytest.mark.gpu


def _images(gpu, oracle_mod, functions, params, cols, rows, subsampling=True, psf=None, regions=()):
    out = []
    for cls in (gpu.ModelObject, oracle_mod.OracleModel):
        m = cls()
        for i, f in enumerate(functions):
            m.add_function(f, i == 0, subsampling=subsampling)
        m.finish_functions()
        if psf is not None:
            m.add_psf(psf)
        m.setup_model_image(cols, rows)
        for r in regions:
            m.add_oversampled_psf(*r)
        m.create_model_image(np.array(params, dtype=float))
        out.append(np.array(m.get_model_image()))
    return out


# a profile's parameters after X0, Y0, and its amplitude
PROFILES = [
    ("Sersic", [33.0, 0.4, 0.3, 25.0, 9.0], 25.0), ("Sersic", [90.0, 0.0, 1.0, 3.0, 0.8], 3.0),
    ("Sersic", [120.0, 0.95, 4.0, 60.0, 2.5], 60.0), ("Sersic", [10.0, 0.2, 10.0, 1.0, 300.0], 1.0),
    ("Exponential", [33.0, 0.6, 20.0, 7.0], 20.0), ("Exponential", [0.0, 0.0, 20.0, 0.3], 20.0),
    ("Exponential", [71.0, 0.3, 1e-30, 4e5], 1e-30),
    ("GaussianRing", [12.0, 0.3, 5.0, 20.0, 2.0], 5.0), ("GaussianRing", [12.0, 0.0, 5.0, 0.0, 30.0], 5.0),
    ("Moffat", [45.0, 0.1, 300.0, 4.0, 3.1], 300.0), ("Moffat", [45.0, 0.5, 300.0, 0.9, 1.01], 300.0),
    ("Gaussian", [70.0, 0.3, 90.0, 2.2], 90.0), ("Gaussian", [70.0, 0.0, 90.0, 0.4], 90.0),
    ("Gaussian", [70.0, 0.8, 90.0, 150.0], 90.0),
]


@pytest.mark.parametrize("subsampling", [True, False])
@pytest.mark.parametrize("name,p,amp", PROFILES)
def test_profiles_pixelwise(gpu, oracle_mod, name, p, amp, subsampling):
    g, o = _images(gpu, oracle_mod, [name], [40.3, 29.8] + p, 97, 70, subsampling)
    far = o > 1e-280
    x = np.abs(np.log(np.where(far, o, amp) / amp))
    rel = np.abs(g - o) / np.where(far, o, 1.0)
    assert np.all(rel[far] <= 1e-15 * (8.0 + 8.0 * x[far]))
    assert np.all(np.abs(g[~far]) <= 1e-279)


@pytest.mark.parametrize("p", [[20.0, -0.5, 2.0, 10.0, 5.0], [20.0, 1.5, 2.0, 10.0, 5.0]])
def test_axis_ratios_outside_the_form(gpu, oracle_mod, p):
    """q >= 1 and q < 0 take the reference's expressions or the form; either way the same image."""
    g, o = _images(gpu, oracle_mod, ["Sersic"], [20.3, 19.8] + p, 45, 40)
    assert np.all(np.abs(g - o) <= 1e-13 * np.abs(o))


def _moffat(n, m, fwhm):
    y, x = np.mgrid[0:m, 0:n]
    r2 = (x - (n - 1) / 2) ** 2 + (y - (m - 1) / 2) ** 2
    p = (1 + r2 / fwhm ** 2) ** -3.0
    return p / p.sum()


BULGE = [["Sersic", "Exponential", "Gaussian", "FlatSky"],
         [30.4, 25.7, 20.0, 0.3, 2.0, 15.0, 5.0, 60.0, 0.5, 8.0, 9.0, 5.0, 0.2, 30.0, 0.7, 4.0]]


# scales with (2, 4, 5) and without (3) the shared lattice; odd, even and
# unequal PSF sides; regions of unequal sides (the reference's row count comes
# from the column count: fewer rows replaced, or rows beyond the region's own)
@pytest.mark.parametrize("scale,psf,region", [
    (5, (15, 15), (24, 37, 19, 32)), (4, (9, 9), (1, 8, 1, 8)), (2, (8, 8), (50, 60, 40, 50)),
    (3, (11, 11), (24, 37, 19, 32)), (5, (15, 25), (24, 37, 19, 32)), (3, (21, 15), (20, 33, 15, 28)),
    (2, (9, 9), (20, 25, 15, 28)), (1, (7, 7), (24, 37, 19, 32))])
def test_regions(gpu, oracle_mod, scale, psf, region):
    reg = (_moffat(*psf, 2.0 * scale), scale, region)
    g, o = _images(gpu, oracle_mod, *BULGE, 61, 52, psf=_moffat(9, 11, 2.0), regions=[reg])
    assert normwise(g, o) < 1e-10


@pytest.mark.parametrize("stat", ["chi2", "model", "cash", "sigma"])
@pytest.mark.parametrize("region", [False, True])
def test_batched_finite_differences(gpu, oracle_mod, stat, region):
    functions, p = BULGE[0], np.array(BULGE[1])
    rng = np.random.default_rng(5)
    pair, data = [], None
    for cls in (oracle_mod.OracleModel, gpu.ModelObject):
        m = cls()
        for i, f in enumerate(functions):
            m.add_function(f, i == 0, subsampling=False)  # no count jumps inside a step
        m.finish_functions()
        m.add_psf(_moffat(9, 11, 2.0))
        if data is None:
            t = oracle_mod.OracleModel()
            for i, f in enumerate(functions):
                t.add_function(f, i == 0)
            t.finish_functions()
            t.setup_model_image(61, 52)
            t.create_model_image(p * 1.05)
            data = rng.poisson(np.clip(t.get_model_image(), 0, None) + 5.0).astype(float)
        m.add_image_data(data)
        m.add_image_characteristics(2.0, 3.0, 1.0, 1, 0.0)
        if region:
            m.add_oversampled_psf(_moffat(15, 15, 6.0), 3, (24, 37, 19, 32))
        if stat == "sigma":
            m.add_error_vector(np.sqrt(data + 4.0))
        if stat == "model":
            m.use_model_errors()
        if stat == "cash":
            m.use_cash()
        assert m.final_setup() == 0
        pair.append(m)
    o, g = pair
    s, grad = g.statistic_and_gradient_fd(p)
    s0 = o.get_fit_statistic(p)
    assert abs(s - s0) <= 1e-10 * abs(s0)
    want = []
    for j in range(len(p)):
        h = 2e-5 * max(abs(p[j]), 0.1)
        q = [p.copy(), p.copy()]
        q[0][j] += h
        q[1][j] -= h
        want.append((o.get_fit_statistic(q[0]) - o.get_fit_statistic(q[1])) / (2 * h))
    want = np.array(want)
    assert np.linalg.norm(grad - want) <= 1e-5 * np.linalg.norm(want)
    # the call leaves the last step's model behind, as evaluating it last does
    last = p.copy()
    last[-1] += 1.490116e-08 * abs(last[-1])
    left = g.get_model_image()
    g.create_model_image(last)
    assert normwise(left, g.get_model_image()) < 1e-10


@pytest.mark.parametrize("n", [1.0, 2.0, 3.0, 2.5, 0.4])
def test_ferrers_indices(gpu, oracle_mod, n):
    p = [25.3, 22.8, 35.0, 70.0, 40.0, 2.0, 14.0, 0.5, 0.3, n]
    g, o = _images(gpu, oracle_mod, ["FerrersBar3D"], p, 50, 45)
    # the integrals are adaptive to 1e-6; below n = 1 the density's edge is steep
    assert np.max(np.abs(g - o)) <= 1e-12 * np.max(o)


# (0.5, 0.02, 90) holds pixels whose whole integrand is denormal, which no
# form integrates within the device's list of subintervals (refused)
@pytest.mark.parametrize("n,z0,inc", [(1.0, 2.0, 85.0), (0.5, 0.02, 89.0), (100.0, 3.0, 0.0), (3.0, 0.7, 40.0)])
def test_disk_vertical_profiles(gpu, oracle_mod, n, z0, inc):
    """Thin disks reach z / (alpha z_0) > 100, where the reference switches to
    the asymptote, and values at the bottom of the FP64 range."""
    p = [25.3, 22.8, 35.0, inc, 4.0, 6.0, n, z0]
    g, o = _images(gpu, oracle_mod, ["ExponentialDisk3D"], p, 50, 45)
    assert np.max(np.abs(g - o)) <= 1e-12 * np.max(o)
