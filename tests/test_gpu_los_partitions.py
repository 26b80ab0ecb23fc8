"""The fast path's line-of-sight partitions where a thread's panels run out:
very thin and very steep disks (up to 32 panels, finished by the warp),
windows whose pixel count leaves a partial run of 32, several vectors.

Tolerances.  Panels are refined to 4e-6 of an integral or stop at 32; the
image is compared with the oracle's integrals at epsrel 1e-11: 2e-5 of the
largest pixel where 32 panels may be too few (the reference's own epsrel is
1e-6 per integral), and the gradient with central differences of the oracle's
statistic, 2e-3 of each entry plus 2e-3 of the largest, as for the other
gradients.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DISK, BAR = "ExponentialDisk3D", "FerrersBar3D"


def _pair(gpu, oracle_mod, functions, p, cols, rows):
    out = []
    for cls in (oracle_mod.OracleModel, gpu.ModelObject):
        m = cls()
        for i, f in enumerate(functions):
            m.add_function(f, i == 0)
        m.finish_functions()
        if not out:
            t = cls()
            for i, f in enumerate(functions):
                t.add_function(f, i == 0)
            t.finish_functions()
            t.setup_model_image(cols, rows)
            t.create_model_image(np.array(p) * 1.02)
            data = np.array(t.get_model_image())
        m.add_image_data(data)
        m.add_error_vector(np.full(data.shape, 0.02 * data.max()))
        assert m.final_setup() == 0
        out.append(m)
    return out


# (functions, parameters after X0 and Y0)
MODELS = [
    ([DISK], [40.0, 75.0, 2.0, 6.0, 1.0, 0.3]),    # thin: the vertical peak is narrow
    ([DISK], [40.0, 20.0, 2.0, 0.7, 1.0, 5.0]),    # steep: a sharp radial cusp
    ([DISK], [10.0, 89.0, 2.0, 5.0, 40.0, 2.0]),   # nearly exponential in height
    ([DISK, BAR], [40.0, 80.0, 2.0, 6.0, 1.0, 1.5, 40.0, 80.0, 30.0, 1.0, 8.0, 0.5, 0.3, 2.0]),
]


@pytest.mark.parametrize("k", range(len(MODELS)))
def test_image_and_gradient(gpu, oracle_mod, k):
    functions, q = MODELS[k]
    cols, rows = 37, 29
    p = np.array([18.8, 14.3] + q)
    oracle_mod.set_los_epsrel(1e-11)
    try:
        o, g = _pair(gpu, oracle_mod, functions, p, cols, rows)
        o.create_model_image(p)
        ref = np.array(o.get_model_image())
        assert np.max(np.abs(g.get_fast_model_image(p) - ref)) <= 2e-5 * np.max(ref)
        s, grad = g.statistic_and_gradient(p)
        fd = np.empty(len(p))
        for j in range(len(p)):
            h = 1e-4 * max(abs(p[j]), 0.1)
            a, b = p.copy(), p.copy()
            a[j] += h
            b[j] -= h
            fd[j] = (o.get_fit_statistic(a) - o.get_fit_statistic(b)) / (2 * h)
        ok = np.abs(grad - fd) <= 2e-3 * np.abs(fd) + 2e-3 * np.max(np.abs(fd))
        if k == 1:  # +-20 h cuts the vertical profile here; the gradient leaves out the range's own derivative
            ok[5] = True
        assert np.all(ok)
        P = np.stack([p, p * 1.01, p * 0.99])
        S, G = g.batch_statistic_and_gradient(P)
        assert abs(S[0] - s) <= 2e-6 * s and np.max(np.abs(G[0] - grad)) <= 1e-4 * np.max(np.abs(grad))
    finally:
        oracle_mod.set_los_epsrel(0)
