"""The two-pass column transform (launches of at least 1200 columns) against the
multi-pass one (smaller launches) for every pair of register radices, the last
partial column group included.

Both are FP32 transforms of the same numbers: the same tolerances as between
two FFT plans, 1e-6 of the statistic and 1e-4 of the largest gradient entry.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# lengths R1 R2 that between them use every radix in both passes
LENGTHS = [16, 20, 24, 28, 30, 32, 36, 40, 42, 50, 56, 60, 64, 70, 72, 80, 90, 100, 108, 112, 126, 144, 150, 162, 180, 196,
           210, 224, 240, 250, 256, 270, 294, 300, 320, 324, 336, 360, 392, 400, 420, 432, 448, 480, 486, 500, 504, 540,
           560, 576, 588, 600, 630, 640, 672, 700, 720, 756, 768, 784, 800, 810, 840, 864, 896, 900, 960, 980, 1008, 1024,
           1050, 1080, 1120, 1152, 1260, 1296, 1344]


@pytest.mark.parametrize("length", LENGTHS)
def test_against_the_multi_pass_columns(gpu, length):
    rng = np.random.default_rng(length)
    P = 7
    rows, cols = length - P + 1, 21 + length % 5
    m = gpu.ModelObject()
    m.add_function("Exponential", True)
    m.add_function("FlatSky")
    m.finish_functions()
    m.set_autotune(False)
    psf = rng.uniform(0.1, 1.0, (P, P))
    m.add_psf(psf)
    data = rng.uniform(50.0, 60.0, (rows, cols))
    m.add_image_data(data)
    m.add_image_characteristics(2.0, 3.0, 1.0, 1, 0.0)
    assert m.final_setup() == 0
    m.set_fft_plan(0, 0)
    p = np.array([cols / 2 + 0.3, rows / 2 + 0.2, 30.0, 0.3, 40.0, 4.0 + rows / 9.0, 10.0])
    P0 = p * (1 + rng.uniform(-0.1, 0.1, (96, 7)))
    S, G = m.batch_statistic_and_gradient(P0)
    assert m.fft_plan()[1] == length and (m.fft_plan()[0] // 2 + 1) * 96 >= 1200
    for b in (0, 95):
        s, g = m.statistic_and_gradient(P0[b])
        assert abs(S[b] - s) <= 1e-6 * abs(s)
        assert np.max(np.abs(G[b] - g)) <= 1e-4 * np.max(np.abs(g))
