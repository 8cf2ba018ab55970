"""The separable blur against SciPy in float64, at kernel sizes and planes around its tiles.

Tolerance: each of the two passes accumulates K products in float32 (K rounding errors of at most 2^-24
of the sum of magnitudes, S = sum |w| max |a|), its factors are rounded once, and the factors stand for the
weights to within 2^-22 S (scars.outer_factors): (2 K + 6) 2^-24 S + 2^-22 S.
"""
import numpy as np
import pytest
import torch
from scipy.signal import convolve2d, fftconvolve

pytestmark = pytest.mark.gpu

CASES = [(17, 23, 8), (64, 64, 9), (65, 33, 25), (63, 513, 10), (130, 515, 41), (300, 70, 120), (5, 40, 120),
         (70, 1025, 64), (600, 520, 512)]


@pytest.mark.parametrize("H,W,K", CASES)
def test_separable_blur_matches_scipy(H, W, K):
    from cardiax_gb300 import scars
    rng = np.random.default_rng(H + W + K)
    a = rng.standard_normal((H, W)).astype(np.float32)
    w = scars.gaussian_weights(K, np.float32(max(1.5, K * rng.uniform(0.15, 0.6))))
    assert scars.outer_factors(w) is not None
    ref = fftconvolve(a.astype(np.float64), w.astype(np.float64), "full")
    s = (K - 1) // 2
    ref = ref[s:s + H, s:s + W]
    if H * W * K * K < 2e7:
        np.testing.assert_allclose(ref, convolve2d(a.astype(np.float64), w.astype(np.float64), "same"), atol=1e-12)
    tol = ((2 * K + 6) * 2.0 ** -24 + 2.0 ** -22) * np.abs(w.astype(np.float64)).sum() * np.abs(a).max()
    got = scars.blur_same(torch.as_tensor(a).cuda(), w).cpu().numpy()
    assert np.abs(got - ref).max() <= tol
    got = scars.blur_same(torch.as_tensor(a).cuda(), w, one_minus=True).cpu().numpy()
    assert np.abs(got - (1.0 - ref)).max() <= tol + 2.0 ** -24 * (1 + np.abs(ref).max())


def test_weights_of_no_outer_product_take_the_direct_sum():
    from cardiax_gb300 import scars
    rng = np.random.default_rng(1)
    for w in (rng.random((20, 20)).astype(np.float32), np.zeros((20, 20), np.float32),
              np.full((20, 20), np.nan, np.float32)):
        assert scars.outer_factors(w) is None
