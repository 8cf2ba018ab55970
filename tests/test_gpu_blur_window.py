"""The separable passes by their own entry point: the sum against float64 at the tile and tap remainders, and what an
infinite input reaches.

Tolerance: each pass accumulates K products in float32 (K rounding errors of at most 2^-24 of the sum of magnitudes,
S = sum |ky| sum |kx| max |a|): 2 (K + 1) 2^-24 S.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _separable(a, ky, kx):
    from cardiax_gb300 import _native as N
    from cardiax_gb300.tissue import stream_handle
    H, W = a.shape
    src, k = torch.as_tensor(a).cuda(), torch.as_tensor(np.stack((ky, kx))).cuda()
    tmp, out = torch.empty_like(src), torch.empty_like(src)
    N.call("fk_conv2d_separable", src.data_ptr(), H, W, W, k[0].data_ptr(), k[1].data_ptr(), len(ky), tmp.data_ptr(),
           W, out.data_ptr(), W, 0, stream_handle())
    return out.cpu().numpy()


@pytest.mark.parametrize("H,W,K", [(17, 23, 1), (5, 9, 7), (64, 64, 8), (65, 33, 9), (63, 513, 15), (130, 70, 16),
                                   (70, 40, 23)])
def test_separable_sum_and_its_window(H, W, K):
    rng = np.random.default_rng(H + W + K)
    a = rng.standard_normal((H, W)).astype(np.float32)
    ky, kx = (0.1 + rng.random((2, K))).astype(np.float32)
    s = (K - 1) // 2
    w = np.outer(ky.astype(np.float64), kx.astype(np.float64))
    ref = np.zeros((H + 2 * K, W + 2 * K))
    for y in range(K):
        for x in range(K):
            ref[y:y + H, x:x + W] += w[y, x] * a
    ref = ref[s:s + H, s:s + W]
    tol = 2 * (K + 1) * 2.0 ** -24 * w.sum() * np.abs(a).max()
    assert np.abs(_separable(a, ky, kx) - ref).max() <= tol
    # an infinite cell: the rows outside its window keep their values
    r, c = H // 2, W // 2
    a[r, c] = np.inf
    got = _separable(a, ky, kx)
    near = np.arange(H)
    out_of_it = (near < r - s) | (near > r - s + K - 1)
    assert np.abs(got[out_of_it] - ref[out_of_it]).max(initial=0.0) <= tol
    window = got[~out_of_it][:, max(0, c - s):c - s + K]
    assert window.size and np.isposinf(window).all()
