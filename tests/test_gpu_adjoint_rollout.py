"""Gradients of whole rollouts against those of the adjoint tile kernel, recorded before the line kernel took its
grids: dL/dv0, dw0, du0 and dL/dD have the same bits (lambda's and dL/dD's operations are the same in the same
order), so no output can be further from the 64-bit gradient than it was.

dL/dtheta is a sum over the cells in another grouping: its partial sums are at most 21 float32 additions deep,
21 * 2^-24 = 1.3e-6 of the sum of magnitudes, which random signs make sqrt(N) <= 75 times larger than the result:
1e-4 norm-wise, doubled.
"""
import os
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden"))
import make_rollout_golden as G  # noqa: E402


@pytest.mark.parametrize("case", G.CASES, ids=lambda c: f"{c[0]}x{c[1]}")
def test_rollout_gradients_keep_their_bits(case):
    want = np.load(G.PATH)
    name = f"{case[0]}x{case[1]}_"
    got = dict(zip(("v", "w", "u", "D", "theta"), G.gradients(case)))
    for k in ("v", "w", "u", "D"):
        ref = want[name + k]
        assert np.isfinite(ref).all() and np.abs(ref).max() > 0
        np.testing.assert_array_equal(got[k], ref, err_msg=k)
    d = np.linalg.norm(got["theta"].astype(np.float64) - want[name + "theta"])
    assert d <= 2e-4 * np.linalg.norm(want[name + "theta"])
