"""One adjoint step against float64 autodiff of the oracle, at the sizes where its tiles, one-sided
rows and partial quads can go wrong.

Tolerances.  lambda and dL/dD of a cell are sums of some 60 float32 products whose partial sums stay
within a few times the result's scale (random data, no systematic cancellation): 60 * 2^-24 = 4e-6
norm-wise, doubled.  A parameter's gradient is a float32 sum of N terms of random sign, so it is
smaller than the sum of their magnitudes by sqrt(N): relative error at most sqrt(N) times a term's
(4e-6 / 10, a term has fewer operations), 1e-4 at the largest N here (2e4 cells), doubled.
"""
import numpy as np
import pytest
import torch

import fk_torch as FT

pytestmark = pytest.mark.gpu

P4A = (3.33, 15.6, 5, 350, 80, 0.407, 9, 34, 26.5, 15, 0.45, 0.15, 0.04, 1)

# the shortest lines of the line kernel (20) and one below, every residue of H mod 2 and W mod 4, one
# and several tiles each way with full, nearly full and nearly empty last ones
SHAPES = [(19, 40), (20, 20), (21, 22), (22, 21), (23, 23), (16 + 16, 64), (33, 65), (34, 66),
          (35, 67), (48, 68), (49, 69), (20, 129), (130, 21), (81, 133), (150, 131)]


@pytest.mark.parametrize("H,W", SHAPES)
def test_adjoint_step_matches_fp64_autodiff(H, W):
    from cardiax_gb300.adjoint import Adjoint
    from cardiax_gb300.stimulus import Protocol, Stimulus
    from cardiax_gb300.tissue import Tissue
    rng = np.random.default_rng(1000 * H + W)
    f32 = np.float32
    u = rng.random((H, W)).astype(f32)
    for th in (P4A[11], P4A[12]):  # no cell on a gate: float32 and float64 take the same side
        u[np.abs(u - th) < 1e-3] += f32(4e-3)
    v, w = rng.random((2, H, W)).astype(f32)
    n = rng.standard_normal((H, W))
    D = (1e-3 * (1 + 0.2 * (n + np.roll(n, 1, 0) + np.roll(n, 1, 1)) / 3)).astype(f32)
    dense = np.zeros((H, W), f32)
    dense[H // 4:H // 2, W // 3:W - 1] = rng.random((H // 2 - H // 4, W - 1 - W // 3)) + f32(0.5)
    box = np.zeros((H, W), f32)
    box[-4:, :6] = 2.0
    lam = rng.standard_normal((3, H, W)).astype(f32)

    t = Tissue((H, W), P4A, D, [Stimulus(Protocol(0, 2, 100), dense), Stimulus(Protocol(0, 2, 50), box),
                                Stimulus(Protocol(9, 2, 50), np.ones((H, W), f32))])
    t.set_state((v, w, u))
    adj = Adjoint(t)
    nxt, out = torch.zeros_like(t.state), torch.full_like(t.state, 7.0)
    nxt[:, :, :W] = torch.as_tensor(lam)
    adj.step(t.state, 1, nxt, out)
    got = [out[k, :, :W].double().cpu().numpy() for k in range(3)]
    got += [adj.grad_D().double().cpu().numpy(), adj.grad_theta().cpu().numpy()]
    assert (out[:, :, W:] == 7.0).all()  # the row padding is not written

    x = [torch.tensor(a.astype(np.float64), requires_grad=True) for a in (v, w, u, D)]
    th = torch.tensor(np.array(P4A[:13], f32).astype(np.float64), requires_grad=True)
    stims = [(0, 2, 100, torch.tensor(dense.astype(np.float64))), (0, 2, 50, torch.tensor(box.astype(np.float64)))]
    y = FT.euler_step(x[:3], 1, th, 1.0, x[3], stims, 0.01, 0.01)
    sum((a * torch.tensor(b.astype(np.float64))).sum() for a, b in zip(y, lam)).backward()
    ref = [a.grad.numpy() for a in x] + [th.grad.numpy()]
    for name, a, b, tol in zip(("v", "w", "u", "D"), got, ref, (8e-6,) * 4):
        assert np.linalg.norm(a - b) <= tol * np.linalg.norm(b), (name, H, W)
    for k in range(12):
        assert abs(got[4][k] - ref[4][k]) <= 2e-4 * abs(ref[4][k]) + 1e-12, (k, H, W)
    assert got[4][12] == 0.0
