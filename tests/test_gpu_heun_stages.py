"""Heun steps at the sizes where the two fused stages can go wrong (partial quads and tiles, one-row
and one-column last tiles), against the float64 oracle.

Tolerance: a step adds dt times derivatives of at most some 30 here (D / dx^2 = 10, u below 0.3), whose
float32 rounding is about 10 * 2^-24 of that: 30 * 6e-7 * 0.01 = 2e-7 per stage and step, and a step's
error reaches the next ones damped; 2 steps of 2 stages, doubled: 2e-6.
"""
import numpy as np
import pytest
import torch

import fk_oracle as O

pytestmark = pytest.mark.gpu

P3 = (3.33, 19.6, 1250, 870, 41, 0.25, 12.5, 33.33, 29, 10, 0.85, 0.13, 0.04, 1)
SHAPES = [(3, 3), (5, 9), (16, 16), (31, 66), (32, 64), (33, 65), (33, 130), (64, 129), (65, 131),
          (97, 67), (130, 260)]


@pytest.mark.parametrize("H,W", SHAPES)
def test_heun_steps_match_oracle(H, W):
    from cardiax_gb300.stimulus import Protocol, Stimulus
    from cardiax_gb300.tissue import Tissue
    rng = np.random.default_rng(77 * H + W)
    f32 = np.float32
    u = (0.3 * rng.random((H, W))).astype(f32)
    for gate in (P3[11], P3[12]):
        u[np.abs(u - gate) < 2e-3] += f32(6e-3)
    v, w = (0.5 + 0.5 * rng.random((2, H, W))).astype(f32)
    D = (1e-3 * (1 + 0.05 * rng.standard_normal((H, W)))).astype(f32)
    f = np.zeros((H, W), f32)
    f[: H // 2, : max(1, W // 3)] = rng.random((H // 2, max(1, W // 3))) + f32(1)
    t = Tissue((H, W), P3, D, [Stimulus(Protocol(0, 2, 1e9), f)])
    t.state.fill_(5.0)
    t.set_state((v, w, u))
    t.advance_heun(0, 2)
    d = np.float64
    ref = O.forward_heun(O.OState(v.astype(d), w.astype(d), u.astype(d)), 0, 2, P3, D.astype(d),
                         [O.OStim(0, 2, 1e9, f.astype(d))], 0.01, 0.01)
    for a, b in zip(t.view(), ref):
        assert np.abs(a.cpu().numpy().astype(d) - b).max() <= 2e-6
    one = Tissue((H, W), P3, D, [Stimulus(Protocol(0, 2, 1e9), f)])
    one.set_state((v, w, u))
    one.advance_heun(0, 1).advance_heun(1, 2)
    for a, b in zip(t.view(), one.view()):
        assert torch.equal(a, b)
