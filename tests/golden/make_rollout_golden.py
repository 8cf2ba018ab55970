"""Gradients of whole rollouts, recorded on a GB300 while every grid took the adjoint tile kernel
(tests/golden/rollout_gradients.npz).  Inputs come from integer hashes and sums in a fixed order, so that they are
the same bits everywhere.

    python tests/golden/make_rollout_golden.py     # on a GPU; run it only with a build whose bits are to be kept
"""
import os

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
PATH = os.path.join(HERE, "rollout_gradients.npz")

# H, W, steps, observed steps; the shortest lines of the line kernel, every residue of H mod 2 and W mod 4, one and
# several tiles each way, the small grids whose edges weigh most
CASES = [(20, 20, 60, (60,)), (21, 35, 40, (13, 40)), (33, 66, 50, (50,)), (48, 52, 90, (30, 60, 90)),
         (49, 67, 60, (60,)), (61, 70, 45, (20, 45)), (70, 57, 30, (30,)), (40, 129, 40, (40,))]


def _hash(seed, n):
    x = (np.arange(n, dtype=np.uint64) + np.uint64(1)) * np.uint64(0x9E3779B97F4A7C15)
    x ^= np.uint64(seed * 0xD1B54A32D192ED03 % 2 ** 64)
    for s, m in ((30, 0xBF58476D1CE4E5B9), (27, 0x94D049BB133111EB)):
        x = (x ^ (x >> np.uint64(s))) * np.uint64(m)
    return ((x ^ (x >> np.uint64(31))) >> np.uint64(40)).astype(np.float64) / 2.0 ** 24


def _smooth(seed, H, W, passes=6):
    a = _hash(seed, H * W).reshape(H, W)
    for _ in range(passes):
        p = np.pad(a, 1, mode="edge")
        a = (p[1:-1, 1:-1] + p[:-2, 1:-1] + p[2:, 1:-1] + p[1:-1, :-2] + p[1:-1, 2:]) * 0.2
    lo, hi = a.min(), a.max()
    return (a - lo) / (hi - lo)


def inputs(case):
    """(v, w, u, D, stimulus field, observed u) of a case: a tissue in mid-activity."""
    H, W = case[:2]
    f32 = np.float32
    n = _smooth(H * 1000 + W, H, W)
    u = np.clip(2.5 * (n - 0.35), 0.0, 0.98).astype(f32)
    v = np.clip(1.2 - 1.4 * n, 0.0, 1.0).astype(f32)
    w = np.clip(1.0 - 0.4 * _smooth(H * 1000 + W + 7, H, W), 0.0, 1.0).astype(f32)
    D = (1e-3 * (0.9 + 0.2 * _smooth(H * 1000 + W + 13, H, W))).astype(f32)
    f = np.zeros((H, W), f32)
    f[H // 4:H // 4 + 6, W // 3:W // 3 + 7] = 20.0
    obs = _smooth(H * 1000 + W + 29, H, W).astype(f32)
    return v, w, u, D, f, obs


def gradients(case):
    """dL/dv0, dw0, du0, dD, dtheta of L = mean over the observations of (u - obs)^2, as numpy arrays."""
    import torch
    from cardiax_gb300 import adjoint, params
    from cardiax_gb300.stimulus import Protocol, Stimulus
    H, W, steps, times = case
    v, w, u, D, f, obs = (torch.as_tensor(a).cuda() for a in inputs(case))
    x = [a.requires_grad_(True) for a in (v, w, u, D)]
    th = torch.tensor(list(params.PARAMSET_3)[:13], dtype=torch.float32, device="cuda", requires_grad=True)
    out = adjoint.rollout(x[0], x[1], x[2], x[3], th, [Stimulus(Protocol(3, 2, 1000), f)], 0, steps, list(times),
                          0.01, 0.01)
    # (powers of two and differences only: the cotangents are the same bits in every torch)
    g = torch.zeros_like(out)
    g[:, 2] = (out[:, 2] - obs).detach() * (2.0 ** -10)
    return [a.cpu().numpy() for a in torch.autograd.grad(out, (*x, th), g)]


if __name__ == "__main__":
    import sys
    sys.path.insert(0, os.path.dirname(os.path.dirname(HERE)))
    to = sys.argv[1] if len(sys.argv) > 1 else PATH
    np.savez_compressed(to, **{f"{c[0]}x{c[1]}_{name}": a for c in CASES
                               for name, a in zip(("v", "w", "u", "D", "theta"), gradients(c))})
