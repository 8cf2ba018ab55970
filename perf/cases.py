"""The work that users of this package have it do, as cases that can be timed and checked.

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges, ``prepare(case, seed)``
makes what a program has in hand before the call (on the GPU), ``run(state)`` is one pass through
the public entry points, ``work(case)`` the bytes and operations a pass cannot do without, and
``exact(case, seed)`` the outputs in 64 bits, from plain torch.

Sizes are the package's own: the 128^2 example configuration, the 256^2 inverse problem, the 1200^2
data generation, the 2048^2 and 4096^2 stepper workloads, the mixed batch of 64^2 .. 256 x 1024
tissues, and odd sizes between them.
"""
from __future__ import annotations

import math

import numpy as np
import torch

DT = DX = 0.01
CELL_STEPS = 4096 * 4096 * 30      # the largest listed case's cell updates
GRAD_STEPS = 16 * 256 * 256 * 80   # the largest listed gradient's (cells x steps)

# operations of one Euler update of a cell (a fused multiply-add counts two): six 4-tap stencils
# and their scalings, the diffusion sum, the gates and currents, the update
FLOPS_UPDATE = 95
# a gradient step: the update, its recomputation, and the transposed operators with the
# derivatives of the gates and currents with respect to the state and 13 parameters
FLOPS_GRADIENT = 2 * FLOPS_UPDATE + 250

BATCH_SHAPES = ((64, 64), (128, 128), (256, 256), (512, 512), (256, 1024))


# ---- the cases ---------------------------------------------------------------------------------
def listed():
    return [
        # one derivative of a mid-sized tissue with a rotated (dense) stimulus on: what a program
        # that brings its own integrator calls, one launch at a time
        {"name": "derivative_512", "kind": "derivative", "H": 512, "W": 512},
        # the 128^2 example configuration through the drop-in call: 1000 steps, 10 states kept
        {"name": "forward_128", "kind": "forward", "H": 128, "W": 128, "steps": 1000, "keep": 10},
        # an interactive simulation of a small tissue, advanced in place
        {"name": "advance_256", "kind": "advance", "H": 256, "W": 256, "steps": 200},
        # a ragged tissue with activation-time maps and three stimuli (a stripe, a rectangle, a
        # rotated stripe), as restitution studies use
        {"name": "tracked_333x517", "kind": "tracked", "H": 333, "W": 517, "steps": 100},
        # data generation: a 1200^2 tissue, a 256^2 state emitted every 100 steps
        {"name": "sequence_1200", "kind": "sequence", "H": 1200, "W": 1200, "steps": 300,
         "every": 100, "out": 256},
        # the stepper workload: 2048^2
        {"name": "advance_2048", "kind": "advance", "H": 2048, "W": 2048, "steps": 60},
        # the largest one: 4096^2 (nothing stays in L2 between steps)
        {"name": "advance_4096", "kind": "advance", "H": 4096, "W": 4096, "steps": 30},
        # the second integrator
        {"name": "heun_2048", "kind": "heun", "H": 2048, "W": 2048, "steps": 20},
        # many tissues of mixed sizes, parameter sets and scars in one batch
        {"name": "batch_mixed_48", "kind": "batch", "tissues": 48, "steps": 64,
         "mix": 1},
        # the inverse problem: 16 experiments on one 256^2 tissue, gradients of D and theta
        {"name": "gradient_16x256", "kind": "gradient_batch", "tissues": 16, "H": 256, "W": 256,
         "steps": 80, "obs": 4},
        # one differentiable rollout on an odd grid, gradients of the initial state, D and theta
        {"name": "gradient_151x203", "kind": "gradient", "H": 151, "W": 203, "steps": 100,
         "obs": 3},
        # the diffusivity taper of a scar: a 1200^2 mask blurred with 120 x 120 weights
        {"name": "scar_blur_1200", "kind": "scar", "H": 1200, "W": 1200, "taps": 120},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi):
    """A size spread over the logarithm of the range; one in three a multiple of 32."""
    n = _log(rng, lo, hi)
    return max(lo, min(hi, n // 32 * 32)) if rng.random() < 1 / 3 and n >= 64 else n


def draw(rng):
    kind = rng.choice(("derivative", "forward", "advance", "advance", "tracked", "sequence",
                       "heun", "batch", "gradient_batch", "gradient", "scar"))
    if kind == "batch":
        return {"kind": kind, "tissues": rng.randint(8, 48), "steps": rng.randint(16, 64),
                "mix": rng.randint(2, 1000000)}
    if kind == "gradient_batch":
        H, W, n = _size(rng, 64, 256), _size(rng, 64, 256), rng.randint(2, 16)
        return {"kind": kind, "tissues": n, "H": H, "W": W,
                "steps": max(10, min(80, GRAD_STEPS // (n * H * W))), "obs": rng.randint(1, 4)}
    if kind == "gradient":
        return {"kind": kind, "H": _size(rng, 48, 512), "W": _size(rng, 48, 512),
                "steps": rng.randint(20, 100), "obs": rng.randint(1, 3)}
    if kind == "scar":
        H = _size(rng, 400, 1200)
        return {"kind": kind, "H": H, "W": _size(rng, 400, 1200), "taps": H // 10}
    if kind == "sequence":
        H, W = _size(rng, 256, 1200), _size(rng, 256, 1200)
        every = rng.randint(20, 100)
        return {"kind": kind, "H": H, "W": W, "steps": every * rng.randint(2, 3), "every": every,
                "out": rng.choice((64, 128, 256))}
    if kind == "forward":
        H, W, keep = _size(rng, 32, 512), _size(rng, 32, 512), rng.randint(1, 10)
        return {"kind": kind, "H": H, "W": W, "keep": keep,
                "steps": keep * rng.randint(10, 60)}
    if kind == "derivative":
        return {"kind": kind, "H": _size(rng, 32, 2048), "W": _size(rng, 32, 2048)}
    if kind == "tracked":
        H, W = _size(rng, 64, 1024), _size(rng, 64, 1024)
        return {"kind": kind, "H": H, "W": W, "steps": rng.randint(20, 150)}
    if kind == "heun":
        H, W = _size(rng, 128, 2048), _size(rng, 128, 2048)
        return {"kind": kind, "H": H, "W": W, "steps": rng.randint(5, 20)}
    H, W = _size(rng, 48, 4096), _size(rng, 48, 4096)
    return {"kind": "advance", "H": H, "W": W,
            "steps": max(4, min(rng.randint(20, 200), CELL_STEPS // (H * W)))}


# ---- inputs --------------------------------------------------------------------------------------
def _device():
    return torch.device("cuda")


def _smooth(g, H, W, cells):
    """A smooth seeded random field of about unit variation over ``cells`` cells."""
    h, w = H // cells + 3, W // cells + 3
    n = torch.randn((1, 1, h, w), generator=g, dtype=torch.float32).to(_device())
    return torch.nn.functional.interpolate(n, size=(H, W), mode="bicubic",
                                           align_corners=True)[0, 0].contiguous()


def _diffusivity(g, H, W):
    """Healthy tissue with smooth 5 % variation (per-cell noise would make the scheme diverge)."""
    return (0.001 * (1.0 + 0.05 * _smooth(g, H, W, 6))).clamp_(2e-4, 1.5e-3)


def _scar_diffusivity(g, H, W):
    """Tissue with one to three smooth-edged scars in which D falls to 2e-4 .. 4e-4."""
    dev = _device()
    y = torch.arange(H, device=dev, dtype=torch.float32)[:, None]
    x = torch.arange(W, device=dev, dtype=torch.float32)[None, :]
    D = torch.full((H, W), 1e-3, device=dev)
    r = torch.rand((3, 5), generator=g).tolist()
    for cy, cx, a, b, f in r[:1 + int(3 * r[0][0])]:
        d = torch.sqrt(((y - cy * H) / (H * (0.08 + 0.15 * a))) ** 2
                       + ((x - cx * W) / (W * (0.08 + 0.15 * b))) ** 2)
        inside = torch.sigmoid((1.0 - d) * 12.0)
        D = D * (1.0 - inside * (0.8 - 0.2 * f))
    return D.clamp_(1e-4, 1e-3)


def _state(g, H, W):
    """A tissue in mid-activity: excited regions (u near 1) with fronts, resting tissue between,
    and gates to match."""
    n = _smooth(g, H, W, max(8, min(H, W) // 6))
    u = torch.sigmoid(9.0 * (n - 0.3))
    v = (1.0 - 0.95 * torch.sigmoid(9.0 * (n - 0.1))).clamp_(0.0, 1.0)
    w = (0.7 + 0.3 * torch.sigmoid(-5.0 * n)).clamp_(0.0, 1.0)
    return v, w, u * 0.98


def _rect(g, H, W, start, period):
    """A 10 x 10 point stimulus (smaller on tiny grids) at a random site."""
    from cardiax_gb300 import stimulus as S
    n = min(10, H // 3, W // 3)
    r, c = (torch.rand(2, generator=g).tolist())
    r, c = int(r * (H - n)), int(c * (W - n))
    f = torch.zeros((H, W), device=_device())
    f[r:r + n, c:c + n] = 20.0
    return S.Stimulus(S.Protocol(start, 2, period), f)


def _stripe(H, W, start, period):
    from cardiax_gb300 import stimulus as S
    return S.linear((H, W), S.Direction.WEST, max(0.02, 2.0 / H), 20.0,
                    S.Protocol(start, 2, period), device=_device())


def _rotated(g, H, W, start, period):
    """A rotated stripe: a dense field."""
    from cardiax_gb300 import stimulus as S
    angle = 20.0 + 40.0 * torch.rand(1, generator=g).item()
    return S.triangular((H, W), S.Direction.EAST, angle, 0.1, 20.0, S.Protocol(start, 2, period),
                        device=_device())


def _mix(case):
    """The sizes and parameter sets of a mixed batch."""
    r = torch.rand((case["tissues"], 2), generator=torch.Generator().manual_seed(case["mix"]))
    return [(*BATCH_SHAPES[int(a * len(BATCH_SHAPES))], ("1A", "3", "4A", "5")[int(b * 4)])
            for a, b in r.tolist()]


def _param_set(name):
    from cardiax_gb300 import params
    return getattr(params, "PARAMSET_" + name)


def _inputs(case, seed):
    """The plain inputs of a case (tensors, stimuli, parameters), from the seed alone."""
    g = torch.Generator().manual_seed(int(seed) * 7919 + 17)
    kind = case["kind"]
    i = {"P": _param_set("3")}
    if kind == "batch":
        i["tissues"] = []
        for H, W, name in _mix(case):
            c = torch.rand(1, generator=g).item()
            P = _param_set(name)
            s = _stripe(H, W, int(c * 30), 5000) if c < 0.5 else _rect(g, H, W, int(c * 30), 5000)
            i["tissues"].append((H, W, P, _scar_diffusivity(g, H, W), [s], _state(g, H, W)))
        return i
    H, W = case["H"], case["W"]
    if kind == "scar":
        y = torch.arange(H, device=_device(), dtype=torch.float32)[:, None]
        x = torch.arange(W, device=_device(), dtype=torch.float32)[None, :]
        r = torch.rand((5, 3), generator=g).tolist()
        cy, cx = r[0][0] * 0.5 + 0.25, r[0][1] * 0.5 + 0.25
        mask = torch.zeros((H, W), dtype=torch.bool, device=_device())
        for a, b, c in r:  # a chain of overlapping blobs
            cy, cx = cy + 0.1 * (a - 0.5), cx + 0.12 * (b - 0.2)
            mask |= (y - cy * H) ** 2 + (x - cx * W) ** 2 <= (min(H, W) * (0.05 + 0.08 * c)) ** 2
        i["mask"] = mask.to(torch.float32)
        K = case["taps"]
        sigma = np.float32(H / 10 * (0.3 + 1.2 * torch.rand(1, generator=g).item()))
        half = (K - 1.0) / 2.0
        ax = np.arange(-half, half + 1, dtype=np.float32)
        wts = np.exp(-(ax[:, None] ** 2 + ax[None, :] ** 2) / (np.float32(2) * sigma * sigma))
        wts[wts < np.finfo(np.float32).eps * wts.max()] = 0
        i["weights"] = (wts / wts.sum(dtype=np.float32)).astype(np.float32)
        return i
    if kind == "gradient_batch":
        i["D"] = _scar_diffusivity(g, H, W)
        n = case["tissues"]
        i["state"] = torch.stack([torch.stack(_state(g, H, W)) for _ in range(n)])
        i["stimuli"] = [[_rect(g, H, W, 3 * k, 20000)] for k in range(n)]
        T, m = case["steps"], case["obs"]
        i["obs_times"] = [T * (k + 1) // m for k in range(m)]
        i["obs"] = torch.stack([torch.stack([_state(g, H, W)[2] for _ in range(m)])
                                for _ in range(n)])
        return i
    i["D"] = _diffusivity(g, H, W)
    i["state"] = _state(g, H, W)
    if kind == "derivative":
        i["stimuli"] = [_rotated(g, H, W, 5, 1000)]
    elif kind == "tracked":
        i["stimuli"] = [_stripe(H, W, 0, 60), _rect(g, H, W, 10, 1000000000),
                        _rotated(g, H, W, 25, 1000)]
    elif kind == "sequence":
        i["stimuli"] = [_rect(g, H, W, 1, 1000000000), _rotated(g, H, W, 40, 700)]
    else:
        i["stimuli"] = [_stripe(H, W, 0, 20000)]
    if kind == "gradient":
        T, m = case["steps"], case["obs"]
        i["obs_times"] = [T * (k + 1) // m for k in range(m)]
        i["obs"] = torch.stack([_state(g, H, W)[2] for _ in range(m)])
    return i


def prepare(case, seed):
    from cardiax_gb300.batch import TissueBatch
    from cardiax_gb300.tissue import Tissue
    kind = case["kind"]
    i = _inputs(case, seed)
    s = {"case": dict(case), "in": i}
    if kind in ("derivative", "advance", "tracked", "heun"):
        t = Tissue((case["H"], case["W"]), i["P"], i["D"], i["stimuli"], dt=DT, dx=DX)
        t.set_state(i["state"])
        if kind == "tracked":
            t.track_activation(0.5)
        s["tissue"] = t
    elif kind == "batch":
        ts = []
        for H, W, P, D, stim, x in i["tissues"]:
            t = Tissue((H, W), P, D, stim, dt=DT, dx=DX)
            t.set_state(x)
            ts.append(t)
        s["batch"] = TissueBatch(ts)
        s["tissues"] = ts
    elif kind in ("gradient", "gradient_batch"):
        s["theta"] = torch.tensor(list(i["P"])[:13], dtype=torch.float32, device=_device())
        s["D"] = i["D"].clone()
    return s


# ---- one pass --------------------------------------------------------------------------------------
def run(s):
    from cardiax_gb300 import adjoint, generate, scars, solve
    case, i = s["case"], s["in"]
    kind = case["kind"]
    if kind == "derivative":
        t = s["tissue"]
        return list(t.view(t.derivative(5)))
    if kind == "forward":
        keep = case["keep"]
        ck = [case["steps"] * k // keep for k in range(keep + 1)]
        return [list(x) for x in solve.forward(solve.State(*i["state"]), ck, i["P"], i["D"],
                                               i["stimuli"], DT, DX)]
    if kind == "advance":
        return list(s["tissue"].advance(0, case["steps"]).view())
    if kind == "tracked":
        t = s["tissue"].advance(0, case["steps"])
        return list(t.view()) + list(t.activation_maps())
    if kind == "heun":
        return list(s["tissue"].advance_heun(0, case["steps"]).view())
    if kind == "sequence":
        return [generate.sequence(0, case["steps"] + 1, case["every"], DT, DX, i["P"], i["D"],
                                  i["stimuli"], reshape=(case["out"], case["out"]))]
    if kind == "batch":
        s["batch"].advance(0, case["steps"])
        return [t.state[:, :, :t.W] for t in s["tissues"]]
    if kind == "scar":
        return [scars.blur_same(i["mask"], i["weights"], one_minus=True)]
    if kind == "gradient_batch":
        D, th = s["D"].detach().requires_grad_(True), s["theta"].detach().requires_grad_(True)
        out = adjoint.rollout_batch(i["state"], D, th, i["stimuli"], 0, case["steps"],
                                    i["obs_times"], DT, DX)
        loss = ((out[:, :, 2] - i["obs"]) ** 2).mean()
        return [loss, out.detach()] + list(torch.autograd.grad(loss, (D, th)))
    D, th = s["D"].detach().requires_grad_(True), s["theta"].detach().requires_grad_(True)
    x = [a.detach().requires_grad_(True) for a in i["state"]]
    out = adjoint.rollout(x[0], x[1], x[2], D, th, i["stimuli"], 0, case["steps"],
                          i["obs_times"], DT, DX)
    loss = ((out[:, 2] - i["obs"]) ** 2).mean()
    return [loss] + list(torch.autograd.grad(loss, (*x, D, th)))


# ---- what a pass cannot do without ----------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "batch":
        n = sum(H * W for H, W, _ in _mix(case))
        return {"bytes": 28 * n, "flops": FLOPS_UPDATE * n * case["steps"]}
    n = case["H"] * case["W"]
    if kind == "derivative":  # u, v, w, D and the stimulus field in, the derivative out
        return {"bytes": 32 * n, "flops": FLOPS_UPDATE * n}
    if kind == "scar":
        return {"bytes": 8 * n + 4 * case["taps"] ** 2, "flops": 2 * n * case["taps"] ** 2}
    steps = case["steps"]
    if kind == "forward":
        return {"bytes": (16 + 12 * case["keep"]) * n, "flops": FLOPS_UPDATE * n * steps}
    if kind == "sequence":  # D and the fields in, the emitted states out
        emitted = (steps // case["every"] + 1) * case["out"] ** 2
        return {"bytes": 12 * n + 12 * emitted, "flops": FLOPS_UPDATE * n * steps}
    if kind == "tracked":  # the three maps are read and written too
        return {"bytes": (28 + 24 + 4) * n, "flops": FLOPS_UPDATE * n * steps}
    if kind == "heun":
        return {"bytes": 28 * n, "flops": 2 * FLOPS_UPDATE * n * steps}
    if kind == "gradient":  # the initial state, D and observations in, their gradients out
        return {"bytes": (16 + 16 + 4 * case["obs"]) * n, "flops": FLOPS_GRADIENT * n * steps}
    if kind == "gradient_batch":
        b = case["tissues"]
        return {"bytes": (12 * b + 8 + 16 * case["obs"] * b) * n,
                "flops": FLOPS_GRADIENT * n * b * steps}
    return {"bytes": 28 * n, "flops": FLOPS_UPDATE * n * steps}


# ---- the same in 64 bits, from plain torch -----------------------------------------------------------
def _gradient(a, dim):
    """The fourth-order derivative along an axis, one-sided on the first and last two rows."""
    L = a.shape[dim]
    n = lambda lo, hi: a.narrow(dim, lo, hi - lo)  # noqa: E731
    mid = (n(0, L - 4) - n(4, L)) / 12.0 + (n(3, L - 1) - n(1, L - 3)) * (2.0 / 3.0)
    head = (-11.0 / 6.0) * n(0, 2) + 3.0 * n(1, 3) - 1.5 * n(2, 4) + n(3, 5) / 3.0
    tail = -n(L - 5, L - 3) / 3.0 + 1.5 * n(L - 4, L - 2) - 3.0 * n(L - 3, L - 1) \
        + (11.0 / 6.0) * n(L - 2, L)
    return torch.cat((head, mid, tail), dim)


def _pad(a):
    return torch.nn.functional.pad(a.reshape((-1, 1) + tuple(a.shape[-2:])), (1, 1, 1, 1),
                                   mode="replicate").reshape(
        tuple(a.shape[:-2]) + (a.shape[-2] + 2, a.shape[-1] + 2))


def _active(proto, t):
    start, duration, period = (float(x) for x in proto)
    return t >= start and math.fmod(math.fmod(start - t + 1.0, period) + period, period) < duration


def _derivative64(x, t, p, D, stimuli, dD=None):
    """(dv, dw, du) of a state (..., H, W) in 64 bits; ``stimuli``: (protocol, field) pairs, the
    field broadcast against u; p: the 14 parameters."""
    v, w, u = x
    (tvp, tv1, tv2, twp, twm, td, t0, tr, tsi, k, vcsi, vc, vv, cm) = p
    zero, one = torch.zeros((), dtype=u.dtype, device=u.device), torch.ones((), dtype=u.dtype,
                                                                            device=u.device)
    a, b = torch.where(u >= vc, one, zero), torch.where(u >= vv, one, zero)
    tvm = (1.0 - b) * tv1 + b * tv2
    j_fi = -v * a * (u - vc) * (1.0 - u) / td
    j_so = u * (1.0 - a) / t0 + a / tr
    j_si = -w * (1.0 + torch.tanh(k * (u - vcsi))) / (2.0 * tsi)
    j = -(j_fi + j_so + j_si) / cm
    for proto, field in stimuli:
        if _active(proto, t):
            j = torch.where(field != 0, field.to(j.dtype), j)
    up = _pad(u)
    ux, uy = _gradient(up, -2) / DX, _gradient(up, -1) / DX
    uxx, uyy = _gradient(ux, -2) / DX, _gradient(uy, -1) / DX
    c = lambda q: q[..., 1:-1, 1:-1]  # noqa: E731
    Dx, Dy = dD if dD is not None else _slopes(D)
    du = D * (c(uxx) + c(uyy)) + Dx * c(ux) + Dy * c(uy) + j
    dv = (1.0 - a) * (1.0 - v) / tvm - a * v / tvp
    dw = (1.0 - a) * (1.0 - w) / twm - a * w / twp
    return dv, dw, du


def _slopes(D):
    Dp = _pad(D)
    return _gradient(Dp, -2)[..., 1:-1, 1:-1] / DX, _gradient(Dp, -1)[..., 1:-1, 1:-1] / DX


def _euler64(x, t0, t1, p, D, stimuli):
    dD = _slopes(D)
    for t in range(t0, t1):
        x = tuple(a + DT * d for a, d in zip(x, _derivative64(x, t, p, D, stimuli, dD)))
    return x


def _resize64(a, n):
    """Antialiased bilinear resampling of the last two axes to (n, n)."""
    def weights(m):
        scale = n / m
        ks = max(1.0 / scale, 1.0)
        at = (torch.arange(n, dtype=torch.float64) + 0.5) / scale - 0.5
        wt = (1.0 - (at[:, None] - torch.arange(m, dtype=torch.float64)[None, :]).abs() / ks)
        wt = wt.clamp(min=0.0)
        return (wt / wt.sum(1, keepdim=True)).to(_device()) if m != n else torch.eye(
            n, dtype=torch.float64, device=_device())
    return weights(a.shape[-2]) @ a @ weights(a.shape[-1]).T


def exact(case, seed):
    kind = case["kind"]
    i = _inputs(case, seed)
    P = [float(x) for x in i["P"]]
    d = lambda a: a.to(torch.float64)  # noqa: E731
    if kind == "scar":
        H, W = i["mask"].shape
        K = case["taps"]
        n, lo = (H + K - 1, W + K - 1), (K - 1) // 2  # "same": centred as scipy centres it
        full = np.fft.irfft2(np.fft.rfft2(i["mask"].double().cpu().numpy(), n)
                             * np.fft.rfft2(i["weights"].astype(np.float64), n), n)
        return [1.0 - np.ascontiguousarray(full[lo:lo + H, lo:lo + W])]
    if kind == "batch":
        out = []
        for H, W, p, D, stim, x in i["tissues"]:
            st = [(q.protocol, d(q.field)) for q in stim]
            y = _euler64(tuple(d(a) for a in x), 0, case["steps"], [float(a) for a in p], d(D), st)
            out.append(torch.stack(y))
        return out
    if kind in ("gradient", "gradient_batch"):
        n = case.get("tissues", 1)
        theta = torch.tensor(P[:13], dtype=torch.float32, device=_device()).double()
        gD = torch.zeros_like(d(i["D"]))
        gth, loss, gx, seen = torch.zeros_like(theta), 0.0, None, []
        obs = i["obs"] if kind == "gradient_batch" else i["obs"][None]
        for e in range(n):
            x0 = i["state"][e] if kind == "gradient_batch" else i["state"]
            stim = i["stimuli"][e] if kind == "gradient_batch" else i["stimuli"]
            x = [d(a).requires_grad_(True) for a in x0]
            D = d(i["D"]).requires_grad_(True)
            th = theta.clone().requires_grad_(True)
            p = list(th.unbind()) + [P[13]]
            st = [(q.protocol, d(q.field)) for q in stim]
            y, t, part = tuple(x), 0, 0.0
            for k, at in enumerate(i["obs_times"]):
                y = _euler64(y, t, at, p, D, st)
                t = at
                part = part + ((y[2] - d(obs[e, k])) ** 2).sum()
                seen.append(torch.stack([a.detach() for a in y]))
            part = part / obs.numel()
            g = torch.autograd.grad(part, (*x, D, th))
            loss, gD, gth, gx = loss + part.detach(), gD + g[3], gth + g[4], g[:3]
            del y, part, g
        if kind == "gradient":
            return [loss, *gx, gD, gth]
        states = torch.stack(seen)
        return [loss, states.reshape((n, -1) + tuple(states.shape[1:])), gD, gth]
    D = d(i["D"])
    x = tuple(d(a) for a in i["state"])
    st = [(q.protocol, d(q.field)) for q in i["stimuli"]]
    if kind == "derivative":
        return list(_derivative64(x, 5, P, D, st))
    if kind == "forward":
        keep, out, at = case["keep"], [], 0
        for k in range(1, keep + 1):
            to = case["steps"] * k // keep
            x = _euler64(x, at, to, P, D, st)
            at = to
            out.append(list(x))
        return out
    if kind == "sequence":
        rows = []
        x = (torch.ones_like(D), torch.ones_like(D), torch.zeros_like(D))
        marks = list(range(0, case["steps"] + 1, case["every"]))
        for a, b in zip(marks[:-1], marks[1:]):
            x = _euler64(x, a, b, P, D, st)
            rows.append(_resize64(torch.stack(x), case["out"]))
        rows.append(torch.zeros_like(rows[0]))
        return [torch.stack(rows)]
    if kind == "heun":
        dD = _slopes(D)
        for t in range(case["steps"]):
            d1 = _derivative64(x, t, P, D, st, dD)
            d2 = _derivative64(tuple(a + DT * b for a, b in zip(x, d1)), t, P, D, st, dD)
            x = tuple(a + (b + c) * (DT / 2) for a, b, c in zip(x, d1, d2))
        return list(x)
    x = list(_euler64(x, 0, case["steps"], P, D, st))
    return x + [None, None, None] if kind == "tracked" else x
