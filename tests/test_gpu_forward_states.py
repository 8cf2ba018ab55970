"""Several states of a rollout by one call, and segments recomputed on chip: the same bits as one launch
per step, whatever lies in the padding of the states that they start from."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from cardiax_gb300 import _native as N  # noqa: E402
from cardiax_gb300 import adjoint as A  # noqa: E402
from cardiax_gb300 import params as Pm  # noqa: E402
from cardiax_gb300.stimulus import Protocol, Stimulus  # noqa: E402
from cardiax_gb300.tissue import Tissue, stream_handle  # noqa: E402


def _inputs(H, W, seed=0):
    g = torch.Generator().manual_seed(seed)
    i, j = torch.meshgrid(torch.arange(H), torch.arange(W), indexing="ij")
    D = 1e-3 * (1 - 0.5 * torch.exp(-((i - H / 2) ** 2 + (j - W / 3) ** 2) / (0.03 * H * W)))
    u = 0.3 * torch.rand((H, W), generator=g)
    f = np.zeros((H, W), np.float32)
    f[: max(2, H // 8), :] = 20.0
    x = torch.stack([1 - u, 1 - 0.5 * u, u]).cuda()
    return D.float().cuda(), x, [Stimulus(Protocol(2, 3, 30), f)]


def _tissue(H, W, seed=0):
    D, x, st = _inputs(H, W, seed)
    t = Tissue((H, W), Pm.PARAMSET_3, D, st, dt=0.01, dx=0.01)
    t.set_state(tuple(x))
    return t


def _stepped(t, t0, t1):
    N.call("fk_forward_euler_tracked", t.grid, t.state.data_ptr(), t.scratch.data_ptr(), t.D.data_ptr(),
           ctypes.byref(t.params), t.stim, t.n_stim, t0, t1, t.dt, t.dx, None, stream_handle())


STEPS = [[3, 9, 17], [0, 0, 12, 12, 13], [4, 4], list(range(1, 41)), [50]]


@pytest.mark.parametrize("H,W", [(16, 16), (40, 52), (151, 203), (64, 65), (1300, 1290)])
@pytest.mark.parametrize("steps", STEPS)
def test_states_of_one_tissue(H, W, steps):
    L = A._lib()
    a, b = _tissue(H, W), _tissue(H, W)
    ws, n = a._resident_workspace()
    outs = [torch.full_like(a.state, float("nan")) for _ in steps]
    args = (a.grid, a.state.data_ptr(), a.scratch.data_ptr(), a.D.data_ptr(), ctypes.byref(a.params), a.stim,
            a.n_stim, 0)
    assert L.fk_forward_states(*args, *A._step_list(steps, outs), a.dt, a.dx, ws, n, stream_handle()) == 0
    at = 0
    for s, o in zip(steps, outs):
        _stepped(b, at, s)
        at = s
        assert torch.equal(o[..., :W], b.state[..., :W])
    assert torch.equal(a.state[..., :W], b.state[..., :W])
    a.state.copy_(outs[-1])  # not-a-number in the padding
    a.advance(at, at + 9)
    _stepped(b, at, at + 9)
    assert torch.equal(a.state[..., :W], b.state[..., :W])
    bad = A._step_list([5, 4], outs[:1] * 2)
    assert L.fk_forward_states(*args, *bad, a.dt, a.dx, ws, n, stream_handle()) != 0


@pytest.mark.parametrize("H,W", [(16, 16), (40, 50), (131, 70)])
@pytest.mark.parametrize("n", [1, 6, 7, 12, 40])
def test_segment_of_one_tissue(H, W, n):
    L = A._lib()
    t = _tissue(H, W)
    ws, nb = t._resident_workspace()
    x = torch.full_like(t.state, float("nan"))
    x[..., :W] = t.state[..., :W]
    args = (t.grid, x.data_ptr(), 4, n, t.D.data_ptr(), ctypes.byref(t.params), t.stim, t.n_stim, t.dt, t.dx)
    got = []
    for fn, more in ((L.fk_recompute, ()), (L.fk_recompute_resident, (ws, nb)),
                     (L.fk_recompute_resident, (ws, nb - 1))):
        buf = torch.full((n + 1,) + tuple(x.shape), 3.0, device="cuda")
        assert fn(*args, buf.data_ptr(), *more, stream_handle()) == 0
        assert (buf[n] == 3.0).all()
        got.append(buf[:n, ..., :W].clone())
    assert torch.isfinite(got[0]).all()
    assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])


@pytest.mark.parametrize("H,W,B", [(64, 64, 3), (41, 70, 5), (96, 257, 2)])
@pytest.mark.parametrize("steps", STEPS)
def test_states_of_a_batch(H, W, B, steps):
    D, x, st = _inputs(H, W)
    xs = torch.stack([x * (1 - 0.01 * k) for k in range(B)])
    got = []
    for on in (1, 0):
        bp = A._BatchPlan(xs, A.to_pitched(D, H, W, A.pitch_of(W), D.device), list(Pm.PARAMSET_3), [st] * B,
                          0.01, 0.01)
        assert bp.resident
        N.call("fk_batch_set_resident", bp.plan, on)
        outs = [torch.full_like(bp.S, float("nan")) for _ in steps]
        bp.states(0, steps, outs)
        got.append([o[..., :W].clone() for o in outs] + [bp.S[..., :W].clone()])
        bp.S.copy_(outs[-1])
        bp.advance(steps[-1], steps[-1] + 8)
        got[-1].append(bp.S[..., :W].clone())
        bp.close()
    for p, q in zip(*got):
        assert torch.isfinite(p).all() and torch.equal(p, q)


@pytest.mark.parametrize("H,W", [(40, 52), (70, 131)])
def test_rollouts_of_many_observations(H, W, monkeypatch):
    """More observations than one call writes, at repeated and at the first steps: outputs and gradients
    with and without the resident path."""
    D, x, st = _inputs(H, W)
    obs = [0, 3, 3] + list(range(5, 45)) + [12]
    got = []
    for stepping in (False, True):
        if stepping:
            monkeypatch.setattr(Tissue, "_resident_workspace", lambda self: (None, 0))
            monkeypatch.setattr(A._BatchPlan, "resident", property(lambda s: False, lambda s, v: N.call(
                "fk_batch_set_resident", s.plan, 0)), raising=False)
        Dl, xl = D.clone().requires_grad_(True), x.clone().requires_grad_(True)
        th = torch.tensor(Pm.PARAMSET_3[:13], device="cuda", requires_grad=True)
        out = A.rollout(xl[0], xl[1], xl[2], Dl, th, st, 0, 50, obs)
        (out * torch.linspace(0.5, 1.5, len(obs), device="cuda").view(-1, 1, 1, 1)).sum().backward()
        xb = torch.stack([x, 0.9 * x]).requires_grad_(True)
        Db = D.clone().requires_grad_(True)
        outb = A.rollout_batch(xb, Db, th, [st, st], 0, 50, obs)
        (outb ** 2).sum().backward()
        got.append([out.detach(), xl.grad, Dl.grad, th.grad, outb.detach(), xb.grad, Db.grad])
    for p, q in zip(*got):
        assert torch.isfinite(p).all() and torch.equal(p, q)


@pytest.mark.parametrize("H,W,B", [(40, 52, 2), (70, 131, 3), (8, 30, 2)])
def test_gradients_with_every_state_kept(H, W, B, monkeypatch):
    """All states kept, against segments of ceil(sqrt(steps)) recomputed: the same bits; and what falls
    back to segments."""
    D, x, st = _inputs(H, W)
    obs = [0, 7, 7, 31, 12]
    taken = []
    room = A._room_for_states

    def spied(*a):
        r = room(*a)
        taken.append(r is not None)
        return r

    monkeypatch.setattr(A, "_room_for_states", spied)
    got = []
    for seg in (None, 6):
        Dl, xl = D.clone().requires_grad_(True), x.clone().requires_grad_(True)
        th = torch.tensor(Pm.PARAMSET_3[:13], device="cuda", requires_grad=True)
        out = A.rollout(xl[0], xl[1], xl[2], Dl, th, st, 0, 40, obs, seg=seg)
        (out ** 2).sum().backward()
        xb = torch.stack([(1 - 0.1 * k) * x for k in range(B)]).requires_grad_(True)
        outb = A.rollout_batch(xb, Dl, th, [st] * B, 0, 40, obs, seg=seg)
        (outb ** 2).sum().backward()
        got.append([out.detach(), xl.grad, Dl.grad, th.grad, outb.detach(), xb.grad])
    assert taken == [True, True]
    for p, q in zip(*got):
        assert torch.isfinite(p).all() and torch.equal(p, q)
    A.rollout(x[0], x[1], x[2], D, th.detach(), st, 0, 40, obs)  # nothing to differentiate
    assert taken == [True, True]
    assert room(0, x) is None and room(A.MOST_KEPT + 1, x) is None
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda *a: (0, 1))
    assert room(10, x) is None
