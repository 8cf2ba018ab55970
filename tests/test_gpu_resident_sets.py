"""Batches through the resident launches whatever the estimate says, against each tissue stepped alone (the same
bits): few steps, the splits of calls longer than one launch, more sets of constants than one launch holds, and the
states written out.  Each call's route is asserted."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from cardiax_gb300 import _native as N  # noqa: E402
from cardiax_gb300 import adjoint as A  # noqa: E402
from cardiax_gb300 import params as Pm  # noqa: E402
from cardiax_gb300.batch import TissueBatch  # noqa: E402
from cardiax_gb300.stimulus import Protocol, Stimulus  # noqa: E402
from cardiax_gb300.tissue import Tissue, stream_handle  # noqa: E402

SETS = (Pm.PARAMSET_1A, Pm.PARAMSET_3, Pm.PARAMSET_4A, Pm.PARAMSET_5)
MOST = 8192  # steps of one launch


def _tissues(shapes, sets=4, seed=5):
    """`sets` different sets of constants, dealt out in turn."""
    rng = np.random.default_rng(seed)
    out = []
    for k, (H, W) in enumerate(shapes):
        c = k % sets
        i, j = np.meshgrid(np.arange(H), np.arange(W), indexing="ij")
        D = (1e-3 * (1 - 0.4 * np.exp(-((i - H / 3) ** 2 + (j - W / 2) ** 2) / (0.05 * H * W)))).astype(np.float32)
        f = np.zeros((H, W), np.float32)
        f[: max(2, H // 8), : W // 2] = 20.0
        if k % 3 == 1:  # a dense field
            f[1, : W // 2] = 17.0
        t = Tissue((H, W), SETS[c % 4], D, [Stimulus(Protocol(k % 5, 2, 900), f)], dt=0.01, dx=0.01)
        t.params.tau_d *= 1.0 + 0.01 * (c // 4)
        u = (0.2 * rng.random((H, W))).astype(np.float32)
        t.set_state((1 - u, 1 - 0.5 * u, u))
        out.append(t)
    return out


def _alone(t, t0, t1):
    N.call("fk_forward_euler_tracked", t.grid, t.state.data_ptr(), t.scratch.data_ptr(), t.D.data_ptr(),
           ctypes.byref(t.params), t.stim, t.n_stim, t0, t1, t.dt, t.dx, None, stream_handle())


def _resident(batch, n):
    N.call("fk_batch_set_resident", batch._plan, 2)
    assert N.lib().fk_batch_takes_resident(batch._plan, n) == 1
    return batch


def _same(a, b):
    for x, y in zip(a, b):
        assert torch.isfinite(x.view()[2]).all()
        for p, q in zip(x.view(), y.view()):
            assert torch.equal(p, q)


LISTS = [[(64, 64)] * 3, [(16, 16), (17, 19), (33, 130), (64, 65), (101, 67)],
         [(64, 64), (128, 128), (256, 256), (512, 512), (256, 1024), (200, 300), (1000, 800)],
         [(40 + k, 48 + 3 * k) for k in range(20)]]


@pytest.mark.parametrize("shapes", LISTS, ids=lambda s: f"{len(s)}x{s[0][0]}")
@pytest.mark.parametrize("n", [2, 3, 33])
def test_few_steps(shapes, n):
    a, b = _tissues(shapes), _tissues(shapes)
    _resident(TissueBatch(a), n).advance(3, 3 + n)
    for t in b:
        _alone(t, 3, 3 + n)
    _same(a, b)


@pytest.mark.parametrize("n", [MOST - 1, MOST, MOST + 1, MOST + 2, 2 * MOST + 1])
def test_calls_longer_than_one_launch(n):
    """One more step than a launch takes: the last launch must not run one step in place."""
    shapes = [(40, 48), (35, 50), (40, 48)]
    a, b = _tissues(shapes), _tissues(shapes)
    _resident(TissueBatch(a), n).advance(0, n)
    for t in b:
        _alone(t, 0, n)
    _same(a, b)


@pytest.mark.parametrize("count,sets", [(16, 16), (17, 17), (37, 37), (40, 20)])
def test_sets_of_constants(count, sets):
    """A launch holds sixteen; 20 sets in turn over 40 tissues meet twice in each launch."""
    shapes = [(48 + k % 3, 52) for k in range(count)]
    a, b = _tissues(shapes, sets), _tissues(shapes, sets)
    _resident(TissueBatch(a), 30).advance(0, 30)
    for t in b:
        _alone(t, 0, 30)
    _same(a, b)


@pytest.mark.parametrize("H,W,B,n", [(64, 64, 3, 3), (64, 64, 3, 4), (48, 52, 37, 12), (200, 300, 9, 5)])
def test_recomputed_segments(H, W, B, n):
    L = A._lib()
    ts = _tissues([(H, W)] * B, sets=20 if B > 16 else 1)
    ns = 3 * H * ts[0].pitch
    batch = TissueBatch(ts)
    got = []
    for on in (2, 0):
        N.call("fk_batch_set_resident", batch._plan, on)
        assert L.fk_batch_takes_resident(batch._plan, n - 1) == (on == 2)
        keep = [t.state.clone() for t in ts]
        buf = torch.full((B, n * ns + 64), 3.0, device="cuda")
        assert L.fk_batch_recompute(batch._plan, 4, n, buf.data_ptr(), buf.shape[1], stream_handle()) == 0
        assert (buf[:, n * ns:] == 3.0).all()
        got.append(buf[:, :n * ns].reshape(B, n, 3, H, -1)[..., :W].clone())
        for t, k in zip(ts, keep):
            t.state.copy_(k)
    assert torch.isfinite(got[0]).all() and torch.equal(*got)


@pytest.mark.parametrize("H,W,B", [(64, 64, 3), (200, 300, 9)])
@pytest.mark.parametrize("steps", [[2], [3, 4], [0, 1, 5], list(range(1, 41))])
def test_states_written_out(H, W, B, steps):
    L = A._lib()
    ts = _tissues([(H, W)] * B, sets=1)
    ns = 3 * H * ts[0].pitch
    batch = TissueBatch(ts)
    keep = [t.state.clone() for t in ts]
    got = []
    for on in (2, 0):
        N.call("fk_batch_set_resident", batch._plan, on)
        for t, k in zip(ts, keep):
            t.state.copy_(k)
        outs = [torch.full((B, ns), float("nan"), device="cuda") for _ in steps]
        assert L.fk_batch_forward_states(batch._plan, 0, *A._step_list(steps, outs), ns, stream_handle()) == 0
        states = outs + [torch.stack([t.state.reshape(-1) for t in ts])]
        got.append(torch.stack([o.reshape(B, 3, H, -1)[..., :W] for o in states]))
    assert torch.isfinite(got[0]).all() and torch.equal(*got)


def test_the_estimate_decides_by_default():
    """A call that gains takes the resident launches, one that does not takes one launch per step."""
    batch = TissueBatch(_tissues([(64, 64)] * 3))
    takes = N.lib().fk_batch_takes_resident
    assert takes(batch._plan, 64) == 1 and takes(batch._plan, 3) == 0 and takes(batch._plan, 1) == 0
    many = TissueBatch(_tissues([(48, 52)] * 37, sets=37))  # three launches
    assert takes(many._plan, 64) == 0
    batch.set_options(4, False)
    assert takes(batch._plan, 64) == 0
