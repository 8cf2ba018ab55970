"""Batches whose tissues run resident, set after set, against each tissue stepped alone (the same bits),
and the choice of that path."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from cardiax_gb300 import _native as N  # noqa: E402
from cardiax_gb300 import params as Pm  # noqa: E402
from cardiax_gb300.batch import TissueBatch  # noqa: E402
from cardiax_gb300.stimulus import Protocol, Stimulus  # noqa: E402
from cardiax_gb300.tissue import Tissue, stream_handle  # noqa: E402

SETS = (Pm.PARAMSET_1A, Pm.PARAMSET_3, Pm.PARAMSET_4A, Pm.PARAMSET_5)


def _tissues(shapes, seed=0, same=False):
    rng = np.random.default_rng(seed)
    out = []
    for k, (H, W) in enumerate(shapes):
        i, j = np.meshgrid(np.arange(H), np.arange(W), indexing="ij")
        D = (1e-3 * (1 - 0.5 * np.exp(-((i - H / 2) ** 2 + (j - W / 3) ** 2) / (0.03 * H * W)))).astype(np.float32)
        f = np.zeros((H, W), np.float32)
        f[: max(2, H // 8), :] = 20.0
        if k % 3 == 2:  # a dense field
            f[: H // 2, : W // 2] *= (1 + rng.random((H // 2, W // 2))).astype(np.float32)
        dt, dx = ((0.01, 0.01) if same else ((0.01, 0.008)[k % 2], (0.01, 0.0125)[k % 2]))
        t = Tissue((H, W), SETS[0 if same else k % 4], D, [Stimulus(Protocol(k % 7, 2, 30), f)], dt=dt, dx=dx)
        u = (0.2 * rng.random((H, W))).astype(np.float32)
        t.set_state((1 - u, 1 - 0.5 * u, u))
        out.append(t)
    return out


def _alone(t, t0, t1):
    N.call("fk_forward_euler_tracked", t.grid, t.state.data_ptr(), t.scratch.data_ptr(), t.D.data_ptr(),
           ctypes.byref(t.params), t.stim, t.n_stim, t0, t1, t.dt, t.dx, None, stream_handle())


MIXED = [(64, 64), (128, 128), (256, 256), (512, 512), (256, 1024)]


@pytest.mark.parametrize("shapes", [
    [(64, 64)] * 3,                                  # one tile each
    [(16, 16), (17, 19), (33, 130), (64, 65), (101, 67)],  # ragged, shifted first groups
    MIXED,
    MIXED * 3 + [(200, 300), (1000, 800)],           # several launches
    [(40 + k, 48 + 3 * k) for k in range(20)],       # twenty sets of constants' worth of tissues
])
@pytest.mark.parametrize("steps", [40, 3])
def test_resident_batch_equals_single_tissues(shapes, steps):
    a, b = _tissues(shapes), _tissues(shapes)
    batch = TissueBatch(a)
    N.call("fk_batch_set_resident", batch._plan, 1)  # every tissue here can take it
    batch.advance(0, steps)
    batch.advance(steps, steps + 9)
    for t in b:
        _alone(t, 0, steps + 9)
    for x, y in zip(a, b):
        assert torch.isfinite(x.view()[2]).all()
        for p, q in zip(x.view(), y.view()):
            assert torch.equal(p, q)
    batch.set_options(4, False)  # a knob of the stepping kernel turns the resident path off
    batch.advance(steps + 9, steps + 20)
    for t in b:
        _alone(t, steps + 9, steps + 20)
    for x, y in zip(a, b):
        for p, q in zip(x.view(), y.view()):
            assert torch.equal(p, q)


def test_more_sets_of_constants_than_one_launch_holds():
    rng = np.random.default_rng(3)
    shapes = [(48, 52)] * 37
    a, b = _tissues(shapes, same=True), _tissues(shapes, same=True)
    for k, (x, y) in enumerate(zip(a, b)):
        for t in (x, y):
            t.params.tau_d = 0.3 + 0.01 * k
    batch = TissueBatch(a)
    N.call("fk_batch_set_resident", batch._plan, 1)
    batch.advance(0, 30)
    for x, y in zip(a, b):
        _alone(y, 0, 30)
        assert torch.equal(x.state, y.state)


def test_batches_the_resident_path_does_not_take():
    small = TissueBatch(_tissues([(64, 64), (8, 40)]))
    tracked = _tissues([(64, 64)])
    tracked[0].track_activation(0.5)
    for batch in (small, TissueBatch(tracked)):
        with pytest.raises(N.FkError):
            N.call("fk_batch_set_resident", batch._plan, 1)
        batch.advance(0, 20)


@pytest.mark.parametrize("H,W,n", [(40, 52, 12), (64, 64, 3), (130, 70, 9)])
def test_resident_recompute_equals_stepping(H, W, n):
    """fk_batch_recompute: every state of a segment, the same bits either way, for two gaps between the
    experiments' segments."""
    from cardiax_gb300.adjoint import _lib
    L = _lib()
    ts = _tissues([(H, W)] * 5, same=True)
    ns = 3 * H * ts[0].pitch
    batch = TissueBatch(ts)
    got = []
    for on in (1, 0):
        N.call("fk_batch_set_resident", batch._plan, on)
        keep = [t.state.clone() for t in ts]
        for gap in (0, 64):
            buf = torch.full((5, (n + 1) * ns + gap), 3.0, device="cuda")
            rc = L.fk_batch_recompute(batch._plan, 4, n, buf.data_ptr(), buf.shape[1], stream_handle())
            assert rc == 0
            got.append(buf[:, :n * ns].reshape(5, n, 3, H, -1)[..., :W].clone())
            assert (buf[:, n * ns:] == 3.0).all()
            for t, k in zip(ts, keep):
                t.state.copy_(k)
    for g in got[1:]:
        assert torch.equal(got[0], g)


def test_tuner_times_the_resident_path_and_restores_states():
    from cardiax_gb300.autotune import tune_batch
    ts = _tissues([(64, 64), (128, 130)] * 4)
    keep = [t.state.clone() for t in ts]
    batch = TissueBatch(ts)
    kw = dict(trial_steps=64, candidates=(0,), tile_rows=(32,), options=((1, False),))
    res = tune_batch(batch, **kw)
    assert res["resident_ms_per_step"] > 0 and len(res["ms_per_step"]) in (1, 2)
    assert res["resident"] == (res["resident_ms_per_step"] < min(res["ms_per_step"].values()))
    for t, k in zip(ts, keep):
        assert torch.equal(t.state, k)
    tracked = _tissues([(64, 64), (128, 130)] * 4)
    for t in tracked:
        t.track_activation(0.5)
    batch = TissueBatch(tracked)
    tune_batch(batch, **kw)  # the same shapes; the resident path does not apply
    assert batch.set_resident(True) is False
