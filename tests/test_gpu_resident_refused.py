"""A launch of the resident kernel that the device refuses: the call steps launch by launch, with the same bits.
(The refusal is made on the host, before the launch.)"""
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


def _tissue(H, W, k=0):
    f = np.zeros((H, W), np.float32)
    f[:5, k:] = 20.0
    return Tissue((H, W), Pm.PARAMSET_3, np.full((H, W), 1e-3, np.float32), [Stimulus(Protocol(1, 2, 900), f)])


def _both(call):
    """What `call` gives on chip, and where its first launch is refused; nothing is left to refuse after it."""
    want = call()
    N.call("fk_selftest_refuse_resident", 1)
    try:
        got = call()
        N.call("fk_selftest_refuse_resident", 0)
        again = call()
    finally:
        N.call("fk_selftest_refuse_resident", 0)
    assert len(want) == len(got) and all(torch.isfinite(x).all() for x in want)
    for x, y, z in zip(want, got, again):
        assert torch.equal(x, y) and torch.equal(x, z)


@pytest.mark.parametrize("H,W", [(64, 64), (200, 333)])  # one cluster; blocks all over the device
def test_one_tissue(H, W):
    L = A._lib()

    def advance():
        t = _tissue(H, W)
        t.track_activation(0.5)
        t.advance(0, 30)
        return [x.clone() for x in t.view()] + list(t.activation_maps())

    def forward():
        t = _tissue(H, W)
        return [t.forward([0, 10, 10, 25])[..., :W].clone()]

    def states():
        t = _tissue(H, W)
        outs = [torch.empty_like(t.state) for _ in range(3)]
        ws, n = t._resident_workspace()
        assert L.fk_forward_states(t.grid, t.state.data_ptr(), t.scratch.data_ptr(), t.D.data_ptr(), t.params, t.stim,
                                   t.n_stim, 0, *A._step_list([4, 4, 20], outs), t.dt, t.dx, ws, n,
                                   stream_handle()) == 0
        return [x[..., :W].clone() for x in outs + [t.state]]

    def segment():
        t = _tissue(H, W)
        buf = torch.empty((12,) + tuple(t.state.shape), device="cuda")
        A.Adjoint(t).recompute(t.state, 0, 12, buf)
        return [buf[..., :W].clone()]

    for call in (advance, forward, states, segment):
        _both(call)


def test_batch():
    H, W, B = 70, 90, 5
    L = A._lib()

    def batch():
        ts = [_tissue(H, W, k) for k in range(B)]
        b = TissueBatch(ts)
        N.call("fk_batch_set_resident", b._plan, 2)
        return ts, b

    def advance():
        ts, b = batch()
        b.advance(0, 30)
        return [t.state[..., :W].clone() for t in ts]

    def states():
        ts, b = batch()
        ns = ts[0].state.numel()
        outs = [torch.empty((B, ns), device="cuda") for _ in range(3)]
        assert L.fk_batch_forward_states(b._plan, 0, *A._step_list([4, 9, 20], outs), ns, stream_handle()) == 0
        return [o.reshape(B, 3, H, -1)[..., :W].clone() for o in outs] + [t.state[..., :W].clone() for t in ts]

    def segment():
        ts, b = batch()
        ns = ts[0].state.numel()
        buf = torch.empty((B, 12 * ns), device="cuda")
        assert L.fk_batch_recompute(b._plan, 0, 12, buf.data_ptr(), 12 * ns, stream_handle()) == 0
        return [buf.reshape(B, 12, 3, H, -1)[..., :W].clone()]

    for call in (advance, states, segment):
        _both(call)
