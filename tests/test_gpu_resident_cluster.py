"""Small tissues, whose tiles run as one thread-block cluster, and those just above: against one launch per
step (the same bits), with several states written out and with activation tracking."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from cardiax_gb300 import _native as N  # noqa: E402
from cardiax_gb300 import params as Pm  # noqa: E402
from cardiax_gb300.stimulus import Protocol, Stimulus  # noqa: E402
from cardiax_gb300.tissue import Tissue, stream_handle  # noqa: E402


def _tissue(H, W):
    rng = np.random.default_rng(H * 1000 + W)
    i, j = np.meshgrid(np.arange(H), np.arange(W), indexing="ij")
    D = (1e-3 * (1 + 0.4 * np.sin(i / 6) * np.cos(j / 9))).astype(np.float32)
    f = np.zeros((H, W), np.float32)
    f[: H // 3, W // 4:] = 3.0 * (1 + rng.random((H // 3, W - W // 4)))
    t = Tissue((H, W), Pm.PARAMSET_3, D, [Stimulus(Protocol(3, 2, 20), f)], dt=0.01, dx=0.01)
    u = (0.4 * rng.random((H, W))).astype(np.float32)
    t.set_state((1 - u, 1 - 0.5 * u, u))
    return t


# one tile, two, four, eight and sixteen; odd row counts, partial quads, long and flat grids; both sides of
# the size up to which a cluster is taken
@pytest.mark.parametrize("H,W", [(16, 16), (17, 19), (16, 200), (211, 18), (33, 34), (64, 65), (87, 49), (127, 130),
                                 (140, 139), (150, 151)])
@pytest.mark.parametrize("track", [False, True])
def test_small_tissues_equal_one_launch_per_step(H, W, track):
    a, b = _tissue(H, W), _tissue(H, W)
    if track:
        for t in (a, b):
            t.track_activation(0.3)
    at = 0
    for n in (6, 45, 7):
        a.advance(at, at + n)
        act = ctypes.byref(b.activation) if track else None
        N.call("fk_forward_euler_tracked", b.grid, b.state.data_ptr(), b.scratch.data_ptr(), b.D.data_ptr(),
               ctypes.byref(b.params), b.stim, b.n_stim, at, at + n, b.dt, b.dx, act, stream_handle())
        at += n
        assert torch.isfinite(a.state[..., :W]).all() and torch.equal(a.state[..., :W], b.state[..., :W])
    if track:
        for x, y in zip(a.activation_maps(), b.activation_maps()):
            assert torch.equal(x, y)
    states = a.forward([at, at + 3, at + 3, at + 20, at + 21])
    for k, s in enumerate((at + 3, at + 3, at + 20, at + 21)):
        c = _tissue(H, W)
        c.state.copy_(b.state)
        N.call("fk_forward_euler_tracked", c.grid, c.state.data_ptr(), c.scratch.data_ptr(), c.D.data_ptr(),
               ctypes.byref(c.params), c.stim, c.n_stim, at, s, c.dt, c.dx, None, stream_handle())
        assert torch.equal(states[k][..., :W], c.state[..., :W])
