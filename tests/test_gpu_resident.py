"""The resident stepper (many steps of a tissue in one launch, the state on chip) against one
launch per step: the same bits at the sizes where its tiling can go wrong."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from cardiax_gb300 import _native as N  # noqa: E402
from cardiax_gb300 import params as Pm  # noqa: E402
from cardiax_gb300.stimulus import Protocol, Stimulus  # noqa: E402
from cardiax_gb300.tissue import Tissue, stream_handle  # noqa: E402


def _tissue(H, W, n_stim=2, seed=0, track=False, P=Pm.PARAMSET_3):
    rng = np.random.default_rng(seed + 1000 * H + W)
    n = rng.standard_normal((H, W)).astype(np.float32)
    for ax in (0, 1):  # smooth D: the scheme diverges on a rough one
        n = (np.roll(n, 1, ax) + n + np.roll(n, -1, ax)) / 3
    D = (1e-3 * (1 + 0.1 * n)).astype(np.float32)
    stims = []
    if n_stim > 0:
        f = np.zeros((H, W), np.float32)
        f[:, :3] = 20.0
        stims.append(Stimulus(Protocol(0, 2, 25), f))
    if n_stim > 1:  # a dense field
        f = np.zeros((H, W), np.float32)
        f[H // 3:H // 2, W // 3:W // 2] = 10.0 + rng.random((H // 2 - H // 3, W // 2 - W // 3))
        stims.append(Stimulus(Protocol(7, 3, 1000), f))
    t = Tissue((H, W), P, D, stims)
    u = rng.random((H, W)).astype(np.float32)
    t.set_state((1 - 0.5 * u, 0.9 * np.ones_like(u), 0.3 * u))
    if track:
        t.track_activation(0.4)
    return t


def _per_step(t, t0, t1):
    act = ctypes.byref(t.activation) if t.activation is not None else None
    N.call("fk_forward_euler_tracked", t.grid, t.state.data_ptr(), t.scratch.data_ptr(),
           t.D.data_ptr(), ctypes.byref(t.params), t.stim, t.n_stim, t0, t1, t.dt, t.dx, act,
           stream_handle())


def _eligible(H, W):
    return int(N.lib().fk_resident_workspace_bytes(N.Grid(H, W, (W + 3) // 4 * 4))) > 0


# the smallest grids, each residue of H mod 2..5 and W mod 4, one tile column, long strips, the
# sizes of the package's own workloads, the largest that fits; and sizes it does not take
SHAPES = [(16, 16), (16, 17), (17, 18), (18, 19), (19, 23), (21, 21), (29, 40), (31, 129), (64, 64),
          (127, 65), (128, 128), (151, 203), (256, 256), (333, 517), (509, 511), (1000, 37),
          (37, 1000), (4099, 40), (768, 770), (1023, 1021), (1200, 1200), (8, 40), (1400, 1400)]


@pytest.mark.parametrize("H,W", SHAPES)
def test_resident_equals_one_launch_per_step(H, W):
    assert _eligible(H, W) == ((H, W) not in ((8, 40), (1400, 1400)))
    a, b = _tissue(H, W), _tissue(H, W)
    for t0, t1 in ((0, 40), (40, 47)):
        a.advance(t0, t1)
        _per_step(b, t0, t1)
        for p, q in zip(a.view(), b.view()):
            assert torch.isfinite(p).all()
            assert torch.equal(p, q)


@pytest.mark.parametrize("H,W", [(130, 131), (700, 333)])
def test_resident_tracks_activations(H, W):
    a, b = _tissue(H, W, track=True), _tissue(H, W, track=True)
    a.advance(0, 70)
    _per_step(b, 0, 70)
    assert int(a.act_count.sum()) > 0
    for p, q in zip(a.activation_maps(), b.activation_maps()):
        assert torch.equal(p, q)


@pytest.mark.parametrize("ck", [[0, 40], [3, 9, 9, 10, 11, 40], [5, 5, 50], list(range(0, 200, 3)),
                                [0, 8192, 8193, 16500]])
def test_resident_checkpoints(ck):
    """Every listed state (more than one launch writes, repeated ones, more steps than one launch
    takes), the input state left alone."""
    t = _tissue(65, 70)
    before = t.state.clone()
    out = t.forward(ck)
    assert torch.equal(t.view()[2], t.view(before)[2])
    ref = torch.empty_like(out)
    arr = (ctypes.c_int64 * len(ck))(*ck)
    N.call("fk_forward", t.grid, t.state.data_ptr(), t.scratch.data_ptr(), t.D.data_ptr(),
           ctypes.byref(t.params), t.stim, t.n_stim, arr, len(ck), t.dt, t.dx, ref.data_ptr(),
           stream_handle())
    assert torch.equal(out[..., :70], ref[..., :70])


def test_resident_long_run_in_place_and_row_padding():
    """More steps than one launch takes, in place; the state's padding columns stay as they were."""
    a, b = _tissue(50, 49), _tissue(50, 49)
    a.state[:, :, 49:] = 7.0
    a.advance(0, 20001)
    _per_step(b, 0, 20001)
    assert torch.equal(a.state[:, :, :49], b.state[:, :, :49])
    assert (a.state[:, :, 49:] == 7.0).all()


def test_resident_in_a_captured_graph_and_on_two_streams():
    a, b, c = (_tissue(96, 100) for _ in range(3))
    a.advance(0, 30)
    _per_step(c, 0, 30)
    want = c.state.clone()
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    keep = b.state.clone()
    with torch.cuda.stream(s):
        b.advance(0, 30)  # allocates the workspace
        b.state.copy_(keep)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        b.advance(0, 30)
    b.state.copy_(keep)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(a.state, want) and torch.equal(b.state, want)
    streams = [torch.cuda.Stream() for _ in range(3)]
    ts = [_tissue(96, 100) for _ in streams]
    torch.cuda.synchronize()
    for t, st in zip(ts, streams):
        with torch.cuda.stream(st):
            t.advance(0, 30)
    torch.cuda.synchronize()
    for t in ts:
        assert torch.equal(t.state, want)
