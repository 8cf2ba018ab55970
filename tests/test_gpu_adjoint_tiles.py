"""The two tile sizes of the adjoint line kernel, and blocks that take several tiles: many experiments
against one at a time.

lambda and dL/dD of a cell are the same operations either way: the same bits.  A parameter's gradient is a
sum over N cells in another grouping: partial sums of at most 16 cells and 32 lanes in float32, 21 additions
deep, 21 * 2^-24 = 1.3e-6 of the sum of magnitudes, which random signs make sqrt(N) <= 90 times larger than
the result: 1.1e-4 norm-wise, doubled.
"""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from cardiax_gb300 import _native as N  # noqa: E402
from cardiax_gb300 import adjoint as A  # noqa: E402
from cardiax_gb300 import params as Pm  # noqa: E402
from cardiax_gb300.stimulus import Protocol, Stimulus  # noqa: E402
from cardiax_gb300.tissue import stream_handle  # noqa: E402


# lines of 20 cells on, every residue of H mod 2 and W mod 4; the experiments together make more tiles
# than the device runs at once (two to some eight per block), or one alone does
@pytest.mark.parametrize("H,W,E", [(20, 20, 330), (21, 35, 310), (33, 66, 160), (40, 129, 90), (87, 85, 40),
                                   (64, 64, 100)])
@pytest.mark.parametrize("n", [1, 4])
def test_many_experiments_equal_one_at_a_time(H, W, E, n):
    L = A._lib()
    g = torch.Generator().manual_seed(H * 1000 + W)
    pitch = A.pitch_of(W)
    grid, ns = N.Grid(H, W, pitch), 3 * H * pitch
    i, j = np.meshgrid(np.arange(H), np.arange(W), indexing="ij")
    D = A.to_pitched(torch.tensor(1e-3 * (1 + 0.3 * np.sin(i / 5) * np.cos(j / 7)), dtype=torch.float32), H, W,
                     pitch, torch.device("cuda"))
    params = Pm.PARAMSET_4A
    f = np.zeros((H, W), np.float32)
    f[H // 3: H // 2, W // 3: W - 2] = 1.5
    stims = [[Stimulus(Protocol(k % 4, 2, 50), f)] if k % 3 else [] for k in range(E)]
    tables = A.stimulus_tables(stims, H, W, pitch, torch.device("cuda"))
    nan = float("nan")

    def padded(*lead):  # not-a-number in the rows' padding: nothing may read it
        x = torch.full(lead + (H, pitch), nan)
        x[..., :W] = torch.rand(lead + (H, W), generator=g)
        return x.cuda()

    buf, lam0, inj = padded(E, n, 3), padded(E, 3) - 0.5, padded(E, 3)
    slots = int(L.fk_adjoint_slots(grid))
    P = A.params_struct(params)
    steps = (ctypes.c_int64 * 1)(7 + n // 2)

    def run(e0, e1):
        m = e1 - e0
        lam, tmp = lam0[e0:e1].clone(), torch.full_like(lam0[e0:e1], nan)
        gD = torch.zeros((m, H, pitch), device="cuda")
        gth = torch.zeros((m, slots, 16), dtype=torch.float64, device="cuda")
        wsb = int(L.fk_adjoint_batch_workspace_bytes(m))
        ws = torch.empty(wsb, dtype=torch.uint8, device="cuda")
        sp = (ctypes.POINTER(N.Stimulus) * m)(*[ctypes.cast(t[0], ctypes.POINTER(N.Stimulus)) for t in tables[e0:e1]])
        nst = (ctypes.c_int * m)(*[t[1] for t in tables[e0:e1]])
        grads = (ctypes.c_void_p * 1)(inj[e0:e1].data_ptr())
        rc = L.fk_adjoint_batch_range(m, grid, buf[e0:e1].data_ptr(), n * ns, 7, n, D.data_ptr(), ctypes.byref(P), sp,
                                      nst, 0.01, 0.01, lam.data_ptr(), tmp.data_ptr(), steps, grads, 1, gD.data_ptr(),
                                      gth.data_ptr(), ws.data_ptr(), wsb, stream_handle())
        assert rc == 0
        return lam[..., :W], gD[..., :W], gth.sum(1)

    many = run(0, E)
    assert all(torch.isfinite(x).all() for x in many)
    for e in sorted({0, 1, 2, E // 2, E - 2, E - 1}):
        one = run(e, e + 1)
        assert torch.equal(one[0][0], many[0][e]) and torch.equal(one[1][0], many[1][e])
        d = (one[2][0] - many[2][e]).norm() / one[2][0].norm()
        assert float(d) < 2.2e-4


@pytest.mark.parametrize("H,W,E", [(16, 16, 1), (21, 35, 3), (64, 65, 17), (300, 131, 2)])
def test_sums_over_the_experiments(H, W, E):
    """dL/dD: the same float32 additions in the same order.  dL/dtheta: float64 sums of some thousand terms of
    one sign, 1e3 * 2^-53 apart at most, then rounded once to float32."""
    L = A._lib()
    pitch = A.pitch_of(W)
    grid = N.Grid(H, W, pitch)
    g = torch.Generator().manual_seed(7)
    gD = torch.full((E, H, pitch), float("nan"))
    gD[..., :W] = torch.randn((E, H, W), generator=g)
    gD = gD.cuda()
    gth = torch.rand((E, int(L.fk_adjoint_slots(grid)), 16), generator=g, dtype=torch.float64).cuda()
    oD, oth = torch.full((H * W + 8,), 7.0, device="cuda"), torch.full((16,), 7.0, device="cuda")
    assert L.fk_adjoint_sum(E, grid, gD.data_ptr(), gth.data_ptr(), oD.data_ptr(), oth.data_ptr(), stream_handle()) == 0
    want = gD[0, :, :W].clone()
    for e in range(1, E):
        want += gD[e, :, :W]
    assert torch.equal(oD[:H * W].view(H, W), want) and (oD[H * W:] == 7.0).all() and (oth[13:] == 7.0).all()
    ref = gth[..., :13].sum((0, 1))
    assert ((oth[:13].double() - ref).abs() <= 2.0 ** -24 * ref * (1 + 1e-6)).all()
