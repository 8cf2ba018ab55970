"""Rollouts by checkpoints with more marks than one call writes: buffers used again by later calls must not reach
states that were kept.  Against every state kept (the same bits), with the calls counted."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from cardiax_gb300 import adjoint as A  # noqa: E402
from cardiax_gb300 import params as Pm  # noqa: E402
from test_gpu_forward_states import _inputs  # noqa: E402

OBS = [0, 3, 3] + list(range(5, 45)) + [12]


@pytest.mark.parametrize("H,W", [(40, 52), (70, 131)])
@pytest.mark.parametrize("seg", [1, 6, 7, 23])
def test_marks_over_several_calls(H, W, seg, monkeypatch):
    D, x, st = _inputs(H, W)
    written = []
    step_list = A._step_list
    monkeypatch.setattr(A, "_step_list", lambda steps, outs: written.append(list(steps)) or step_list(steps, outs))

    def run(seg):
        Dl, xl = D.clone().requires_grad_(True), x.clone().requires_grad_(True)
        th = torch.tensor(Pm.PARAMSET_3[:13], device="cuda", requires_grad=True)
        out = A.rollout(xl[0], xl[1], xl[2], Dl, th, st, 0, 50, OBS, seg=seg)
        one = len(written)
        (out * torch.linspace(0.5, 1.5, len(OBS), device="cuda").view(-1, 1, 1, 1)).sum().backward()
        xb = torch.stack([x, 0.9 * x, 0.8 * x]).requires_grad_(True)
        Db = D.clone().requires_grad_(True)
        outb = A.rollout_batch(xb, Db, th, [st] * 3, 0, 50, OBS, seg=seg)
        (outb ** 2).sum().backward()
        return one, [out.detach(), xl.grad, Dl.grad, th.grad, outb.detach(), xb.grad, Db.grad]

    _, want = run(None)
    assert not written  # every state kept
    one, got = run(seg)
    marks = sorted(set(OBS) | set(range(0, 44, seg)))
    assert len(marks) > A.STATES_PER_CALL
    calls = -(-len(marks) // A.STATES_PER_CALL)
    assert one == calls and len(written) == 2 * calls
    assert sum(written[:calls], []) == marks and sum(written[calls:], []) == marks
    for p, q in zip(want, got):
        assert torch.isfinite(p).all() and torch.equal(p, q)
