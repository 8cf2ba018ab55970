"""The schedules and the tuners run the kernels that they name."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from cardiax_gb300 import _native as N  # noqa: E402
from cardiax_gb300 import params as Pm  # noqa: E402
from cardiax_gb300.batch import TissueBatch  # noqa: E402
from cardiax_gb300.stimulus import Protocol, Stimulus  # noqa: E402
from cardiax_gb300.tissue import Tissue  # noqa: E402


def _tissue(H, W, k=0):
    f = np.zeros((H, W), np.float32)
    f[:4] = 20.0
    t = Tissue((H, W), Pm.PARAMSET_3, np.full((H, W), 1e-3, np.float32), [Stimulus(Protocol(0, 2, 900), f)])
    t.params.tau_d *= 1.0 + 0.01 * k
    return t


def _takes_resident(plan, steps=64):
    return N.lib().fk_batch_takes_resident(plan, steps)


@pytest.mark.parametrize("rows", [16, 32])
def test_the_batch_schedule_is_the_batched_kernel(rows):
    t, u = _tissue(64, 80), _tissue(64, 80)
    assert _takes_resident(TissueBatch([t])._plan) == 1  # a batch's own default
    t.advance(0, 64, schedule="batch", tile_rows=rows)
    assert _takes_resident(t._one_batch(rows)._plan) == 0
    u.advance(0, 64)
    for a, b in zip(t.view(), u.view()):
        assert torch.equal(a, b)


KNOBS = dict(trial_steps=64, candidates=(0,), tile_rows=(32,), options=((1, False),), depths=(1,))


def test_batches_of_the_same_shapes_are_tuned_apart():
    """37 sets of constants are three resident launches, which the plan never takes; one set is one launch.
    Tracked tissues cannot take it.  Whichever is tuned first must not decide for the others."""
    from cardiax_gb300.autotune import tune_batch
    for turn in range(2):  # measured, then from the cache
        many = TissueBatch([_tissue(48, 52, k) for k in range(37)])
        res = tune_batch(many, **KNOBS)
        assert res["resident"] is False and res["resident_ms_per_step"] is None
        one = TissueBatch([_tissue(48, 52) for _ in range(37)])
        res = tune_batch(one, **KNOBS)
        assert res["resident_ms_per_step"] > 0
        assert res["resident"] == (res["resident_ms_per_step"] < min(res["ms_per_step"].values()))
        assert _takes_resident(one._plan) == res["resident"]
        tracked = TissueBatch([_tissue(48, 52).track_activation(0.5) for _ in range(37)])
        res = tune_batch(tracked, **KNOBS)
        assert res["resident"] is False and res["resident_ms_per_step"] is None
