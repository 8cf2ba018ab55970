"""Classification of stimulus fields on the device against the definition, one field at a time and
many in one call."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _definition(f):
    nz = f != 0
    rows, cols = np.flatnonzero(nz.any(1)), np.flatnonzero(nz.any(0))
    if rows.size == 0:
        return ("empty",)
    r0, r1, c0, c1 = rows[0], rows[-1] + 1, cols[0], cols[-1] + 1
    box = f[r0:r1, c0:c1]
    return ("rect", r0, r1, c0, c1, float(box[0, 0])) if (box == box[0, 0]).all() else ("dense",)


def _fields(H, W):
    rng = np.random.default_rng(H * 100 + W)
    out = []

    def add(edit, base=0.0):
        f = np.full((H, W), base, np.float32)
        edit(f)
        out.append(f)

    add(lambda f: None)                                        # empty
    add(lambda f: f.__setitem__((0, 0), -0.0))                 # a negative zero is zero
    add(lambda f: f.__setitem__((H - 1, W - 1), 2.5))          # one cell
    add(lambda f: None, base=-3.0)                             # everything
    add(lambda f: f.__setitem__((slice(0, 3), slice(None)), 20.0))
    add(lambda f: f.__setitem__((slice(1, H), slice(W // 2, W)), -1e-40))  # a subnormal
    add(lambda f: f.__setitem__((slice(0, 2), slice(0, 2)), np.inf))
    add(lambda f: f.__setitem__((slice(0, 2), slice(0, 2)), np.nan))

    def hole(f):
        f[0:3, 0:3] = 4.0
        f[1, 1] = 0.0

    def two(f):
        f[0, 0] = f[H - 1, W - 1] = 1.0

    def signs(f):
        f[0:2, 0:2] = 1.0
        f[0, 0] = -1.0

    def last_bit(f):
        f[0:2, 0:3] = 1.0
        f[1, 2] = np.nextafter(np.float32(1), np.float32(2))

    for edit in (hole, two, signs, last_bit, lambda f: f.__setitem__(slice(None), rng.random((H, W)))):
        add(edit)
    return out


@pytest.mark.parametrize("H,W", [(3, 3), (5, 257), (700, 3), (64, 64), (333, 517), (1200, 1200)])
def test_field_kinds(H, W):
    from cardiax_gb300.tissue import analyse_field, analyse_fields
    fields = _fields(H, W)
    dev = [torch.as_tensor(f).cuda() for f in fields]
    many = analyse_fields(dev * 6)  # more than one launch takes
    for k, f in enumerate(fields):
        want = _definition(f)
        assert analyse_field(dev[k]) == want
        assert many[k] == want and many[k + 5 * len(fields)] == want
    t = dev[4].t()  # strides of a transpose, and of a wider buffer
    assert analyse_field(t) == _definition(fields[4].T)
    wide = torch.zeros((H, W + 3), device="cuda")
    wide[:, :W] = dev[4]
    wide[:, W:] = 9.0
    assert analyse_field(wide[:, :W]) == _definition(fields[4])
