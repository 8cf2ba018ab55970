"""Stimulus fields of any type and device are classified by their own values."""
import pytest
import torch

from cardiax_gb300.tissue import analyse_field, analyse_fields

TYPES = [torch.float64, torch.float16, torch.bfloat16, torch.bool, torch.int8, torch.uint8, torch.int32, torch.int64]


def _check(device):
    H, W = 7, 9
    for dtype in TYPES + [torch.float32]:
        f = torch.zeros((H, W), dtype=dtype, device=device)
        assert analyse_field(f) == ("empty",)
        f[2:5, 3:8] = 1
        assert analyse_field(f) == ("rect", 2, 5, 3, 8, 1.0)
        f[3, 4] = 0
        assert analyse_field(f) == ("dense",)
    # values that float32 does not tell apart, or from zero
    f = torch.zeros((H, W), dtype=torch.float64, device=device)
    f[:2, :2] = 1.0
    f[1, 1] += 2.0 ** -50
    assert analyse_field(f) == ("dense",)
    f[:2, :2] = 1e-60
    assert analyse_field(f) == ("rect", 0, 2, 0, 2, 1e-60)
    assert analyse_field(torch.zeros((0, 5), device=device)) == ("empty",)


def test_fields_on_the_cpu():
    _check("cpu")


@pytest.mark.gpu
def test_fields_on_the_gpu():
    _check("cuda")
    # types and devices mixed in one call keep their places
    f = torch.zeros((6, 5))
    f[1:3, 2:4] = 2.0
    g = f.clone()
    g[0, 0] = 1.0
    fields = [f, f.cuda(), g.cuda(), g.cuda().half(), f.cuda().double(), torch.zeros(6, 5).cuda()]
    rect = ("rect", 1, 3, 2, 4, 2.0)
    assert analyse_fields(fields) == [rect, rect, ("dense",), ("dense",), rect, ("empty",)]


def test_fields_of_different_shapes_are_refused():
    with pytest.raises(ValueError):
        analyse_fields([torch.zeros((4, 5)), torch.zeros((5, 4))])
    assert analyse_fields([]) == []
