"""Which calls of the blur factor their weights: those whose direct sum takes longer than that costs."""
import numpy as np
import pytest
import torch

from cardiax_gb300 import scars


@pytest.mark.parametrize("H,W,K,two_passes", [
    (64, 64, 8, False), (64, 64, 20, False), (256, 256, 25, False), (400, 400, 16, False), (800, 800, 16, False),
    (1200, 1200, 10, False), (1200, 1200, 513, False), (64, 64, 64, True), (400, 400, 50, True),
    (800, 800, 40, True), (1200, 1200, 32, True), (1200, 1200, 120, True), (2000, 2000, 20, True)])
def test_blur_route(H, W, K, two_passes, monkeypatch):
    taken = []
    monkeypatch.setattr(scars.N, "call", lambda name, *a: taken.append(name))
    monkeypatch.setattr(scars, "stream_handle", lambda: 0)
    w = scars.gaussian_weights(K, np.float32(K / 3))
    scars.blur_same(torch.zeros((H, W)), w)
    assert taken == ["fk_conv2d_separable" if two_passes else "fk_conv2d_same"]
