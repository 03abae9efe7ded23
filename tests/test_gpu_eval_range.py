"""The sums of the distance errors (csrc/ssg_eval.cu) beyond float32's range: finite errors whose sum,
or whose squares' sum, exceeds 3.4e38 give the finite mean that float64 sums give."""
from __future__ import annotations

import importlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("scale", [1.0, 1e10, 1e15, 8e18])
@pytest.mark.parametrize("rows,cols", [(64, 512), (37, 111), (1100, 2048), (999, 2051)])
def test_sums_of_large_errors(rows, cols, scale):
    """Errors are float32 differences, squares float32 products; their sums are compared with float64's,
    which are within 2^-53 of a sum of n terms per addition (n 2^-53 < 1e-10)."""
    ev = importlib.import_module("sphere-stereo_gb300.evaluation")
    rng = np.random.default_rng(rows)
    rgb = rng.integers(0, 256, (2, rows, cols, 3)).astype(np.uint8)
    gt_inv = rng.random((2, rows, cols), dtype=np.float32)
    inv = (gt_inv + rng.random(gt_inv.shape, dtype=np.float32)).astype(np.float32)
    large = rng.random(inv.shape) < 0.3
    inv[large] = (scale * (1 + rng.random(int(large.sum())))).astype(np.float32)
    e = np.abs(inv - gt_inv)
    squares = e * e
    assert e.dtype == squares.dtype == np.float32
    out = ev.evaluate_panoramas(*(torch.as_tensor(a, device=DEV) for a in (rgb, inv, rgb, gt_inv))).cpu().numpy()
    for f in range(2):
        np.testing.assert_allclose(out[f, 2], e[f].astype(np.float64).mean(), rtol=1e-10)
        np.testing.assert_allclose(out[f, 3], np.sqrt(squares[f].astype(np.float64).mean()), rtol=1e-10)


def test_the_largest_errors():
    """Errors of the float32 maximum: their sum is held, their squares are infinite as float32 products."""
    ev = importlib.import_module("sphere-stereo_gb300.evaluation")
    rgb = np.zeros((40, 64, 3), np.uint8)
    inv, gt = np.full((40, 64), np.finfo(np.float32).max), np.zeros((40, 64), np.float32)
    inv = inv.astype(np.float32)
    out = ev.evaluate_panoramas(*(torch.as_tensor(a, device=DEV) for a in (rgb, inv, rgb, gt)), [1.0]).cpu().numpy()
    assert out[0, 2] == float(np.finfo(np.float32).max) and np.isposinf(out[0, 3]) and out[0, 4] == 100.0
