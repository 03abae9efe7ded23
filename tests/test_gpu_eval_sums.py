"""The evaluation sums (csrc/ssg_eval.cu) where their partition has edges: map columns around a warp's
58, one row of windows, strips of one row more than a whole number, arrays that are not 16-byte
aligned, sixteen thresholds, and distances that are not finite."""
from __future__ import annotations

import importlib

import numpy as np
import pytest
import torch

import prep_eval_oracle as po

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _frames(rows, cols, frames, seed):
    rng = np.random.default_rng(seed)
    gt = rng.integers(0, 256, (frames, rows, cols, 3)).astype(np.uint8)
    gt[:, : rows // 2] = np.clip(gt[:, : rows // 2] // 32 + 100, 0, 255)  # flat and textured halves
    est = np.clip(gt.astype(int) + rng.integers(-9, 10, gt.shape), 0, 255).astype(np.uint8)
    gt_inv = rng.random((frames, rows, cols), dtype=np.float32)
    inv = (gt_inv + 0.05 * rng.standard_normal(gt_inv.shape)).astype(np.float32)
    return est, inv, gt, gt_inv


@pytest.mark.parametrize("rows,cols,frames", [(7, 63, 2), (8, 64, 1), (65, 65, 3), (39, 122, 2), (520, 123, 1), (9, 7, 2)])
def test_partition_edges(rows, cols, frames):
    """Relative error of a window: two floats, 2^-43 for the ratio and 2^-41 for the corrections; the
    oracle's float64 window sums are about as far from the exact value: 1e-11 leaves a factor of ten."""
    ev = importlib.import_module("sphere-stereo_gb300.evaluation")
    data = _frames(rows, cols, frames, rows * cols)
    thresholds = [0.01 * k for k in range(16)]
    t = [torch.as_tensor(a, device=DEV) for a in data]
    out = ev.evaluate_panoramas(*t, thresholds).cpu().numpy()
    # the same values from arrays that start off a 16-byte boundary
    off = []
    for a in t:
        room = torch.empty(a.numel() + 1, dtype=a.dtype, device=DEV)[1:].view(a.shape)
        off.append(room.copy_(a))
    shifted = ev.evaluate_panoramas(*off, thresholds).cpu().numpy()
    for f in range(frames):
        want = po.evaluate(*(d[f] for d in data), thresholds)
        for got in (out[f], shifted[f]):
            np.testing.assert_allclose(got[:4], [want[k] for k in ("psnr", "ssim", "mae", "rmse")], rtol=1e-11)
            np.testing.assert_array_equal(got[4:], want["bad_px_ratios"])


def test_distances_that_are_not_finite():
    ev = importlib.import_module("sphere-stereo_gb300.evaluation")
    est, inv, gt, gt_inv = _frames(32, 64, 3, 1)
    inv[1, 3, 5] = np.inf
    inv[2, 4, 6] = np.nan
    out = ev.evaluate_panoramas(*(torch.as_tensor(a, device=DEV) for a in (est, inv, gt, gt_inv)), [0.1]).cpu().numpy()
    assert np.isfinite(out[0]).all() and np.isfinite(out[:, :2]).all()
    assert np.isposinf(out[1, 2:4]).all() and np.isnan(out[2, 2:4]).all()
