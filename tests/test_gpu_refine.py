"""The differentiable sweep of several references at once (csrc/ssg_refine.cu) against the per-step entry
points, one reference after the other: inverse distances, filter gradients and image gradients bit
for bit, pose gradients within float64 rounding of sums in another order.  Sizes around the 32-pixel
groups, the 32 x 8 tiles and the small levels' launch, odd ones, more references than one launch
takes, and a gradient that is not finite."""
from __future__ import annotations

import importlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _per_step(N, isb, sweep, images, rel, grad_q):
    """Forward and backward with the per-step entry points."""
    stream = torch.cuda.current_stream().cuda_stream
    cols, rows, n, L, shapes = sweep.cols, sweep.rows, sweep.N, sweep.L, sweep.shapes
    weights, var = isb.level_weights(L, sweep.sigma_s), 1 / (2 * sweep.sigma_i ** 2)
    f32, u8 = dict(dtype=torch.float32, device=DEV), dict(dtype=torch.uint8, device=DEV)
    costs, gf, gc = ([torch.empty(n, r, c, **f32) for r, c in shapes] for _ in range(3))
    g_orig, g_filt = ([torch.empty(r, c, 3, **u8) for r, c in shapes] for _ in range(2))
    grads, pose = torch.zeros_like(images), torch.zeros(sweep.C, 6, dtype=torch.float64, device=DEV)
    bytes_ = N.library().ssg_sweep_backward_scratch_bytes(cols, rows, sweep.C)
    scratch = torch.empty((bytes_ + 255) // 256 * 256, **u8)
    im = N.pointers([images[c].data_ptr() for c in range(sweep.C)])
    gi = N.pointers([grads[c].data_ptr() for c in range(sweep.C)])
    q = torch.empty(len(sweep.refs), rows, cols, device=DEV)
    for slot, r in enumerate(sweep.refs):
        poses = N.floats(rel[slot])
        N.call("ssg_rgb_to_guide", images[r].data_ptr(), rows * cols, g_orig[0].data_ptr(), stream)
        N.call("ssg_sweep_cost", cols, rows, sweep.C, sweep._cams, r, poses, im, sweep.selected[slot].data_ptr(),
               sweep._cand, n, costs[0].data_ptr(), stream)
        for s in range(1, L):
            N.call("ssg_isb_downsample", g_orig[s - 1].data_ptr(), costs[s - 1].data_ptr(), *shapes[s - 1],
                   g_orig[s].data_ptr(), costs[s].data_ptr(), *shapes[s], n, var, stream)
            g_filt[s].copy_(g_orig[s])
        for s in range(L - 2, 0, -1):
            N.call("ssg_isb_upsample", g_filt[s + 1].data_ptr(), costs[s + 1].data_ptr(), *shapes[s + 1],
                   g_filt[s].data_ptr(), costs[s].data_ptr(), *shapes[s], n, *weights[s], var, stream)
        last = (g_filt[1].data_ptr(), costs[1].data_ptr(), *shapes[1], g_orig[0].data_ptr(), costs[0].data_ptr(), rows,
                cols, n, *weights[0], var, sweep._cand, sweep.temperature)
        N.call("ssg_isb_upsample_softargmin", *last, q[slot].data_ptr(), stream)
        N.call("ssg_isb_upsample_softargmin_backward", *last, grad_q[slot].data_ptr(), gf[0].data_ptr(), stream)
        for s in range(L - 1):
            N.call("ssg_isb_upsample_transpose", g_filt[s + 1].data_ptr(), *shapes[s + 1], g_orig[s].data_ptr(),
                   *shapes[s], n, *weights[s], var, gf[s].data_ptr(), gc[s].data_ptr(), gf[s + 1].data_ptr(), stream)
        gc[L - 1].copy_(gf[L - 1])
        for s in range(L - 1, 0, -1):
            N.call("ssg_isb_downsample_transpose", g_orig[s - 1].data_ptr(), *shapes[s - 1], *shapes[s], n, var,
                   gc[s].data_ptr(), gc[s - 1].data_ptr(), stream)
        N.call("ssg_sweep_cost_backward", cols, rows, sweep.C, sweep._cams, r, poses, im, gi,
               sweep.selected[slot].data_ptr(), sweep._cand, n, gc[0].data_ptr(), pose.data_ptr(), scratch.data_ptr(),
               stream)
    return q, grads, pose, gc[0]


@pytest.mark.parametrize("cols,rows,n,refs", [(64, 64, 16, [2, 3]), (33, 40, 5, [1]), (97, 75, 17, [0, 1, 2, 3, 1]),
                                              (130, 66, 9, [3, 0]), (40, 200, 8, [2]),
                                              (264, 250, 3, [0, 1, 2, 3, 1]), (263, 251, 5, [0, 1, 2, 3, 1])])
@pytest.mark.parametrize("finite", [True, False])
def test_equals_the_per_step_entry_points(ss, native, synthetic, cols, rows, n, refs, finite):
    N = ss._native
    rng = np.random.default_rng(cols * rows + n)
    cals = ss.parse_json_calib(synthetic.basalt_calibration(synthetic.square_rig(cols, rows)), [cols, rows], "cpu")
    masks = [torch.ones(1, rows, cols) for _ in cals]
    sweep = ss.DifferentiableSweep(cals, 0.4, 100.0, n, refs, masks, (cols, rows), 10.0, 6.0, DEV)
    smooth = rng.random((4, rows // 4 + 2, cols // 4 + 2, 3)).repeat(4, 1).repeat(4, 2)[:, :rows, :cols] * 255
    images = torch.as_tensor(np.floor(smooth).astype(np.float32), device=DEV)
    images[:, : rows // 3] += torch.as_tensor(rng.random((4, rows // 3, cols, 3)).astype(np.float32), device=DEV)
    grad_q = torch.as_tensor(rng.standard_normal((len(refs), rows, cols)).astype(np.float32), device=DEV)
    grad_q[0, rows // 2:, : cols // 2] = 0
    if not finite:
        grad_q[-1, 3, 4] = float("inf")
    zero = torch.zeros(len(cals), 6, dtype=torch.float64, device=DEV)
    poses = sweep._poses(zero)
    isb = importlib.import_module("sphere-stereo_gb300.isb_filter")
    want_q, want_images, want_pose, want_gc = _per_step(N, isb, sweep, images, poses.relative, grad_q)
    assert torch.equal(sweep.forward(images, zero), want_q)
    got_images, got_pose = sweep.backward(images, zero, grad_q)
    last = (len(refs) - 1) % sweep.group
    got_gc = sweep.gc[0].view(sweep.group, n, rows, cols)[last]
    assert torch.equal(got_gc.nan_to_num(), want_gc.nan_to_num())
    assert torch.equal(got_images.nan_to_num(), want_images.nan_to_num())
    assert torch.equal(got_images.isnan(), want_images.isnan()) and bool(got_images.isnan().any()) != finite
    if finite:
        # float64 sums of the same float32 values: the order's rounding, of the values' magnitude
        torch.testing.assert_close(got_pose, want_pose, rtol=1e-10, atol=1e-12 * float(want_pose.abs().max()))
