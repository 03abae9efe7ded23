"""ssg_sweep_backward_references with more references than one launch takes (4): five in one call equal
the same five in a call of four and one of one, which is what DifferentiableSweep makes of them."""
from __future__ import annotations

import importlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("cols,rows,n", [(33, 40, 5), (97, 24, 9)])
def test_five_references_in_one_call(ss, native, synthetic, cols, rows, n):
    N, utils = ss._native, importlib.import_module("sphere-stereo_gb300.utils")
    rng = np.random.default_rng(cols)
    refs = [0, 3, 1, 2, 3]
    cals = ss.parse_json_calib(synthetic.basalt_calibration(synthetic.square_rig(cols, rows)), [cols, rows], "cpu")
    C, R, P = len(cals), len(refs), cols * rows
    cams = N.cameras_array([utils.camera_struct(c) for c in cals])
    poses = [v for r in refs for v in utils.relative_poses(cals, r)]
    images = torch.as_tensor((rng.random((C, rows, cols, 3)) * 255).astype(np.float32), device=DEV)
    packed = torch.nn.functional.pad(images, (0, 1)).contiguous()
    selected = torch.as_tensor(rng.integers(-1, C, (R, rows, cols)).astype(np.int8), device=DEV)
    grad = torch.as_tensor(rng.standard_normal((R, n, rows, cols)).astype(np.float32), device=DEV)
    absmax = grad.abs().amax((1, 2, 3)).view(torch.int32).contiguous()
    cand = N.floats(ss.distance_candidates(0.3, 100.0, n).tolist())
    stream = torch.cuda.current_stream().cuda_stream

    def run(calls):
        out, pose = torch.zeros_like(images), torch.zeros(C, 6, dtype=torch.float64, device=DEV)
        targets = N.pointers([out[c].data_ptr() for c in range(C)])
        for first, count in calls:
            size = N.library().ssg_sweep_backward_references_scratch_bytes(cols, rows, C, count)
            scratch = torch.empty((size + 255) // 256 * 256, dtype=torch.uint8, device=DEV)
            N.call("ssg_sweep_backward_references", cols, rows, C, cams, count, N.ints(refs[first:first + count]),
                   N.floats(poses[12 * C * first:12 * C * (first + count)]), packed.data_ptr(), targets,
                   selected[first].data_ptr(), cand, n, grad[first].data_ptr(), absmax[first:].data_ptr(),
                   pose.data_ptr(), scratch.data_ptr(), stream)
        return out, pose

    got, got_pose = run([(0, R)])
    want, want_pose = run([(0, 4), (4, 1)])
    assert bool(want.any()) and torch.equal(got, want)
    # float64 sums of the same float32 values in another order
    torch.testing.assert_close(got_pose, want_pose, rtol=1e-10, atol=1e-12 * float(want_pose.abs().max()))
