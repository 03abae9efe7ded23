"""The sweep of several references from packed images (csrc/ssg_sweep.cu) equals ssg_sweep_cost bit for
bit: sizes that are and are not powers of two, one to five references (two launches), a reference
listed twice, candidate counts on both sides of the sharing rule, pixels without a camera, and samples
outside the images; and the packed guides equal ssg_rgb_to_guide."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("cols,rows,n,refs", [(64, 64, 32, [2, 3]), (67, 45, 17, [0]), (130, 97, 64, [1, 0, 3, 2, 1]),
                                              (33, 128, 5, [3, 3])])
def test_equals_the_sweep_per_reference(ss, native, synthetic, cols, rows, n, refs):
    N = ss._native
    stream = torch.cuda.current_stream().cuda_stream
    rng = np.random.default_rng(cols + n)
    cals = ss.parse_json_calib(synthetic.basalt_calibration(synthetic.square_rig(128, 100)), [cols, rows], "cpu")
    utils = __import__("importlib").import_module("sphere-stereo_gb300.utils")
    cams = N.cameras_array([utils.camera_struct(c) for c in cals])
    images = [torch.as_tensor((rng.random((rows, cols, 3)) * 255).astype(np.float32), device=DEV) for _ in cals]
    poses = [utils.relative_poses(cals, r) for r in refs]
    selected = torch.as_tensor(rng.integers(-1, len(cals), (len(refs), rows, cols)).astype(np.int8), device=DEV)
    cand = N.floats(ss.distance_candidates(0.3, 100.0, n).tolist())
    pointers = N.pointers([im.data_ptr() for im in images])
    packed = torch.empty(len(cals), rows, cols, 4, device=DEV)
    guides = torch.empty(len(refs), rows, cols, 3, dtype=torch.uint8, device=DEV)
    cost = torch.empty(len(refs), n, rows, cols, device=DEV)
    N.call("ssg_pack_images", pointers, len(cals), rows * cols, N.ints(refs), len(refs), packed.data_ptr(),
           guides.data_ptr(), stream)
    N.call("ssg_sweep_cost_references", cols, rows, len(cals), cams, len(refs), N.ints(refs),
           N.floats([v for p in poses for v in p]), packed.data_ptr(), selected.data_ptr(), cand, n, cost.data_ptr(),
           stream)
    for slot, r in enumerate(refs):
        want = torch.empty(n, rows, cols, device=DEV)
        N.call("ssg_sweep_cost", cols, rows, len(cals), cams, r, N.floats(poses[slot]), pointers,
               selected[slot].data_ptr(), cand, n, want.data_ptr(), stream)
        assert torch.equal(cost[slot], want)
        assert torch.equal(guides[slot], ss.rgb_to_guide(images[r]))
