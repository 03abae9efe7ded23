"""float -> uint8 of the images to stitch (csrc/ssg_sweep_batch.cu, convert_u8_kernel) for values outside
[0, 255], as torch's copy converts them (the low byte of the truncated integer): no value reaches
another one's byte, with and without 16-byte alignment, in whole blocks and in the last one."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

SPECIAL = [-0.5, -1.0, -1.5, -255.0, -256.0, -300.25, -2.0 ** 31, -3e9, -1e19, -1e30, -np.inf, np.nan, 255.999, 256.0,
           257.5, 300.5, 511.0, 65535.75, 2147483520.0, 2.0 ** 31, 2.0 ** 31 + 256, 2.0 ** 32, 5e9, 9.2e18, 2.0 ** 63,
           1e30, np.inf]


@pytest.mark.parametrize("offset", [0, 1, 3])
@pytest.mark.parametrize("n", [1, 17, 4096, 3 * 4096 + 2047])
def test_values_outside_a_byte(ss, native, n, offset):
    rng = np.random.default_rng(n + offset)
    values = rng.uniform(-700, 700, n + offset).astype(np.float32)
    at = rng.integers(0, n + offset, (n + offset) // 3)
    values[at] = rng.choice(np.array(SPECIAL, np.float32), at.size)
    src = torch.as_tensor(values, device=DEV)[offset:]
    dst = torch.empty(n + offset, dtype=torch.uint8, device=DEV)[offset:]
    ss._native.call("ssg_convert_u8", src.data_ptr(), dst.data_ptr(), n, torch.cuda.current_stream().cuda_stream)
    want = torch.empty_like(dst).copy_(src)
    bad = (dst != want).nonzero().flatten()[:5]
    assert torch.equal(dst, want), (src[bad], dst[bad], want[bad])


def test_a_frame_with_values_outside_a_byte(ss, native, golden_small):
    """The frame path converts its images to stitch as copy_ would."""
    from test_gpu_pipeline import _build

    est, _ = _build(ss, golden_small)
    match = [torch.as_tensor(im, device=DEV).float() for im in golden_small["images_to_match"]]
    stitch = [torch.as_tensor(im, device=DEV).float() * 1.5 - 40 for im in golden_small["images_to_stitch"]]
    est.estimate_RGBD_panorama(match, stitch)
    for image, got in zip(stitch, est.fishey_stitcher.images_to_stitch_list):
        assert torch.equal(got, torch.empty_like(got).copy_(image))
