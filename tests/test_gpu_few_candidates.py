"""The fp32 path sweeps one reference with few candidates from the images as they are, everything else from
packed images: the same maps, on both sides of the line (as many candidates as cameras)."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("n", [1, 3, 4, 5])
@pytest.mark.parametrize("cameras", [3, 4])
def test_one_reference_equals_a_group(ss, native, synthetic, n, cameras):
    cols, rows = 70, 45
    cals = ss.parse_json_calib(synthetic.basalt_calibration(synthetic.square_rig(cols, rows)), [cols, rows], DEV)[:cameras]
    masks = [torch.ones(1, rows, cols, device=DEV) for _ in cals]

    def estimator(refs):
        return ss.RGBD_Estimator(cals, 0.4, 100.0, n, refs, torch.zeros(3, device=DEV), masks, (cols, rows), (64, 48),
                                 (80, 40), 10.0, 25.0, DEV)

    gen = torch.Generator(device=DEV).manual_seed(n)
    match = [torch.floor(torch.rand(rows, cols, 3, generator=gen, device=DEV) * 255) for _ in cals]
    stitch = [torch.zeros(48, 64, 3, device=DEV) for _ in range(2)]
    views = [im.permute(2, 0, 1)[None, :, None] for im in match]
    both = estimator([2, 0])
    both.estimate_RGBD_panorama(match, stitch)
    want = [both.fishey_stitcher.distances_stacked.clone(), both.distance_raw_maps.clone(), both.index_maps.clone()]
    for slot, r in enumerate((2, 0)):
        alone = estimator([r])
        alone.estimate_RGBD_panorama(match, stitch[:1])
        for a, w in zip((alone.fishey_stitcher.distances_stacked, alone.distance_raw_maps, alone.index_maps), want):
            assert torch.equal(a[0], w[slot])
        out = both.estimate_fisheye_distance(views[r], ss.rgb_to_guide(match[r]), None, None, views)
        assert torch.equal(out, want[0][slot])
