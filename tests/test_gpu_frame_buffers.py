"""The fp32 path's cost filter holds the pyramid of the reference worked on last, whichever call that
was, and the same object holds it from call to call."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _inputs(g):
    match = [torch.as_tensor(im, device=DEV).float() for im in g["images_to_match"]]
    return match, [torch.zeros(100, 120, 3, device=DEV) for _ in range(4)]


@pytest.mark.parametrize("refs", [[2, 3], [3, 0, 1], [0, 1, 2, 3]])
def test_cost_filter_is_the_last_reference(ss, native, golden_small, refs):
    from test_gpu_pipeline import _build

    g = golden_small
    est, cfg = _build(ss, g, references_indices=refs)
    match, stitch = _inputs(g)
    held = est.cost_filter

    def expect(reference):
        alone, _ = _build(ss, g, references_indices=[reference])
        alone.estimate_RGBD_panorama(match, stitch[:1])
        want = alone.cost_filter
        for level in range(len(want.costs)):
            assert torch.equal(held.costs[level], want.costs[level]), (reference, level)
            assert torch.equal(held.guides[level], want.guides[level]), (reference, level)
            assert torch.equal(est.cost_filter.costs[level], want.costs[level])

    est.estimate_RGBD_panorama(match, stitch[:len(refs)])
    expect(refs[-1])
    views = [im.permute(2, 0, 1)[None, :, None] for im in match]
    for slot, r in enumerate(refs):
        est.estimate_fisheye_distance(views[r], ss.rgb_to_guide(match[r]), est.calibrations[r],
                                      est.selected_cameras[slot], views)
        expect(r)
