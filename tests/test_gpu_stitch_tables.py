"""Entries of Stitcher.inpainting_weights_list that a caller replaces are the tables the holes are filled
with, in the frame path as in the batched ones."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def test_a_replaced_table_is_used(ss, native, golden_small):
    from test_gpu_pipeline import _build

    (est, _), (other, _) = _build(ss, golden_small), _build(ss, golden_small)
    st, so = est.fishey_stitcher, other.fishey_stitcher
    maps = [(1 + 50 * torch.rand(st.rows, st.cols, generator=torch.Generator().manual_seed(r))).to(DEV)
            for r in range(st.reference_count)]
    images = [torch.zeros_like(im) for im in st.images_to_stitch_list]
    _, before = st.stitch(images, maps)
    before = before.clone()
    table = st.inpainting_weights_list[1].roll(5, 1).contiguous()
    so.inpainting_weights_list[1].copy_(table)  # in place
    _, want = so.stitch(images, maps)
    st.inpainting_weights_list[1] = table  # replaced
    _, got = st.stitch(images, maps)
    assert torch.equal(got, want) and not torch.equal(got, before)


def test_one_reference_at_a_time(ss, native, golden_small):
    """reproject_and_inpaint of each reference gives that reference's map of a whole stitch."""
    from test_gpu_pipeline import _build

    est, _ = _build(ss, golden_small, references_indices=[2, 0, 3])
    st = est.fishey_stitcher
    maps = [(1 + 50 * torch.rand(st.rows, st.cols, generator=torch.Generator().manual_seed(r))).to(DEV) for r in range(3)]
    st.stitch(st.images_to_stitch_list, maps)
    want = st.reprojected_distances.clone()
    st.reprojected_distances.zero_()
    for r in (1, 2, 0):
        st.reproject_and_inpaint(r, maps[r])
    assert torch.equal(st.reprojected_distances, want)
    for r in (-1, 3):
        with pytest.raises(IndexError):
            st.reproject_and_inpaint(r, maps[0])
