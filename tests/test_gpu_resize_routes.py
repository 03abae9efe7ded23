"""Both kernels of the linear resize give equal values: a batch large enough for the kernel of whole rows
against the same images two at a time, which the kernel of single pixels takes (and which
test_gpu_resize_rows.py compares with the oracle).  Sizes at the edges of the blocks (768 values of 8
rows), rows that are not whole fours, results at any offset, kept rows, area averages."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("src,dst,ch,images", [
    ((300, 40), (256, 16), 3, 200), ((300, 40), (257, 17), 3, 600), ((91, 33), (255, 15), 3, 200),
    ((41, 9), (385, 33), 2, 200), ((800, 7), (769, 5), 1, 300), ((64, 90), (193, 31), 4, 1200),
    ((500, 100), (130, 20), 3, 1000), ((514, 66), (257, 33), 3, 1000), ((30, 20), (15, 10), 1, 9000),
    ((90, 130), (45, 65), 2, 12000), ((900, 700), (1021, 997), 3, 2)])
@pytest.mark.parametrize("offset", [0, 1])
def test_batches_equal_single_images(ss, native, src, dst, ch, images, offset):
    N = ss._native
    rng = np.random.default_rng(src[0] * 7 + dst[0])
    two = torch.as_tensor(rng.integers(0, 256, (2, src[1], src[0], ch), dtype=np.uint8), device=DEV)
    values = dst[0] * dst[1] * ch
    code = {torch.float32: N.PIXEL_F32, torch.uint8: N.PIXEL_U8}

    def resize(t, kind):
        n = t.shape[0]
        out = torch.full((n * values + offset + 4,), 77, dtype=kind, device=DEV)
        N.call("ssg_resize_linear", t.data_ptr(), code[t.dtype], src[0], src[1], ch, out[offset:].data_ptr(), code[kind],
               dst[0], dst[1], n, torch.cuda.current_stream().cuda_stream)
        assert bool((out[:offset] == 77).all()) and bool((out[offset + n * values:] == 77).all())
        return out[offset: offset + n * values].view(n, values)

    for x, kind in ((two, torch.float32), (two.float() + 0.25, torch.float32), (two, torch.uint8)):
        # one image at a time for the last size, whose two images already make a batch
        want = torch.cat([resize(x[i:i + 1], kind) for i in range(2)])
        got = resize(x.repeat(images // 2, 1, 1, 1), kind).view(images // 2, 2, values)
        assert torch.equal(got, want.expand_as(got))
