"""The linear resize at the edges of its blocks (768 values of 16 rows), of its four-value stores (rows
that are not whole fours, results at any offset) and of its kept rows (enlarged, equal, reduced by
more than 2), against the oracle: equal values."""
from __future__ import annotations

import numpy as np
import prep_eval_oracle as po
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("src,dst,ch", [((300, 40), (256, 16), 3), ((300, 40), (257, 17), 3), ((91, 33), (255, 15), 3),
                                        ((41, 9), (385, 33), 2), ((800, 7), (769, 5), 1), ((64, 90), (193, 31), 4),
                                        ((500, 100), (130, 20), 3), ((1, 1), (5, 3), 3), ((514, 66), (257, 33), 3),
                                        ((30, 20), (15, 10), 1)])
@pytest.mark.parametrize("offset", [0, 1])
def test_resize_at_block_edges(ss, native, src, dst, ch, offset):
    N = ss._native
    rng = np.random.default_rng(src[0] * 11 + dst[0])
    u8 = rng.integers(0, 256, (2, src[1], src[0], ch), dtype=np.uint8)
    f32 = (rng.random((2, src[1], src[0], ch), dtype=np.float32) * 255).astype(np.float32)
    count = 2 * dst[0] * dst[1] * ch
    for x, kind in ((u8, torch.float32), (f32, torch.float32), (u8, torch.uint8)):
        t = torch.as_tensor(x, device=DEV)
        out = torch.full((count + offset + 4,), 77, dtype=kind, device=DEV)
        at = out[offset: offset + count]
        code = {torch.float32: N.PIXEL_F32, torch.uint8: N.PIXEL_U8}
        N.call("ssg_resize_linear", t.data_ptr(), code[t.dtype], src[0], src[1], ch, at.data_ptr(), code[kind], dst[0],
               dst[1], 2, torch.cuda.current_stream().cuda_stream)
        got = at.view(2, dst[1], dst[0], ch).cpu().numpy()
        for i in range(2):
            want = po.resize_linear(x[i], dst, np.uint8) if kind == torch.uint8 else po.resize_linear(x[i], dst)
            assert np.array_equal(got[i], want.reshape(got[i].shape))
        assert bool((out[:offset] == 77).all()) and bool((out[offset + count:] == 77).all())
