"""The exact merge reads pairs of RGB texels as words where every image starts and ends on a 4-byte
boundary, and as bytes otherwise: the same panoramas from the same images at another offset."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("cols,rows,image,refs", [(40, 32, (64, 48), 2), (33, 29, (36, 31), 1), (64, 50, (52, 44), 3)])
def test_word_and_byte_reads_agree(ss, native, cols, rows, image, refs):
    N = ss._native
    gen = torch.Generator(device=DEV).manual_seed(cols)
    rand = lambda *shape: torch.rand(*shape, generator=gen, device=DEV)  # noqa: E731
    frames, pano_cols, pano_rows = 2, 65, 37
    Q, P, pixels = pano_cols * pano_rows, cols * rows, image[0] * image[1] * 3
    lut = torch.stack([0.1 + rand(refs, Q) * (cols - 1.2), 0.1 + rand(refs, Q) * (rows - 1.2)], -1).contiguous()
    lut[:, :4] = torch.tensor([cols - 1.1, rows - 1.1], device=DEV)  # the last texels
    weights = rand(refs, Q)
    weights /= weights.sum(0)
    reproj, dists = 0.5 + 20 * rand(frames, refs, P), 0.5 + 20 * rand(frames, refs, P)
    data = torch.randint(0, 256, (frames * refs * pixels,), generator=gen, device=DEV).to(torch.uint8)
    held = torch.empty(data.numel() + 8, dtype=torch.uint8, device=DEV)
    k = N.ssg_intrinsics(cols / 3, rows / 3, cols / 2, rows / 2, -0.2, 0.6)
    intrinsics = N.intrinsics_array([k] * refs)
    translations = N.floats([0.05, -0.02, 0.01] * refs)
    outs = []
    for offset in (0, 1, 4, 7):
        images = held[offset: offset + data.numel()]
        images.copy_(data)
        d = torch.empty(frames, Q, device=DEV)
        rgb = torch.empty(frames, Q, 3, dtype=torch.uint8, device=DEV)
        N.call("ssg_merge_panorama_batch", lut.data_ptr(), weights.data_ptr(), reproj.data_ptr(), dists.data_ptr(),
               images.data_ptr(), image[1], image[0], translations, intrinsics, refs, cols, rows, pano_cols, pano_rows, frames,
               d.data_ptr(), rgb.data_ptr(), torch.cuda.current_stream().cuda_stream)
        outs.append((d, rgb))
    for d, rgb in outs[1:]:
        assert torch.equal(d, outs[0][0]) and torch.equal(rgb, outs[0][1])
    assert bool(outs[0][1].any())
