"""Tiled hole filling (csrc/ssg_stitch.cu, fill_holes_kernel) against one Jacobi step per launch on the
CPU: tile and halo edges, maps smaller than a tile, rows that are not 16-byte aligned, chains as
long as the halos, and iteration counts around the 8 and 24 steps of a launch."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("iterations", [1, 8, 9, 16, 32, 33, 56, 57])
@pytest.mark.parametrize("cols,rows", [(64, 32), (65, 33), (5, 3), (200, 131), (131, 70), (96, 96)])
def test_tiles_equal_jacobi_steps(ss, native, oracle_mod, cols, rows, iterations):
    rng = np.random.default_rng(cols * rows + iterations)
    refs, frames = 2, 2
    d = (1 + rng.random((refs * frames, rows, cols)) * 5).astype(np.float32)
    d[:, rows // 5:, cols // 6: cols - cols // 7] = 1e8  # one wide hole: chains of every length
    d[rng.random(d.shape) < 0.1] = 1e8
    d[0, rows // 2, cols // 2] = np.nan
    # slot 0: directions as the table kernel writes them (all chains run left), slot 1: any bytes
    tables = rng.integers(0, 256, (refs, rows, cols, 2)).astype(np.uint8)
    tables[0, :, :, 0], tables[0, :, :, 1] = 160 + 4 * 1 + 0, 64 + 4 * 2 + 0
    N = ss._native
    stream = torch.cuda.current_stream().cuda_stream
    tab, out = torch.as_tensor(tables, device=DEV), torch.as_tensor(d, device=DEV)
    scratch = torch.empty_like(out)
    N.call("ssg_inpaint_batch", out.data_ptr(), tab.data_ptr(), scratch.data_ptr(), cols, rows, refs * frames, refs,
           100.0, iterations, stream)
    o = oracle_mod.Oracle("f32", exp_mode="device")
    for i in range(refs * frames):
        np.testing.assert_array_equal(out[i].cpu().numpy(), o.inpaint(d[i], tables[i % refs], 100.0, iterations))
