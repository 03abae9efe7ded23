"""Hole filling (csrc/ssg_stitch.cu) at values on its two bounds: a hole is at least max_dist + 0.1, a usable
neighbour at most max_dist + 0.1f, which is larger.  Where a float32 lies in both (10.0 for a max_dist of 9.9)
a hole of that value is a usable neighbour, and where an average of values next to the bound is
rounded up to it, the filled pixel is a hole again: Jacobi steps on the CPU are the yardstick."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("iterations", [1, 2, 8, 9, 32, 57])
@pytest.mark.parametrize("max_dist", [9.9, 0.9, 100.0, 1.6, 3.3])
@pytest.mark.parametrize("cols,rows", [(64, 32), (131, 70), (200, 131)])
@pytest.mark.parametrize("near", [0.02, 0.6])
def test_values_on_the_bounds(ss, native, oracle_mod, cols, rows, max_dist, iterations, near):
    rng = np.random.default_rng(cols + iterations)
    bound = np.float32(max_dist + float(np.float32(0.1)))  # the largest usable value, or the float above it
    if float(bound) > max_dist + float(np.float32(0.1)):
        bound = np.nextafter(bound, np.float32(0))
    d = (rng.random((2, rows, cols)) * 0.5 * max_dist).astype(np.float32)
    at = rng.random(d.shape) < near
    steps = rng.integers(0, 3, int(at.sum()))
    d[at] = np.where(steps == 0, bound, np.nextafter(bound, np.float32(0)))
    d[:, rows // 5:, cols // 6: cols - cols // 7] = np.where(
        rng.random(d[:, rows // 5:, cols // 6: cols - cols // 7].shape) < 0.03, bound, np.float32(1e8))
    d[rng.random(d.shape) < 0.1] = 1e8
    tables = rng.integers(0, 256, (1, rows, cols, 2)).astype(np.uint8)
    N = ss._native
    stream = torch.cuda.current_stream().cuda_stream
    tab, out = torch.as_tensor(tables, device=DEV), torch.as_tensor(d, device=DEV)
    scratch = torch.empty_like(out)
    N.call("ssg_inpaint_batch", out.data_ptr(), tab.data_ptr(), scratch.data_ptr(), cols, rows, 2, 1, max_dist,
           iterations, stream)
    o = oracle_mod.Oracle("f32", exp_mode="device")
    for i in range(2):
        np.testing.assert_array_equal(out[i].cpu().numpy(), o.inpaint(d[i], tables[0], max_dist, iterations))
