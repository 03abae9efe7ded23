"""DifferentiableSweep with the selection and gradient maps a caller may hand over, against the same values
set and given as whole tensors."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("refs", [[2, 3], [0, 1, 2, 3, 1]])
def test_replaced_maps_and_expanded_gradients(ss, native, synthetic, refs):
    cols, rows, n = 40, 33, 6
    rng = np.random.default_rng(3)
    cals = ss.parse_json_calib(synthetic.basalt_calibration(synthetic.square_rig(cols, rows)), [cols, rows], "cpu")
    masks = [torch.ones(1, rows, cols) for _ in cals]
    sweep, plain = (ss.DifferentiableSweep(cals, 0.4, 100.0, n, refs, masks, (cols, rows), 10.0, 6.0, DEV)
                    for _ in range(2))
    images = torch.as_tensor((rng.random((4, rows, cols, 3)) * 255).astype(np.float32), device=DEV)
    deltas = torch.zeros(4, 6, dtype=torch.float64)
    assert all(isinstance(p, torch.Tensor) and torch.equal(p, c.rt.double()) for p, c in zip(sweep.base_poses, cals))
    before = sweep.forward(images, deltas)
    maps = [t.clone() for t in plain.selected]
    maps[1] = (maps[1] + 1) % 4
    sweep.selected[1] = maps[1]
    plain.set_selection(maps)
    want = plain.forward(images, deltas)
    assert torch.equal(sweep.forward(images, deltas), want) and not torch.equal(want, before)
    one = torch.as_tensor(rng.standard_normal((rows, cols)).astype(np.float32), device=DEV)
    grad = one.expand(len(refs), rows, cols)
    got = sweep.backward(images, deltas, grad)
    for a, b in zip(got, plain.backward(images, deltas, grad.contiguous())):
        assert torch.equal(a, b)
