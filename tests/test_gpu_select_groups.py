"""The selecting level of the chunked filter, which takes four candidates at a time, against the
filtered volume and a selection candidate by candidate: the same index and distance bit for bit, at
candidate counts around the groups of 4 and 8, with ties, infinite and NaN costs, and whatever lies
in the cells beyond the last candidate."""
from __future__ import annotations

import importlib

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 7, 8, 9, 12, 31, 32, 33, 36, 70])
@pytest.mark.parametrize("storage", ["f16", "unorm16", "f32"])
def test_equals_selection_of_the_filtered_volume(ss, native, n, storage):
    N, tune = ss._native, importlib.import_module("sphere-stereo_gb300.autotune")
    f32 = 2
    kind = {"f16": 0, "unorm16": 1, "f32": f32}[storage]
    rows, cols, inst = 21, 291, 2
    crows, ccols, chunks = (rows + 1) // 2, (cols + 1) // 2, (n + 7) // 8
    gen = torch.Generator(device=DEV).manual_seed(n)
    rand = lambda *shape: torch.rand(*shape, generator=gen, device=DEV)  # noqa: E731
    fine = rand(inst, chunks, rows * cols, 8) * 400
    coarse = rand(inst, chunks, crows * ccols, 8) * 400
    fine[:, :, : 4 * cols] = 37.5  # every candidate alike
    coarse[:, :, : 4 * ccols] = 12.25
    fine[0, :, 9 * cols: 11 * cols] = fine[0, :, 9 * cols: 11 * cols].div(100).floor()  # ties of some
    coarse[0, :, 4 * ccols: 7 * ccols] = 3.0
    if storage != "unorm16":
        fine[1, :, 12 * cols: 12 * cols + 90, 1::2] = float("inf")
        fine[1, :, 13 * cols: 13 * cols + 90] = float("inf")
        fine[1, :, 14 * cols: 14 * cols + 90, ::3] = float("nan")
        fine[1, :, 15 * cols: 15 * cols + 90] = float("nan")
    if n % 8:
        fine[:, -1, :, n % 8:] = 0  # below every cost
        coarse[:, -1, :, n % 8:] = 0
    if storage == "f16":
        stored = fine.half()
        fine = stored.float()
    elif storage == "unorm16":
        codes = (fine * (65535 / 500)).round().to(torch.int32)
        stored = codes.to(torch.int16)  # the low 16 bits
        fine = codes.float() * torch.tensor(500 / 65535, dtype=torch.float32, device=DEV)
    else:
        stored = fine.clone()
    guides = torch.randint(16, 236, (inst, rows * cols, 4), generator=gen, device=DEV).to(torch.uint8)
    guide_in = torch.randint(16, 236, (inst, crows * ccols, 4), generator=gen, device=DEV).to(torch.uint8)
    guides[..., 3] = guide_in[..., 3] = 0
    cand = N.floats([100.0 / (1 + 2.0 * i) for i in range(n)])
    weights, stream = (0.9, 0.1, 1 / 200.0), torch.cuda.current_stream().cuda_stream
    size = (crows, ccols), (rows, cols)

    filtered, scratch = fine.clone(), guides.clone()
    N.call("ssg_isb_upsample_batch", guide_in.data_ptr(), coarse.data_ptr(), *size[0], scratch.data_ptr(),
           filtered.data_ptr(), *size[1], n, inst, f32, *weights, stream)
    want_d, want_i = (torch.empty(inst, rows * cols, dtype=t, device=DEV) for t in (torch.float32, torch.int32))
    N.call("ssg_select_distance_batch", filtered.data_ptr(), n, rows * cols, inst, f32, cand,
           want_d.data_ptr(), want_i.data_ptr(), stream)
    knobs = ("select_whole", "isb_select_blocks")
    before = {k: tune.get(k) for k in knobs}
    try:
        for values in ((1, 3), (1, 2), (0, 3)):
            for k, v in zip(knobs, values):
                tune.set_knob(k, v)
            d, copy = torch.full_like(want_d, -1), torch.full_like(want_d, -1)
            i = torch.full_like(want_i, -1)
            N.call("ssg_isb_upsample_select_batch", guide_in.data_ptr(), coarse.data_ptr(), *size[0],
                   guides.data_ptr(), stored.data_ptr(), *size[1], n, inst, kind, *weights, cand, d.data_ptr(),
                   i.data_ptr(), copy.data_ptr(), stream)
            assert torch.equal(i, want_i)
            torch.testing.assert_close(d, want_d, rtol=0, atol=0, equal_nan=True)
            torch.testing.assert_close(copy, want_d, rtol=0, atol=0, equal_nan=True)
    finally:
        for k, v in before.items():
            tune.set_knob(k, v)
