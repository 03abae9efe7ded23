"""ISB steps on planar volumes of several candidates (csrc/ssg_isb_planar.cuh): every way the candidates
are shared out, at the edges of pixel groups, rows and ranges, equals the oracle bit for bit; and
the fused selection equals the two separate steps on costs that are not finite."""
from __future__ import annotations

import importlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _case(cols, rows, n, seed):
    rng = np.random.default_rng(seed)
    guide = (rng.integers(0, 6, (rows, cols, 3)) * 11 + 40).astype(np.uint8)
    return guide, (rng.random((n, rows, cols)) * 120).astype(np.float32)


# candidate counts around the ranges (fewer than 8, one more than a multiple, a short last range),
# widths and heights around the 32-pixel groups, odd ones on the unpaired path; the last two reach
# the fewer ranges of large levels
@pytest.mark.parametrize("cols,rows,n", [(64, 64, 2), (66, 17, 7), (67, 65, 8), (129, 66, 9), (33, 130, 43),
                                         (130, 131, 64), (641, 331, 5), (642, 640, 33)])
def test_filter_equals_oracle(ss, native, oracle_mod, cols, rows, n):
    o = oracle_mod.Oracle("f32", exp_mode="device")
    guide, cost = _case(cols, rows, n, cols * rows + n)
    c, g = ss.ISB_Filter(n, (cols, rows), DEV).apply(torch.as_tensor(guide, device=DEV),
                                                     torch.as_tensor(cost, device=DEV), 10.0, 12.5)
    want_c, want_g = o.isb_apply(guide, cost, 10.0, 12.5)
    np.testing.assert_array_equal(g.cpu().numpy(), want_g)
    np.testing.assert_array_equal(c.cpu().numpy(), want_c)


def test_levels_that_are_not_8_byte_aligned(ss, native):
    guide, cost = _case(96, 70, 12, 5)
    f = ss.ISB_Filter(12, (96, 70), DEV)
    want, _ = f.apply(torch.as_tensor(guide, device=DEV), torch.as_tensor(cost, device=DEV), 8.0, 6.0)
    room = torch.empty(cost.size + 1, device=DEV)
    shifted = room[1:].view(cost.shape)
    shifted.copy_(torch.as_tensor(cost))
    assert shifted.data_ptr() % 8 == 4
    got, _ = f.apply(torch.as_tensor(guide, device=DEV), shifted, 8.0, 6.0)
    assert torch.equal(got, want)


@pytest.mark.parametrize("n", [2, 9, 32])
def test_fused_selection_of_costs_that_are_not_finite(ss, native, n):
    cols, rows = 68, 50
    rng = np.random.default_rng(n)
    guide, fine = _case(cols, rows, n, n)
    cguide, coarse = _case(34, 25, n, n + 1)
    for volume in (fine, coarse):
        volume[rng.random(volume.shape) < 0.05] = np.inf
        volume[rng.random(volume.shape) < 0.02] = np.nan
        volume[rng.random(volume.shape) < 0.02] = -np.inf
    fine[:, 0], coarse[:, 0] = np.inf, np.inf
    fine[:, 7] = np.nan
    N = ss._native
    cand = N.floats(ss.distance_candidates(0.55, 100.0, n).tolist())
    stream = torch.cuda.current_stream().cuda_stream
    out = []
    for fused in (True, False):
        g, c = torch.as_tensor(guide, device=DEV).clone(), torch.as_tensor(fine, device=DEV).clone()
        gc, cc = torch.as_tensor(cguide, device=DEV), torch.as_tensor(coarse, device=DEV)
        d = torch.empty(rows, cols, device=DEV)
        i = torch.empty(rows, cols, dtype=torch.int32, device=DEV)
        head = (gc.data_ptr(), cc.data_ptr(), 25, 34, g.data_ptr(), c.data_ptr(), rows, cols, n, 0.3, 0.7, 0.005)
        if fused:
            N.call("ssg_isb_upsample_select", *head, cand, d.data_ptr(), i.data_ptr(), stream)
        else:
            N.call("ssg_isb_upsample", *head, stream)
            N.call("ssg_select_distance", c.data_ptr(), n, rows * cols, cand, d.data_ptr(), i.data_ptr(), stream)
        out.append((d.cpu().numpy(), i.cpu().numpy(), g.cpu().numpy()))
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("cols,rows,n,instances", [(65, 33, 3, 2), (64, 64, 32, 1), (131, 70, 9, 3), (40, 300, 5, 2),
                                                   (258, 257, 2, 1), (96, 80, 1, 2)])
def test_filter_of_several_volumes_equals_a_launch_per_step(ss, native, cols, rows, n, instances):
    """ssg_isb_filter, its small levels in one launch, with the filtered guides apart and in place, and
    ssg_isb_filter_select, against ssg_isb_downsample / _upsample / _upsample_select per volume."""
    isb = importlib.import_module("sphere-stereo_gb300.isb_filter")
    N = ss._native
    stream = torch.cuda.current_stream().cuda_stream
    shapes, si, sg = isb.level_shapes((cols, rows)), 9.0, 7.5
    L = len(shapes)
    weights, var = isb.level_weights(L, sg), 1 / (2 * si * si)
    cases = [_case(cols, rows, n, 31 * i + n) for i in range(instances)]
    g0 = torch.as_tensor(np.stack([g for g, _ in cases]), device=DEV)
    c0 = torch.as_tensor(np.stack([c for _, c in cases]), device=DEV)

    def levels(level0, channels, dtype):
        return [level0.clone()] + [torch.zeros(instances, *channels(r, c), dtype=dtype, device=DEV) for r, c in shapes[1:]]

    def guides():
        return levels(g0, lambda r, c: (r, c, 3), torch.uint8)

    def costs():
        return levels(c0, lambda r, c: (n, r, c), torch.float32)

    def ptrs(ts):
        return N.pointers([t.data_ptr() for t in ts])

    want_orig, want, want_c = guides(), guides(), costs()
    cand = N.floats(ss.distance_candidates(0.55, 100.0, n).tolist())
    want_d = torch.empty(instances, rows, cols, device=DEV)
    want_i = torch.empty(instances, rows, cols, dtype=torch.int32, device=DEV)
    for i in range(instances):
        for s in range(1, L):
            N.call("ssg_isb_downsample", want_orig[s - 1][i].data_ptr(), want_c[s - 1][i].data_ptr(), *shapes[s - 1],
                   want_orig[s][i].data_ptr(), want_c[s][i].data_ptr(), *shapes[s], n, var, stream)
            want[s][i].copy_(want_orig[s][i])
        for s in range(L - 2, 0, -1):
            N.call("ssg_isb_upsample", want[s + 1][i].data_ptr(), want_c[s + 1][i].data_ptr(), *shapes[s + 1],
                   want[s][i].data_ptr(), want_c[s][i].data_ptr(), *shapes[s], n, *weights[s], var, stream)
        fine = g0[i].clone()
        N.call("ssg_isb_upsample_select", want[1][i].data_ptr(), want_c[1][i].data_ptr(), *shapes[1], fine.data_ptr(),
               want_c[0][i].data_ptr(), rows, cols, n, *weights[0], var, cand, want_d[i].data_ptr(),
               want_i[i].data_ptr(), stream)
    g, f, c = guides(), [torch.zeros_like(t) for t in guides()], costs()
    N.call("ssg_isb_filter", ptrs(g), ptrs(f), ptrs(c), L, rows, cols, n, instances, si, sg, stream)
    for s in range(L):
        assert torch.equal(g[s], want_orig[s]) and torch.equal(c[s], want_c[s])
        assert s == 0 or torch.equal(f[s], want[s])
    g, c = guides(), costs()
    d, copy, i = torch.empty_like(want_d), torch.empty_like(want_d), torch.empty_like(want_i)
    N.call("ssg_isb_filter_select", ptrs(g), ptrs(c), L, rows, cols, n, instances, si, sg, cand, d.data_ptr(),
           i.data_ptr(), copy.data_ptr(), stream)
    assert torch.equal(d, want_d) and torch.equal(copy, want_d) and torch.equal(i, want_i)
    assert torch.equal(g[0], g0) and all(torch.equal(g[s], want[s]) for s in range(1, L))
