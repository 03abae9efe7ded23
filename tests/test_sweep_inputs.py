"""What DifferentiableSweep hands to its kernels, on the CPU with the library's calls recorded: the camera
selection and gradient maps of every reference of a launch lie one after the other in memory that
holds them all, whatever the caller gave; too few of them are refused."""
from __future__ import annotations

import ctypes
import importlib

import numpy as np
import pytest
import torch

ROWS, COLS, N, CAMERAS = 16, 24, 3, 3
P = ROWS * COLS


@pytest.fixture
def sweep_of(ss, monkeypatch):
    """sweep_of(references, group): a sweep on the CPU whose library calls are recorded, with what its
    kernels would read at the recorded addresses."""
    module = importlib.import_module("sphere-stereo_gb300.differentiable")
    native = module.N
    calls = []

    def call(name, *args):
        if name == "ssg_sweep_cost_references":
            calls.append(("selection", args[4], _bytes(args[8], args[4] * P, np.int8)))
        elif name == "ssg_sweep_backward_references":
            calls.append(("selection", args[4], _bytes(args[9], args[4] * P, np.int8)))
        elif name == "ssg_soft_argmin_backward":
            calls.append(("gradient", args[7], _bytes(args[12], args[7] * P, np.float32)))

    monkeypatch.setattr(native, "call", call)
    monkeypatch.setattr(native, "stream_of", lambda t: 0)
    monkeypatch.setattr(native, "require", lambda *a, **k: None)

    def build(refs, group=4):
        s = module.DifferentiableSweep.__new__(module.DifferentiableSweep)
        s.device, s.C, s.refs, s.rows, s.cols, s.P, s.N = torch.device("cpu"), CAMERAS, list(refs), ROWS, COLS, P, N
        s.shapes, s.L, s.group = [(ROWS, COLS), (ROWS // 2, COLS // 2)], 2, group
        s.sigma_i, s.sigma_s, s.temperature, s._cams, s._cand = 10.0, 6.0, 2.0, None, None
        one = torch.zeros(1)
        s.packed = s._tables = s._absmax = s._bwd_scratch = one
        s.g_orig = s.g_filt = s.costs = s.gf = s.gc = [one, one]
        s._levels = dict.fromkeys(("g_orig", "g_filt", "costs", "gf", "gc"))
        s.base_poses = [torch.eye(4, dtype=torch.float64) for _ in range(CAMERAS)]
        s.calls = calls
        return s

    return build


def _bytes(address, count, dtype):
    size = count * np.dtype(dtype).itemsize
    return np.frombuffer((ctypes.c_uint8 * size).from_address(address), dtype).copy().reshape(-1, ROWS, COLS)


def _maps(count, seed=0):
    return [torch.as_tensor(m) for m in np.random.default_rng(seed).integers(-1, CAMERAS, (count, ROWS, COLS)).astype(np.int8)]


IMAGES = torch.zeros(CAMERAS, ROWS, COLS, 3)
ZERO = torch.zeros(CAMERAS, 6, dtype=torch.float64)


def _seen(sweep, kind):
    return np.concatenate([a for k, _, a in sweep.calls if k == kind])


@pytest.mark.parametrize("refs,group", [([0, 1], 4), ([2, 0, 1, 0, 2], 4), ([0, 1, 2], 1)])
def test_every_reference_needs_a_selection_map(sweep_of, refs, group):
    sweep = sweep_of(refs, group)
    sweep.set_selection(_maps(len(refs) - 1))
    with pytest.raises(IndexError):
        sweep.forward(IMAGES, ZERO)
    with pytest.raises(IndexError):
        sweep.backward(IMAGES, ZERO, torch.zeros(len(refs), ROWS, COLS))
    sweep.calls.clear()
    maps = _maps(len(refs) + 1)  # one more than needed is left unused
    sweep.set_selection(maps)
    sweep.forward(IMAGES, ZERO)
    np.testing.assert_array_equal(_seen(sweep, "selection"), torch.stack(maps[:len(refs)]).numpy())


@pytest.mark.parametrize("group", [4, 2, 1])
def test_replaced_selection_entries_are_used(sweep_of, group):
    sweep = sweep_of([0, 1, 2], group)
    maps = _maps(3)
    sweep.set_selection(maps)
    other = torch.stack(_maps(2, 1))
    sweep.selected[1] = other[0]
    sweep.selected[2][3] = 1  # in place
    want = torch.stack([maps[0], other[0], maps[2]])
    want[2, 3] = 1
    sweep.forward(IMAGES, ZERO)
    sweep.backward(IMAGES, ZERO, torch.zeros(3, ROWS, COLS))
    np.testing.assert_array_equal(_seen(sweep, "selection"), torch.cat([want, *[w for g in range(0, 3, group) for w in
                                                                                2 * [want[g:g + group]]]]).numpy())
    sweep.selected[0] = torch.zeros(P - 1, dtype=torch.int8)
    with pytest.raises(RuntimeError):
        sweep.forward(IMAGES, ZERO)


@pytest.mark.parametrize("group", [4, 1])
def test_gradient_maps(sweep_of, group):
    sweep = sweep_of([0, 1], group)
    sweep.set_selection(_maps(2))
    room = torch.arange(6 * P, dtype=torch.float32)
    grad = room[:P].view(ROWS, COLS)
    with pytest.raises(IndexError):
        sweep.backward(IMAGES, ZERO, grad[None])
    strided = room.view(2, ROWS, COLS, 3)[..., 1]
    for given, want in ((grad.expand(2, ROWS, COLS), [grad, grad]),  # the sum of both maps, say
                        (room[:3 * P].view(3, ROWS, COLS), list(room[:2 * P].view(2, ROWS, COLS))),
                        ([grad, grad + 1], [grad, grad + 1]), (strided, list(strided))):
        sweep.calls.clear()
        sweep.backward(IMAGES, ZERO, given)
        np.testing.assert_array_equal(_seen(sweep, "gradient"), torch.stack(want).numpy())
