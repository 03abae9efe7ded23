"""Pose deltas of the differentiable sweep, on the CPU with the library's calls recorded."""
from __future__ import annotations

import ctypes
import importlib

import numpy as np
import pytest
import torch

from test_sweep_inputs import CAMERAS, COLS, IMAGES, ROWS, _maps, sweep_of  # noqa: F401


@pytest.fixture
def module(ss):
    return importlib.import_module("sphere-stereo_gb300.differentiable")


def _poses(monkeypatch, module, sweep):
    """The relative poses of each sweep launch of the calls that follow."""
    seen, record = [], module.N.call

    def call(name, *args):
        if name == "ssg_sweep_cost_references":
            seen.append(np.array(args[6][:], np.float32).reshape(args[4], CAMERAS, 12))
        record(name, *args)

    monkeypatch.setattr(module.N, "call", call)
    return seen


def test_one_row_per_camera(sweep_of, module, monkeypatch):
    """Fewer rows are refused (one row does not stand for all cameras), more are left unused."""
    sweep = sweep_of([0, 2])
    sweep.set_selection(_maps(2))
    seen = _poses(monkeypatch, module, sweep)
    deltas = torch.as_tensor(0.1 * np.random.default_rng(0).standard_normal((CAMERAS + 2, 6)))
    for rows in (0, 1, CAMERAS - 1):
        with pytest.raises(IndexError):
            sweep.forward(IMAGES, deltas[:rows])
    sweep.forward(IMAGES, deltas[:CAMERAS])
    sweep.forward(IMAGES, deltas)  # more rows than cameras
    np.testing.assert_array_equal(seen[0], seen[1])
    _, grad = sweep.backward(IMAGES, deltas, torch.zeros(2, ROWS, COLS))
    assert tuple(grad.shape) == (CAMERAS, 6)


def test_rotation_and_translation_gradients_stay_apart(sweep_of, module, monkeypatch):
    """A translation gradient that is not finite leaves the rotation's as it is."""
    sweep = sweep_of([0])
    sweep.set_selection(_maps(1))
    local = np.arange(1.0, 1 + 6 * CAMERAS).reshape(CAMERAS, 6)
    local[1, 4], local[2, 0] = np.inf, np.nan
    record = module.N.call

    def call(name, *args):
        if name == "ssg_sweep_backward_references":
            (ctypes.c_double * local.size).from_address(args[14])[:] = local.reshape(-1).tolist()
        else:
            record(name, *args)

    monkeypatch.setattr(module.N, "call", call)
    deltas = torch.as_tensor(0.2 * np.random.default_rng(1).standard_normal((CAMERAS, 6)))
    _, grad = sweep.backward(IMAGES, deltas, torch.zeros(1, ROWS, COLS))
    finite = torch.as_tensor(np.isfinite(local))
    assert bool(torch.isfinite(grad[0]).all()) and bool(torch.isfinite(grad[1, :3]).all())
    assert not bool(torch.isfinite(grad[1, 3:]).all()) and not bool(torch.isfinite(grad[2, :3]).all())
    assert bool(torch.isfinite(grad[2, 3:]).all()) and not bool(finite.all())
