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


@pytest.mark.parametrize("w", [[0.0, 0.0, 0.0], [3e-9, -1e-9, 2e-9], [4e-7, 1e-7, -2e-7], [0.3, -1.1, 0.4], [2.0, 1.0, -2.0]])
def test_rotation_functions_return_tensors(module, w):
    """Exp(w), the skew matrix and the right Jacobian as float64 tensors; the Jacobian is the derivative of
    Exp(-w) Exp(w + d) by d."""
    t = torch.tensor(w, dtype=torch.float64)
    for given in (t, t.float()):
        k, r, j = module.skew(given), module.so3_exp(given), module.so3_right_jacobian(given)
        for m in (k, r, j):
            assert isinstance(m, torch.Tensor) and m.dtype == torch.float64 and tuple(m.shape) == (3, 3)
        torch.testing.assert_close(k, torch.linalg.cross(given.double().expand(3, 3), torch.eye(3, dtype=torch.float64)).T,
                                   rtol=0, atol=0)
        # the series below 1e-8 stops at third order
        torch.testing.assert_close(r, torch.linalg.matrix_exp(k), rtol=0, atol=1e-14)
    h = 1e-6
    for a in range(3):
        d = torch.zeros(3, dtype=torch.float64)
        d[a] = h
        col = module.so3_exp(-t) @ (module.so3_exp(t + d) - module.so3_exp(t - d)) / (2 * h)
        torch.testing.assert_close(module.so3_right_jacobian(t)[:, a], torch.stack([col[2, 1], col[0, 2], col[1, 0]]),
                                   rtol=0, atol=1e-7)


def test_replaced_base_poses_are_used(sweep_of, module, monkeypatch):
    """base_poses is a list of float64 4 x 4 tensors, read at every call."""
    sweep = sweep_of([0])
    sweep.set_selection(_maps(1))
    seen = _poses(monkeypatch, module, sweep)
    zero = torch.zeros(CAMERAS, 6, dtype=torch.float64)
    moved = torch.eye(4, dtype=torch.float64)
    moved[:3, 3] = torch.tensor([0.5, -2.0, 4.0], dtype=torch.float64)
    sweep.base_poses[1] = moved
    sweep.base_poses[2][0, 3] = 1.0
    sweep.forward(IMAGES, zero)
    want = np.tile(np.eye(4)[:3].reshape(-1), (CAMERAS, 1))
    want[1, [3, 7, 11]] = -0.5, 2.0, -4.0  # inverse(T_c) T_0
    want[2, 3] = -1.0
    np.testing.assert_array_equal(seen[0][0], want.astype(np.float32))

