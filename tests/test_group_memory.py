"""References are worked on in smaller groups where the GPU's memory does not hold the buffers of a larger
one: the allocations are made to fail here, on the CPU, above a number of bytes."""
from __future__ import annotations

import importlib
import types
import weakref

import pytest
import torch


@pytest.fixture
def limit(monkeypatch):
    """limit(bytes): torch.empty and torch.zeros fail once as many bytes are held."""
    held = types.SimpleNamespace(bytes=0, most=float("inf"))

    def wrap(make):
        def allocate(*size, dtype=torch.float32, **kwargs):
            n = torch.Size(size[0] if isinstance(size[0], (tuple, list)) else size).numel() * dtype.itemsize
            if held.bytes + n > held.most:
                raise torch.cuda.OutOfMemoryError("no room")
            t = make(*size, dtype=dtype, **kwargs)
            held.bytes += n
            weakref.finalize(t, lambda: setattr(held, "bytes", held.bytes - n))
            return t
        return allocate

    monkeypatch.setattr(torch, "empty", wrap(torch.empty))
    monkeypatch.setattr(torch, "zeros", wrap(torch.zeros))

    def set_limit(most):
        held.most = held.bytes + most

    return set_limit


SHAPES = [(32, 40), (16, 20), (8, 10)]
PYRAMID = sum(r * c for r, c in SHAPES)


def _fp32(module, references=4):
    return module._Fp32Buffers(5, references, 8, SHAPES, "cpu")


@pytest.mark.parametrize("fits,group", [(4, 4), (3, 2), (2, 2), (1, 1)])
def test_fp32_groups(ss, limit, fits, group):
    module = importlib.import_module("sphere-stereo_gb300.depth_estimation")
    one = 4 * 8 * PYRAMID + 3 * PYRAMID + 7 * (PYRAMID - 32 * 40)
    packed = 16 * 5 * 32 * 40
    limit(packed + fits * one)
    b = _fp32(module)
    assert b.group == group and all(c.shape[0] == group for c in b.costs)
    assert b.levels(group)[0] == 0 and b.levels(1)[0] == group - 1


def test_no_room_for_one_reference(ss, limit):
    module = importlib.import_module("sphere-stereo_gb300.depth_estimation")
    limit(16 * 5 * 32 * 40 + 1000)
    with pytest.raises(torch.cuda.OutOfMemoryError):
        _fp32(module)


@pytest.mark.parametrize("group", [4, 2, 1])
def test_sweep_groups(ss, native, limit, group):
    module = importlib.import_module("sphere-stereo_gb300.differentiable")
    s = module.DifferentiableSweep.__new__(module.DifferentiableSweep)
    s.device, s.C, s.refs, (s.rows, s.cols), s.N = torch.device("cpu"), 3, [0, 1, 2, 0, 1], SHAPES[0], 8
    s.P, s.shapes, s.L = 32 * 40, SHAPES, 3

    def size(references):
        lib = module.N.library()
        scratch = lib.ssg_sweep_backward_references_scratch_bytes(s.cols, s.rows, s.C, references)
        return (16 * s.C * s.P + references * (12 * s.N * PYRAMID + 3 * (2 * PYRAMID - s.P) + 4
                                               + 4 * lib.ssg_isb_table_floats(s.rows, s.cols, s.L))
                + (scratch + 255) // 256 * 256)

    limit(size(group))
    s._allocate()
    assert s.group == group and s.costs[0].numel() == group * s.N * s.P
    del s.costs, s.gf, s.gc, s.packed, s.g_orig, s.g_filt, s._tables, s._bwd_scratch, s._absmax
    limit(size(1) - 1)
    with pytest.raises(torch.cuda.OutOfMemoryError):
        s._allocate()
