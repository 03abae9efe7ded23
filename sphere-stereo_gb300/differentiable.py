"""Differentiable sphere sweep for calibration refinement (no counterpart in the reference, which
selects distances with a hard argmin, python/depth_estimation.py:179-198).

``DifferentiableSweep(...)(images, pose_deltas)`` returns, for every reference camera, the
soft-argmin inverse distance

    q = sum_k softmax(-F_k / temperature) / d_k ,

F being the ISB-filtered sweep cost (python/depth_estimation.py:141-177, the fp32 kernels of the
library).  It is differentiable with respect to the matching images and to per-camera 6-DoF
pose deltas delta_c = (omega_c, v_c), the camera poses being T_c [Exp(omega_c), v_c].  The
backward pass recomputes the cost volume and the filter pyramid instead of storing them, runs
the filter transposed (its weights come from uint8 guides and get no gradient), and reduces the
pose gradient per camera in float64; the pose composition is float64 on the host.  The gradients
are bit-reproducible run to run: the transposed filter steps gather in a fixed order, the image
gradient is summed in 64-bit fixed point and the pose gradient by a fixed float64 tree.

Temperature: 2 cost units by default.  Costs are sums of three absolute 8-bit differences; near
the minimum, neighbouring candidates typically differ by a few units, so tau = 2 keeps the
weights concentrated on the best few candidates while staying smooth.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from . import _native as N
from .isb_filter import level_shapes
from .utils import _cpu32, camera_struct, relative_poses


_EYE3, _EYE4 = np.eye(3), np.eye(4)


def _skew(w) -> np.ndarray:
    x, y, z = w.tolist()
    return np.array([[0.0, -z, y], [z, 0.0, -x], [-y, x, 0.0]])


def _so3_exp(w) -> np.ndarray:
    th = math.sqrt(w.dot(w))
    k = _skew(w)
    if th < 1e-8:
        return _EYE3 + k + 0.5 * k @ k
    return _EYE3 + math.sin(th) / th * k + (1 - math.cos(th)) / th ** 2 * k @ k


def _so3_right_jacobian(w) -> np.ndarray:
    th = math.sqrt(w.dot(w))
    k = _skew(w)
    if th < 1e-6:
        return _EYE3 - 0.5 * k + k @ k / 6
    return _EYE3 - (1 - math.cos(th)) / th ** 2 * k + (th - math.sin(th)) / th ** 3 * k @ k


def _vector(w) -> np.ndarray:
    return torch.as_tensor(w).detach().to("cpu", torch.float64).numpy()


def skew(w) -> torch.Tensor:
    return torch.from_numpy(_skew(_vector(w)))


def so3_exp(w) -> torch.Tensor:
    return torch.from_numpy(_so3_exp(_vector(w)))


def so3_right_jacobian(w) -> torch.Tensor:
    return torch.from_numpy(_so3_right_jacobian(_vector(w)))


class _Poses:
    """The composed poses of one evaluation, in float64 on the host: T_c [Exp(omega_c), v_c] and, per
    reference, the relative poses of every camera."""

    def __init__(self, base: np.ndarray, refs: list[int], deltas: np.ndarray):
        self.deltas = deltas
        E = np.empty((len(deltas), 4, 4))
        E[:] = _EYE4
        for c, d in enumerate(deltas):
            E[c, :3, :3] = _so3_exp(d[:3])
        E[:, :3, 3] = deltas[:, 3:]
        T = base @ E
        inverse = np.linalg.inv(T)
        self.relative = [(inverse @ T[r])[:, :3].reshape(-1) for r in refs]  # camera_count x 12 each

    def to_deltas(self) -> np.ndarray:
        """[cameras, 2, 3, 3]: gradients of local right perturbations at T [Exp(omega), v] -> gradients with
        respect to omega and to v."""
        out = np.empty((len(self.deltas), 2, 3, 3))
        for c, d in enumerate(self.deltas):
            out[c, 0] = _so3_right_jacobian(d[:3]).T
            out[c, 1] = _so3_exp(d[:3])
        return out


class DifferentiableSweep:
    def __init__(self, calibrations, min_dist, max_dist, candidate_count, references_indices, masks,
                 matching_resolution, sigma_i, sigma_s, device, temperature: float = 2.0):
        """Same camera, range and filter arguments as RGBD_Estimator (python/depth_estimation.py:39-40)."""
        device = torch.device(device)
        if device.type != "cuda":
            raise ValueError(f"DifferentiableSweep runs on a CUDA device, got {device}; there is no CPU path")
        if device.index is None:
            device = torch.device("cuda", torch.cuda.current_device())
        N.library()
        if temperature <= 0:
            raise ValueError("temperature must be positive")
        self.device = device
        self.calibrations = calibrations
        self.C = len(calibrations)
        self.refs = list(references_indices)
        self.cols, self.rows = matching_resolution
        self.P = self.cols * self.rows
        self.N = candidate_count
        self.sigma_i, self.sigma_s = float(sigma_i), float(sigma_s)
        self.temperature = float(temperature)
        self.shapes = level_shapes(matching_resolution)
        self.L = len(self.shapes)
        if self.L < 2:
            raise ValueError("the matching resolution is too small for the filter pyramid")
        self.candidates = (1 / torch.linspace(1 / min_dist, 1 / max_dist, candidate_count)).tolist()
        self._cand = N.floats(self.candidates)
        self._cams = N.cameras_array([camera_struct(c) for c in calibrations])
        self.base_poses = [_cpu32(c.rt).double() for c in calibrations]
        dev = device
        # camera selection of the unperturbed rig (a discrete choice: no gradient)
        mask_stack = torch.stack([torch.as_tensor(m, dtype=torch.float32).reshape(self.rows, self.cols)
                                  for m in masks]).to(dev).contiguous()
        selected = torch.empty([len(self.refs), self.rows, self.cols], dtype=torch.int8, device=dev)
        for slot, r in enumerate(self.refs):
            N.call("ssg_select_camera", self.cols, self.rows, self.C, self._cams, r,
                   N.floats(relative_poses(calibrations, r)), mask_stack.data_ptr(), float(min_dist),
                   float(max_dist), selected[slot].data_ptr(), torch.cuda.current_stream(dev).cuda_stream)
        self._selected = selected
        self.selected = list(selected)
        self._allocate()

    # References are worked on together as long as their volumes (costs, and the two gradients of the
    # filter) fit these bytes (the launches of one reference do not fill the GPU) and the GPU's memory
    GROUP_BYTES = 4 << 30

    def _allocate(self) -> None:
        pyramid = sum(r * c for r, c in self.shapes)
        per_reference = 12 * self.N * pyramid + 24 * self.C * self.P
        self.group = N.largest_group(max(1, min(len(self.refs), 4, self.GROUP_BYTES // per_reference)), self._buffers)
        self._levels = {name: N.pointers([t.data_ptr() for t in getattr(self, name)])
                        for name in ("g_orig", "g_filt", "costs", "gf", "gc")}

    def _buffers(self, G: int) -> None:
        f32 = dict(dtype=torch.float32, device=self.device)
        u8 = dict(dtype=torch.uint8, device=self.device)
        lib = N.library()
        self.packed = self.g_orig = self.g_filt = self.costs = self.gf = self.gc = None
        self._tables = self._absmax = self._bwd_scratch = None
        self.packed = torch.empty(self.C, self.rows, self.cols, 4, **f32)
        self.g_orig = [torch.empty(G * r * c * 3, **u8) for r, c in self.shapes]
        self.g_filt = [self.g_orig[0]] + [torch.empty(G * r * c * 3, **u8) for r, c in self.shapes[1:]]
        self.costs, self.gf, self.gc = ([torch.empty(G * self.N * r * c, **f32) for r, c in self.shapes]
                                        for _ in range(3))
        self._tables = torch.empty(G * lib.ssg_isb_table_floats(self.rows, self.cols, self.L), **f32)
        self._absmax = torch.empty(G, dtype=torch.int32, device=self.device)
        scratch = lib.ssg_sweep_backward_references_scratch_bytes(self.cols, self.rows, self.C, G)
        self._bwd_scratch = torch.empty((scratch + 255) // 256 * 256, **u8)

    def set_selection(self, selected):
        """Use another run's camera-selection maps ([references][rows, cols])."""
        maps = [self._map(s, torch.int8) for s in selected]
        self._selected = torch.stack(maps) if maps else torch.empty(0, self.rows, self.cols, dtype=torch.int8)
        self.selected = list(self._selected)

    def _map(self, m, dtype: torch.dtype) -> torch.Tensor:
        return torch.as_tensor(m).reshape(self.rows, self.cols).to(self.device, dtype)

    def _selection(self, g0: int, count: int) -> torch.Tensor:
        """The maps of ``self.selected`` of ``count`` references from slot g0 on, one after the other as the
        kernels read them: ``self._selected``'s own, or a copy where entries were replaced."""
        maps = [self.selected[g0 + i] for i in range(count)]  # IndexError: a reference without a map
        own = self._selected[g0:g0 + count]
        first = own.data_ptr()
        if len(own) == count and all(m.data_ptr() == first + i * self.P for i, m in enumerate(maps)):
            return own
        return torch.stack([self._map(m, torch.int8) for m in maps])

    def _gradient_maps(self, grad_q) -> torch.Tensor:
        """The incoming gradient's maps, one after the other as the kernels read them."""
        shape = (len(self.refs), self.rows, self.cols)
        if (isinstance(grad_q, torch.Tensor) and tuple(grad_q.shape) == shape and grad_q.dtype == torch.float32
                and grad_q.device == self.device and grad_q.is_contiguous()):
            return grad_q
        maps = [grad_q[slot] for slot in range(len(self.refs))]  # IndexError: a reference without a map
        return torch.stack([self._map(m, torch.float32) for m in maps])

    # ------------------------------------------------------------------------------------
    def _poses(self, deltas: torch.Tensor) -> _Poses:
        """deltas: a row per camera (rows after the last camera's are not read)."""
        d = deltas.detach().to("cpu", torch.float64).numpy()
        if len(d) < self.C:
            raise IndexError(f"pose_deltas has {len(d)} rows, one for each of the {self.C} cameras is required")
        base = torch.stack(self.base_poses[:self.C]).numpy()
        return _Poses(base, self.refs, d[:self.C].copy())

    def _groups(self):
        """(first slot, references, how many) of each group of references."""
        for g0 in range(0, len(self.refs), self.group):
            refs = self.refs[g0:g0 + self.group]
            yield g0, refs, len(refs)

    def _pyramid(self, g0: int, refs: list[int], images: torch.Tensor, poses: _Poses, stream):
        """Sweep + filter of a group of references (levels 1..L-1 filtered; level 0 left raw).  Returns
        what the sweep was called with: the references, their relative poses and their selection maps."""
        count = len(refs)
        selection = self._selection(g0, count)
        refs_c, rel = N.ints(refs), N.floats(np.concatenate(poses.relative[g0:g0 + count]).tolist())
        N.call("ssg_pack_images", N.pointers([images[c].data_ptr() for c in range(self.C)]), self.C, self.P, refs_c,
               count, self.packed.data_ptr(), self.g_orig[0].data_ptr(), stream)
        N.call("ssg_sweep_cost_references", self.cols, self.rows, self.C, self._cams, count, refs_c, rel,
               self.packed.data_ptr(), selection.data_ptr(), self._cand, self.N, self.costs[0].data_ptr(), stream)
        N.call("ssg_isb_filter", self._levels["g_orig"], self._levels["g_filt"], self._levels["costs"], self.L,
               self.rows, self.cols, self.N, count, self.sigma_i, self.sigma_s, stream)
        return refs_c, rel, selection

    def _last_level(self, count: int):
        """The arguments of the soft-argmin's last filter level."""
        return (self.g_filt[1].data_ptr(), self.costs[1].data_ptr(), self.g_orig[0].data_ptr(),
                self.costs[0].data_ptr(), self.rows, self.cols, self.N, count, self.sigma_i, self.sigma_s, self._cand,
                self.temperature)

    def forward(self, images: torch.Tensor, deltas: torch.Tensor, poses: _Poses | None = None) -> torch.Tensor:
        """poses: the composed poses of ``deltas``, where the caller has them."""
        N.require(images, "images", torch.float32, (self.C, self.rows, self.cols, 3), self.device)
        stream = N.stream_of(images)
        poses = self._poses(deltas) if poses is None else poses
        q = torch.empty(len(self.refs), self.rows, self.cols, device=self.device)
        for g0, refs, count in self._groups():
            self._pyramid(g0, refs, images, poses, stream)
            N.call("ssg_soft_argmin", *self._last_level(count), q[g0].data_ptr(), stream)
        return q

    def backward(self, images: torch.Tensor, deltas: torch.Tensor, grad_q: torch.Tensor, poses: _Poses | None = None):
        stream = N.stream_of(images)
        poses = self._poses(deltas) if poses is None else poses
        grad_q = self._gradient_maps(grad_q)
        grad_images = torch.zeros_like(images)
        grad_local = torch.zeros(self.C, 6, dtype=torch.float64, device=self.device)
        targets = N.pointers([grad_images[c].data_ptr() for c in range(self.C)])
        for g0, refs, count in self._groups():
            refs_c, rel, selection = self._pyramid(g0, refs, images, poses, stream)
            # dL/dF of the filtered level 0, then the filter transposed, then the sweep
            N.call("ssg_soft_argmin_backward", *self._last_level(count), grad_q[g0].data_ptr(), self.gf[0].data_ptr(),
                   stream)
            N.call("ssg_isb_filter_transpose", self._levels["g_orig"], self._levels["g_filt"], self.L, self.rows,
                   self.cols, self.N, count, self.sigma_i, self.sigma_s, self._levels["gf"], self._levels["gc"],
                   self._tables.data_ptr(), self._absmax.data_ptr(), stream)
            N.call("ssg_sweep_backward_references", self.cols, self.rows, self.C, self._cams, count, refs_c, rel,
                   self.packed.data_ptr(), targets, selection.data_ptr(), self._cand, self.N,
                   self.gc[0].data_ptr(), self._absmax.data_ptr(), grad_local.data_ptr(), self._bwd_scratch.data_ptr(),
                   stream)
        to_deltas = torch.from_numpy(poses.to_deltas()).to(self.device, non_blocking=True)
        out = (to_deltas * grad_local.view(self.C, 2, 1, 3)).sum(-1).view(self.C, 6)
        return grad_images, out.to(deltas.device)

    def __call__(self, images: torch.Tensor, pose_deltas: torch.Tensor | None = None) -> torch.Tensor:
        """images [cameras, rows, cols, 3] float32; pose_deltas [cameras, 6] float64 (zeros if
        None).  Returns the soft-argmin inverse distance [references, rows, cols]."""
        if pose_deltas is None:
            pose_deltas = torch.zeros(self.C, 6, dtype=torch.float64, device=self.device)
        return _SoftSweep.apply(images, pose_deltas, self)


class _SoftSweep(torch.autograd.Function):
    @staticmethod
    def forward(ctx, images, pose_deltas, sweep):
        images_c = images.detach().contiguous()
        ctx.save_for_backward(images_c, pose_deltas.detach())
        ctx.sweep = sweep
        ctx.poses = sweep._poses(pose_deltas)  # host values: the backward need not read the deltas again
        return sweep.forward(images_c, pose_deltas, ctx.poses)

    @staticmethod
    def backward(ctx, grad_q):
        images, deltas = ctx.saved_tensors
        gi, gd = ctx.sweep.backward(images, deltas, grad_q.contiguous(), ctx.poses)
        return gi, gd, None
