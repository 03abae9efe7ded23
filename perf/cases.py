"""Workloads that stand for what a user of sphere_stereo_gb300 runs, each through the package's
public entry points, with inputs made from a seed on the GPU.

``listed()`` names the workloads, ``draw(rng)`` gives another one of the same ranges.  For a case,
``prepare(case, seed)`` builds what a program has in hand before the call (the rig's estimator,
filter or stitcher, and the input images, maps or volumes), ``run(state)`` is one pass, ``work``
the bytes and operations a pass cannot do without, and ``exact`` the outputs in 64 bits where they
are computed numbers that have such a value.

The scenes are ray-cast on the GPU with torch: a 6 x 5 x 3 m room with spheres of radius
0.2-1.0 m and value-noise textures, seen by outward double-sphere rigs, as 8-bit images.
"""
from __future__ import annotations

import importlib
import math

import torch

DEV = "cuda:0"


def _ss(module: str = ""):
    return importlib.import_module("sphere-stereo_gb300" + module)


# ---------------------------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------------------------

def listed():
    frame = dict(op="frame", cameras=4, sigma_i=10.0)
    batch = dict(op="batch", cols=1024, rows=1024, image_cols=1216, image_rows=1216, pano_cols=2048, pano_rows=1024,
                 cameras=4, sigma_i=10.0, sigma_s=25.0, storage="fp16")
    return [
        # the drop-in call of the reference's main loop, one frame per call: the small quick-look
        # configuration (latency), the prototype configuration, and rectangular images of odd
        # sizes with all four cameras as references
        dict(frame, name="frame_256_n32", cols=256, rows=256, image_cols=512, image_rows=512, pano_cols=1024,
             pano_rows=512, candidates=32, references=2, sigma_s=6.25),
        dict(frame, name="frame_1024_n32", cols=1024, rows=1024, image_cols=1216, image_rows=1216, pano_cols=2048,
             pano_rows=1024, candidates=32, references=2, sigma_s=25.0),
        dict(frame, name="frame_637x479_n43", cols=637, rows=479, image_cols=801, image_rows=603, pano_cols=1275,
             pano_rows=637, candidates=43, references=4, sigma_s=12.5),
        # offline processing of a recording in batches of 8 frames on the 16-bit path: images
        # already resized to float32, and the decoded 8-bit images as they come from the decoder
        dict(batch, name="batch8_1024_n32_f32", frames=8, candidates=32, references=2, inputs="f32"),
        dict(batch, name="batch8_1024_n32_decoded", frames=8, candidates=32, references=2, inputs="decoded"),
        # the dense configuration of a long stream: twice the candidates, every camera a reference
        dict(batch, name="stream8_1024_n64_r4", frames=8, candidates=64, references=4, inputs="decoded"),
        # a server's mixed load: one frame of nine rigs of different sizes, candidate counts and
        # camera counts in one launch sequence
        dict(op="uneven", name="uneven_9_rigs", jobs=9, rig_seed=5000, smallest=512, largest=1024),
        # the cost filter on its own (a program with its own matching cost): a full volume
        dict(op="isb", name="isb_1024_n32", cols=1024, rows=1024, candidates=32, sigma_i=10.0, sigma_s=25.0),
        # the stitcher on its own: distance maps that come from elsewhere (a network, a sensor)
        dict(op="stitch", name="stitch_2048x1024", cols=1024, rows=1024, image_cols=1216, image_rows=1216,
             pano_cols=2048, pano_rows=1024, references=2),
        # a step of extrinsics refinement: soft-argmin distances forward, gradients of an L1 loss
        # with respect to images and poses backward
        dict(op="refine", name="refine_512_n48", cols=512, rows=512, candidates=48, references=2, cameras=4,
             sigma_i=10.0, sigma_s=12.5),
        # scoring a batch of panoramas against ground truth
        dict(op="evaluate", name="evaluate_4x2048x1024", frames=4, cols=2048, rows=1024, thresholds=3),
        # input preparation of one frame: the cameras' decoded images to the matching resolution
        dict(op="resize", name="resize_4x1216_1024", images=4, src_cols=1216, src_rows=1216, cols=1024, rows=1024),
    ]


def _size(rng, low, high):
    """An integer spread over the logarithm of [low, high], odd ones among them."""
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    op = rng.choice(["frame", "frame", "batch", "batch", "uneven", "isb", "stitch", "refine", "evaluate", "resize"])
    sigma_i = round(rng.uniform(6.0, 16.0), 2)
    sigma_s = round(rng.uniform(4.0, 25.0), 2)
    if op in ("frame", "batch"):
        cols = _size(rng, 96 if op == "frame" else 192, 1024)
        rows = max(64, int(cols * rng.choice([1.0, 1.0, 0.75, 0.63])))
        image_cols = int(cols * rng.choice([1.0, 1.1875, 1.5, 2.0]))
        image_rows = max(64, int(round(rows * image_cols / cols)))
        if image_cols > 1300:
            image_cols, image_rows = cols, rows
        case = dict(op=op, cols=cols, rows=rows, image_cols=image_cols, image_rows=image_rows, pano_cols=2 * cols,
                    pano_rows=cols, cameras=4, candidates=rng.choice([16, 24, 32, 32, 37, 48, 64]),
                    references=rng.choice([1, 2, 2, 3, 4]), sigma_i=sigma_i, sigma_s=sigma_s)
        if op == "batch":
            case.update(frames=rng.randint(1, 8), storage=rng.choice(["fp16", "fp16", "unorm16"]),
                        inputs=rng.choice(["f32", "u8", "decoded"]))
        return case
    if op == "uneven":
        return dict(op=op, jobs=rng.randint(2, 9), rig_seed=rng.randint(1, 1 << 20), smallest=rng.choice([256, 512]),
                    largest=rng.choice([768, 1024]))
    if op == "isb":
        cols = _size(rng, 64, 1024)
        return dict(op=op, cols=cols, rows=max(64, int(cols * rng.choice([1.0, 0.75, 0.63]))),
                    candidates=rng.choice([1, 8, 17, 32, 32, 64]), sigma_i=sigma_i, sigma_s=sigma_s)
    if op == "stitch":
        cols = _size(rng, 128, 1024)
        return dict(op=op, cols=cols, rows=cols, image_cols=int(1.1875 * cols), image_rows=int(1.1875 * cols),
                    pano_cols=2 * cols, pano_rows=cols, references=rng.choice([1, 2, 3, 4]))
    if op == "refine":
        cols = _size(rng, 96, 512)
        return dict(op=op, cols=cols, rows=max(64, int(cols * rng.choice([1.0, 0.75]))),
                    candidates=rng.choice([16, 24, 32, 41, 48]), references=rng.choice([1, 2, 3]), cameras=4,
                    sigma_i=sigma_i, sigma_s=sigma_s)
    if op == "evaluate":
        rows = _size(rng, 128, 1024)
        return dict(op=op, frames=rng.randint(1, 4), cols=2 * rows, rows=rows, thresholds=rng.randint(0, 4))
    cols = _size(rng, 128, 1280)
    src = _size(rng, 128, 1600)
    return dict(op=op, images=rng.randint(1, 6), src_cols=src, src_rows=max(64, int(src * rng.choice([1.0, 0.75]))),
                cols=cols, rows=max(64, int(cols * rng.choice([1.0, 0.75]))))


# ---------------------------------------------------------------------------------------------
# Inputs: rigs and ray-cast scenes
# ---------------------------------------------------------------------------------------------
MIN_DIST, MAX_DIST = 0.55, 100.0
ROOM = (3.0, 1.5, 2.5)


def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _uniform(g, *shape, low=0.0, high=1.0):
    return low + (high - low) * torch.rand(*shape, generator=g, device=DEV)


def _scene(seed, spheres=20):
    g = _generator(seed)
    radius = _uniform(g, spheres, low=0.2, high=1.0)
    room = torch.tensor(ROOM, device=DEV)
    centre = (room - radius[:, None]) * _uniform(g, spheres, 3, low=-1.0, high=1.0)
    # spheres are kept 0.6 m away from the rig
    dist = centre.norm(dim=1, keepdim=True).clamp(min=1e-3)
    centre = centre * ((radius[:, None] + 0.6) / dist).clamp(min=1.0)
    return {"radius": radius, "centre": centre, "colour": _uniform(g, spheres + 1, 3, low=0.25, high=1.0),
            "lattice": _uniform(g, 32, 32, 32)}


def _noise(lattice, p, frequency):
    q = p * frequency
    f = torch.floor(q)
    t = q - f
    t = t * t * (3 - 2 * t)
    i = f.long()
    out = 0.0
    for dz in (0, 1):
        for dy in (0, 1):
            for dx in (0, 1):
                w = 1.0
                for axis, d in ((0, dx), (1, dy), (2, dz)):
                    w = w * (t[..., axis] if d else 1 - t[..., axis])
                out = out + w * lattice[(i[..., 2] + dz) % 32, (i[..., 1] + dy) % 32, (i[..., 0] + dx) % 32]
    return out


def _cast(scene, origin, dirs):
    room = torch.tensor(ROOM, device=DEV)
    step = torch.where(dirs.abs() > 1e-9, dirs, torch.full_like(dirs, 1e-9))
    best = ((torch.where(step > 0, room, -room) - origin) / step).amin(-1)
    ids = torch.full(best.shape, scene["radius"].numel(), dtype=torch.long, device=DEV)
    for s in range(scene["radius"].numel()):
        oc = origin - scene["centre"][s]
        b = dirs @ oc
        disc = b * b - (oc @ oc - scene["radius"][s] ** 2)
        t = -b - disc.clamp(min=0).sqrt()
        hit = (disc >= 0) & (t > 1e-6) & (t < best)
        best = torch.where(hit, t, best)
        ids = torch.where(hit, s, ids)
    return best, ids


def _render(scene, cam, cols, rows):
    """One camera's [rows, cols, 3] uint8 image and its distance map."""
    c = cam.scaled(cols, rows)
    v, u = torch.meshgrid(torch.arange(rows, device=DEV, dtype=torch.float32),
                          torch.arange(cols, device=DEV, dtype=torch.float32), indexing="ij")
    mx, my = (u - c.cx) / c.fx, (v - c.cy) / c.fy
    r2 = mx * mx + my * my
    disc = 1 - (2 * c.alpha - 1) * r2
    mz = (1 - c.alpha ** 2 * r2) / (c.alpha * disc.clamp(min=0).sqrt() + 1 - c.alpha)
    s = (mz * c.xi + (mz * mz + (1 - c.xi ** 2) * r2).clamp(min=0).sqrt()) / (mz * mz + r2)
    ray = torch.stack([s * mx, s * my, s * mz - c.xi], -1)
    dirs = (ray / ray.norm(dim=-1, keepdim=True)) @ torch.tensor(c.rotation, device=DEV, dtype=torch.float32).T
    origin = torch.tensor(c.position, device=DEV, dtype=torch.float32)
    t, ids = _cast(scene, origin, dirs)
    p = origin + t[..., None] * dirs
    n = sum(w * _noise(scene["lattice"], p, f) for w, f in ((0.45, 3.0), (0.35, 17.0), (0.2, 61.0)))
    rgb = scene["colour"][ids] * (0.2 + 0.8 * n[..., None]) * 255
    rgb = torch.where((disc >= 0)[..., None], rgb, torch.zeros_like(rgb))
    return rgb.clamp(0, 255).to(torch.uint8), t


def _square_rig(case):
    rig = _ss(".synthetic").square_rig(case["image_cols"], case["image_rows"])
    return rig[:case.get("cameras", 4)]


def _calibrations(rig, cols, rows):
    return _ss().parse_json_calib(_ss(".synthetic").basalt_calibration(rig), [cols, rows], "cpu")


def _masks(count, cols, rows):
    return [torch.ones(1, rows, cols) for _ in range(count)]


def _to_size(images, cols, rows):
    """uint8 [..., H, W, 3] -> float32 at (cols, rows), the linear resize of the input path."""
    x = images.reshape(-1, *images.shape[-3:]).permute(0, 3, 1, 2).float()
    if x.shape[2:] != (rows, cols):
        x = torch.nn.functional.interpolate(x, (rows, cols), mode="bilinear", align_corners=False)
    return x.permute(0, 2, 3, 1).reshape(*images.shape[:-3], rows, cols, 3).contiguous()


def _references(case):
    # the prototype's references are cameras 2 and 3; three or four take the first ones too
    return [2, 3, 0, 1][:case["references"]]


def _estimator(case, rig, references, **options):
    cols, rows = case["cols"], case["rows"]
    return _ss().RGBD_Estimator(_calibrations(rig, cols, rows), MIN_DIST, MAX_DIST, case["candidates"], references,
                                torch.zeros(3), _masks(len(rig), cols, rows), [cols, rows],
                                [case["image_cols"], case["image_rows"]], [case["pano_cols"], case["pano_rows"]],
                                case["sigma_i"], case["sigma_s"], DEV, **options)


# ---------------------------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------------------------

def prepare(case, seed):
    return globals()["_prepare_" + case["op"]](case, seed)


def run(state):
    return state["run"](state)


def _prepare_frame(case, seed):
    rig, refs = _square_rig(case), _references(case)
    scene = _scene(seed)
    images = torch.stack([_render(scene, cam, case["image_cols"], case["image_rows"])[0] for cam in rig])
    match = list(_to_size(images, case["cols"], case["rows"]))
    stitch = [images[r].float().contiguous() for r in refs]
    return {"run": _run_frame, "estimator": _estimator(case, rig, refs), "match": match, "stitch": stitch}


def _run_frame(s):
    rgb, distance = s["estimator"].estimate_RGBD_panorama(s["match"], s["stitch"])
    return {"rgb": rgb, "distance": distance}


def _prepare_batch(case, seed):
    rig, refs = _square_rig(case), _references(case)
    images = torch.stack([torch.stack([_render(scene, cam, case["image_cols"], case["image_rows"])[0] for cam in rig])
                          for scene in (_scene(seed * 64 + f) for f in range(case["frames"]))])
    stitch = images[:, refs].contiguous()
    if case["inputs"] == "decoded":
        match, stitch = images, None
    elif case["inputs"] == "u8":
        match = _to_size(images, case["cols"], case["rows"]).round().to(torch.uint8)
    else:
        match, stitch = _to_size(images, case["cols"], case["rows"]), stitch.float()
    est = _estimator(case, rig, refs, cost_storage=case["storage"], max_batch=case["frames"])
    return {"run": _run_batch, "estimator": est, "match": match, "stitch": stitch}


def _run_batch(s):
    rgb, distance = s["estimator"].estimate_RGBD_panoramas(s["match"], s["stitch"])
    return {"rgb": rgb, "distance": distance}


def _uneven_jobs(case):
    """Per job: size, candidates, cameras and the rig, from the case alone."""
    import numpy as np

    rng = np.random.Generator(np.random.PCG64(case["rig_seed"]))
    jobs = []
    sizes = [s for s in (256, 512, 768, 1024) if case["smallest"] <= s <= case["largest"]]
    for j in range(case["jobs"]):
        size, candidates = sizes[j % len(sizes)], (32, 64, 96)[(j // len(sizes)) % 3]
        cameras = int(rng.integers(3, 7))
        rig = _ss(".synthetic").ring_rig(rng, size, cameras)
        jobs.append(dict(cols=size, rows=size, image_cols=size, image_rows=size, pano_cols=2 * size, pano_rows=size,
                         candidates=candidates, cameras=cameras, sigma_i=10.0, sigma_s=25.0 * size / 1024, rig=rig))
    return jobs


def _prepare_uneven(case, seed):
    estimators, match, stitch = [], [], []
    for j, job in enumerate(_uneven_jobs(case)):
        scene = _scene(seed * 64 + j)
        images = torch.stack([_render(scene, cam, job["cols"], job["rows"])[0] for cam in job["rig"]])
        estimators.append(_estimator(job, job["rig"], [0, 1], cost_storage="fp16"))
        match.append(images)
        stitch.append(images[[0, 1]].contiguous())
    batch = _ss(".uneven").UnevenBatch(estimators, input_dtype=torch.uint8)
    return {"run": _run_uneven, "batch": batch, "match": match, "stitch": stitch}


def _run_uneven(s):
    return [{"rgb": rgb, "distance": distance} for rgb, distance in s["batch"].run(s["match"], s["stitch"])]


def _guide(image):
    """uint8 YCbCr of a [rows, cols, 3] uint8 image (float32, BT.709 limited range)."""
    r, g, b = image.float().unbind(-1)
    y = (r * 0.1826 + 16 + g * 0.6142 + b * 0.062).clamp(16, 235)
    cb = (128 - r * 0.1006 - g * 0.3386 + b * 0.4392).clamp(16, 240)
    cr = (r * 0.4392 + 128 - g * 0.3989 - b * 0.0403).clamp(16, 240)
    return torch.stack([y, cb, cr], -1).to(torch.uint8).contiguous()


def _isb_inputs(case, seed):
    """A guide, and a volume as matching costs are: a valley around each pixel's own candidate,
    with noise, clamped at 500."""
    rig = _ss(".synthetic").square_rig(case["cols"], case["rows"])
    image, distance = _render(_scene(seed), rig[0], case["cols"], case["rows"])
    n = case["candidates"]
    own = (1 / distance - 1 / MIN_DIST) / (1 / MAX_DIST - 1 / MIN_DIST) * max(n - 1, 1)
    g = _generator(seed + 1)
    k = torch.arange(n, device=DEV, dtype=torch.float32)[:, None, None]
    slope = _uniform(g, *own.shape, low=5.0, high=60.0)
    cost = (slope * (k - own).abs() + _uniform(g, n, *own.shape, high=40.0)).clamp(max=500)
    return _guide(image), cost.contiguous()


def _prepare_isb(case, seed):
    guide, cost = _isb_inputs(case, seed)
    f = _ss().ISB_Filter(case["candidates"], [case["cols"], case["rows"]], DEV)
    return {"run": _run_isb, "filter": f, "guide": guide, "cost": cost, "sigma": (case["sigma_i"], case["sigma_s"])}


def _run_isb(s):
    # the filter works in place: a program that keeps its volume filters a copy
    cost, guide = s["filter"].apply(s["guide"].clone(), s["cost"].clone(), *s["sigma"])
    return {"cost": cost, "guide": guide}


def _prepare_stitch(case, seed):
    rig, refs = _square_rig(case), _references(case)
    scene, g = _scene(seed), _generator(seed + 1)
    images = [_render(scene, rig[r], case["image_cols"], case["image_rows"])[0].contiguous() for r in refs]
    maps = []
    for r in refs:
        d = _render(scene, rig[r], case["cols"], case["rows"])[1]
        maps.append((d * _uniform(g, *d.shape, low=0.99, high=1.01)).clamp(MIN_DIST, MAX_DIST).contiguous())
    cal = _calibrations(rig, case["cols"], case["rows"])
    st = _ss().Stitcher([cal[r] for r in refs], torch.zeros(3), _masks(len(refs), case["cols"], case["rows"]), MIN_DIST,
                        MAX_DIST, [case["cols"], case["rows"]], [case["image_cols"], case["image_rows"]],
                        [case["pano_cols"], case["pano_rows"]], DEV)
    return {"run": _run_stitch, "stitcher": st, "images": images, "maps": maps}


def _run_stitch(s):
    rgb, distance = s["stitcher"].stitch(s["images"], s["maps"])
    return {"rgb": rgb, "distance": distance}


def _refine_inputs(case, seed):
    """The perturbed rig, its images (8-bit values in float32), the target inverse distances and
    the camera each reference pixel is matched with."""
    import numpy as np

    synthetic = _ss(".synthetic")
    rig, refs = synthetic.square_rig(case["cols"], case["rows"]), _references(case)
    scene = _scene(seed)
    views = [_render(scene, cam, case["cols"], case["rows"]) for cam in rig]
    images = torch.stack([v[0] for v in views]).float().contiguous()
    target = torch.stack([1 / views[r][1] for r in refs])
    noisy = synthetic.perturb_rig(rig, np.random.Generator(np.random.PCG64(seed)))
    cal = _calibrations(noisy, case["cols"], case["rows"])
    return cal, refs, images, target, [_largest_displacement(cal, r, case["cols"], case["rows"]) for r in refs]


def _prepare_refine(case, seed):
    cal, refs, images, target, selected = _refine_inputs(case, seed)
    size = [case["cols"], case["rows"]]
    sweep = _ss().DifferentiableSweep(cal, MIN_DIST, MAX_DIST, case["candidates"], refs, _masks(len(cal), *size), size,
                                      case["sigma_i"], case["sigma_s"], DEV)
    sweep.set_selection(selected)
    deltas = torch.zeros(len(cal), 6, dtype=torch.float64, device=DEV, requires_grad=True)
    return {"run": _run_refine, "sweep": sweep, "images": images.requires_grad_(), "deltas": deltas, "target": target}


def _run_refine(s):
    q = s["sweep"](s["images"], s["deltas"])
    loss = (q - s["target"]).abs().mean()
    gi, gd = torch.autograd.grad(loss, [s["images"], s["deltas"]])
    return {"inverse_distance": q.detach(), "grad_images": gi, "grad_poses": gd}


def _prepare_evaluate(case, seed):
    f, rows, cols = case["frames"], case["rows"], case["cols"]
    g = _generator(seed)
    y, x = torch.meshgrid(torch.arange(rows, device=DEV) / rows, torch.arange(cols, device=DEV) / cols, indexing="ij")
    p = torch.stack([x * 6, y * 3, x * 0 + 0.5], -1)
    gt_rgb, gt_inv = [], []
    for _ in range(f):
        lattice = _uniform(g, 32, 32, 32)
        n = torch.stack([sum(w * _noise(lattice, p + 3 * ch, s) for w, s in ((0.5, 2.0), (0.3, 9.0), (0.2, 41.0)))
                         for ch in range(3)], -1)
        gt_rgb.append((n * 255).clamp(0, 255).to(torch.uint8))
        gt_inv.append(0.1 + 1.6 * _noise(lattice, p, 1.3))
    gt_rgb, gt_inv = torch.stack(gt_rgb), torch.stack(gt_inv).float().contiguous()
    noise = torch.randn(gt_rgb.shape, generator=g, device=DEV) * 4
    rgb = (gt_rgb.float() + noise).round().clamp(0, 255).to(torch.uint8)
    inv = (gt_inv + 0.03 * torch.randn(gt_inv.shape, generator=g, device=DEV)).contiguous()
    return {"run": _run_evaluate, "args": (rgb, inv, gt_rgb, gt_inv),
            "thresholds": [0.1, 0.3, 0.5, 0.05][:case["thresholds"]]}


def _run_evaluate(s):
    return _ss(".evaluation").evaluate_panoramas(*s["args"], s["thresholds"])


def _prepare_resize(case, seed):
    scene = _scene(seed)
    rig = _ss(".synthetic").square_rig(case["src_cols"], case["src_rows"], count=case["images"])
    images = torch.stack([_render(scene, cam, case["src_cols"], case["src_rows"])[0] for cam in rig]).contiguous()
    return {"run": _run_resize, "images": images, "size": (case["cols"], case["rows"])}


def _run_resize(s):
    return _ss(".utils").resize_linear(s["images"], s["size"])


# ---------------------------------------------------------------------------------------------
# Work of one pass: inputs read once, outputs written once; operations of the method
# ---------------------------------------------------------------------------------------------

def _filter_flops(cols, rows, candidates):
    """Per candidate and fine pixel of a level pair: 9 taps down on a quarter of the pixels, 25
    weighted taps up per four pixels; the levels below add a third."""
    return cols * rows * candidates * (18 / 4 + 58 / 4) * 4 / 3


def _frame_work(c, image_bytes):
    """One frame: images to match and to stitch, the rig's tables and the two panoramas; per
    sample of the sweep about 60 operations to transform, project, sample and compare."""
    P, Q = c["cols"] * c["rows"], c["pano_cols"] * c["pano_rows"]
    S, R, n = c["image_cols"] * c["image_rows"], c["references"], c["candidates"]
    if image_bytes == 0:  # the decoded images, stitched in place
        images = 3 * S * c["cameras"]
    else:
        images = 3 * image_bytes * (P * c["cameras"] + S * R)
    return {"bytes": images + R * (P * 3 + Q * 12) + Q * 7,
            "flops": R * (60.0 * P * n + _filter_flops(c["cols"], c["rows"], n) + 200.0 * P) + 150.0 * Q * R}


def work(case):
    op = case["op"]
    if op == "frame":
        return _frame_work(case, 4)
    if op == "batch":
        w = _frame_work(case, {"f32": 4, "u8": 1, "decoded": 0}[case["inputs"]])
        return {k: v * case["frames"] for k, v in w.items()}
    if op == "uneven":
        parts = [_frame_work(dict(j, references=2), 1) for j in _uneven_jobs(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    if op == "stitch":
        P, Q, R = case["cols"] * case["rows"], case["pano_cols"] * case["pano_rows"], case["references"]
        return {"bytes": R * (6 * P + 12 * Q + 3 * case["image_cols"] * case["image_rows"]) + 7 * Q,
                "flops": 100.0 * P * R + 150.0 * Q * R}
    P = case["cols"] * case["rows"]
    if op == "isb":
        return {"bytes": 2 * P * (4 * case["candidates"] + 3),
                "flops": _filter_flops(case["cols"], case["rows"], case["candidates"])}
    if op == "refine":
        n, R, C = case["candidates"], case["references"], case["cameras"]
        # the backward evaluates the forward again and the transposed filter and samples
        return {"bytes": 2 * 12 * P * C + R * P * (1 + 4 + 4 + 4),
                "flops": R * (60.0 * P * n * 2 + 150.0 * P * n + 3 * _filter_flops(case["cols"], case["rows"], n))}
    if op == "evaluate":
        return {"bytes": case["frames"] * P * 14, "flops": case["frames"] * P * 3 * 60.0}
    return {"bytes": 3 * case["images"] * (case["src_cols"] * case["src_rows"] + 4 * P),
            "flops": case["images"] * P * 3 * 9.0}


# ---------------------------------------------------------------------------------------------
# 64-bit values.  Panoramas have none: the candidate of smallest cost and the z-buffer of the
# reprojection are choices between values that 32 and 64 bits order differently.
# ---------------------------------------------------------------------------------------------

def exact(case, seed):
    f = globals().get("_exact_" + case["op"])
    return None if f is None else f(case, seed)


def _exact_resize(case, seed):
    images = _prepare_resize(case, seed)["images"]
    if (2 * case["cols"], 2 * case["rows"]) == (case["src_cols"], case["src_rows"]):
        x = images.double().reshape(images.shape[0], case["rows"], 2, case["cols"], 2, 3)
        return x.mean(dim=(2, 4))

    def taps(dst, src):
        at = (torch.arange(dst, device=DEV, dtype=torch.float64) + 0.5) * (src / dst) - 0.5
        at = at.clamp(0, src - 1)
        i = at.floor().clamp(max=max(src - 2, 0)).long()
        return i, (i + 1).clamp(max=src - 1), at - i

    y0, y1, fy = taps(case["rows"], case["src_rows"])
    x0, x1, fx = taps(case["cols"], case["src_cols"])
    out = []
    for image in images.double():
        h = image[:, x0] * (1 - fx)[None, :, None] + image[:, x1] * fx[None, :, None]
        out.append(h[y0] * (1 - fy)[:, None, None] + h[y1] * fy[:, None, None])
    return torch.stack(out)


def _exact_evaluate(case, seed):
    s = _prepare_evaluate(case, seed)
    rows = []
    for rgb, inv, gt_rgb, gt_inv in zip(*s["args"]):
        # the images are float32 values in [0, 1]; everything after that in 64 bits
        x, y = (gt_rgb.float() / 255).double(), (rgb.float() / 255).double()
        psnr = 10 * torch.log10(1 / ((x - y) ** 2).mean())

        def mean(v):
            return torch.nn.functional.avg_pool2d(v.permute(2, 0, 1)[:, None], 7, 1)

        ux, uy = mean(x), mean(y)
        k = 49 / 48
        vx, vy, vxy = k * (mean(x * x) - ux * ux), k * (mean(y * y) - uy * uy), k * (mean(x * y) - ux * uy)
        c1, c2 = (0.01 * 2) ** 2, (0.03 * 2) ** 2
        ssim = ((2 * ux * uy + c1) * (2 * vxy + c2) / ((ux * ux + uy * uy + c1) * (vx + vy + c2))).mean()
        e = (inv.double() - gt_inv.double()).abs()
        bad = [100 * (e.float() > torch.tensor(t, device=DEV)).double().mean() for t in s["thresholds"]]
        rows.append(torch.stack([psnr, ssim, e.mean(), (e * e).mean().sqrt(), *bad]))
    return torch.stack(rows)


# --- the ISB filter in 64 bits: the guides are bytes and follow their definition in float32 ------

def _levels(cols, rows):
    count = int(min(math.log2(cols), math.log2(rows)) - 1)
    return [(math.ceil(rows / 2 ** s), math.ceil(cols / 2 ** s)) for s in range(count)]


def _range_weight(a, b, var):
    d = (a - b).abs().sum(-1)
    return torch.exp(-d * d * var) + 0.01


def _at(x, rows, cols, channels_last):
    return x[rows][:, cols] if channels_last else x[:, rows][:, :, cols]


_DOWN = ((-1, -1), (0, -1), (1, -1), (1, 0), (1, 1), (0, 1), (-1, 1), (-1, 0))  # (row, column)
_UP = {(0, 0): ([(r, c) for r in (-1, 0, 1) for c in (-1, 0, 1)], [1, 1, 1, 1, 8, 1, 1, 1, 1]),
       (1, 0): ([(0, 0), (1, 0), (0, -1), (1, -1), (0, 1), (1, 1)], [8, 8, 1, 1, 1, 1]),
       (0, 1): ([(0, 0), (0, 1), (-1, 0), (-1, 1), (1, 0), (1, 1)], [8, 8, 1, 1, 1, 1]),
       (1, 1): ([(0, 0), (0, 1), (1, 0), (1, 1)], [1, 1, 1, 1])}


def _down_step(guide, cost, shape, sigma_i):
    """(coarse guide, coarse cost) of a level: 3 x 3 taps around every second pixel."""
    (ri, ci), (ro, co) = guide.shape[:2], shape
    y, x = 2 * torch.arange(ro, device=DEV), 2 * torch.arange(co, device=DEV)
    centre = _at(guide, y, x, True).float()
    gsum, wsum, csum, wsum64 = centre, 1.0, _at(cost, y, x, False), 1.0
    for dr, dc in _DOWN:
        yy, xx = (y + dr).clamp(0, ri - 1), (x + dc).clamp(0, ci - 1)
        tap = _at(guide, yy, xx, True).float()
        base = 0.25 if dr and dc else 0.5
        w = base * _range_weight(centre, tap, 1 / (2 * sigma_i ** 2))
        gsum, wsum = gsum + tap * w[..., None], wsum + w
        w64 = base * _range_weight(centre.double(), tap.double(), 1 / (2 * sigma_i ** 2))
        csum, wsum64 = csum + _at(cost, yy, xx, False) * w64, wsum64 + w64
    return (gsum * (1 / wsum)[..., None]).to(torch.uint8), csum / wsum64


def _up_step(coarse_guide, coarse_cost, guide, cost, level, sigma_i, sigma_s):
    """(filtered guide, filtered cost) of the finer level of a pair."""
    (ri, ci), (ro, co) = coarse_guide.shape[:2], guide.shape[:2]
    down = math.exp(-((2 ** level - 0.5) ** 2) / (2 * sigma_s ** 2))
    up = 1 - down
    out_guide, out_cost = guide.clone(), [None] * 4
    for f, ((fr, fc), (taps, bases)) in enumerate(_UP.items()):
        y, x = torch.arange(fr, ro, 2, device=DEV), torch.arange(fc, co, 2, device=DEV)
        own = _at(guide, y, x, True).float()
        gsum, wsum = own * torch.tensor(up, dtype=torch.float32), torch.tensor(up, dtype=torch.float32, device=DEV)
        csum, wsum64 = up * _at(cost, y, x, False), up
        for (dr, dc), base in zip(taps, bases):
            yy, xx = (y // 2 + dr).clamp(0, ri - 1), (x // 2 + dc).clamp(0, ci - 1)
            tap = _at(coarse_guide, yy, xx, True).float()
            w = base * (torch.tensor(down, dtype=torch.float32) * _range_weight(own, tap, 1 / (2 * sigma_i ** 2)))
            gsum, wsum = gsum + tap * w[..., None], wsum + w
            w64 = base * down * _range_weight(own.double(), tap.double(), 1 / (2 * sigma_i ** 2))
            csum, wsum64 = csum + _at(coarse_cost, yy, xx, False) * w64, wsum64 + w64
        out_guide[fr::2, fc::2] = (gsum * (1 / wsum)[..., None]).to(torch.uint8)
        out_cost[f] = csum / wsum64
    # the four phases back into one map, differentiably
    full = torch.zeros_like(cost)
    for (fr, fc), part in zip(_UP, out_cost):
        rows, cols = torch.arange(fr, ro, 2, device=DEV), torch.arange(fc, co, 2, device=DEV)
        full = full.index_put((torch.arange(cost.shape[0], device=DEV)[:, None, None], rows[:, None], cols), part)
    return out_guide, full


def _filter64(guide, cost, sigma_i, sigma_s):
    guides, costs = [guide], [cost]
    for shape in _levels(guide.shape[1], guide.shape[0])[1:]:
        g, c = _down_step(guides[-1], costs[-1], shape, sigma_i)
        guides.append(g)
        costs.append(c)
    for s in range(len(guides) - 2, -1, -1):
        guides[s], costs[s] = _up_step(guides[s + 1], costs[s + 1], guides[s], costs[s], s, sigma_i, sigma_s)
    return costs[0]


def _exact_isb(case, seed):
    guide, cost = _isb_inputs(case, seed)
    return {"cost": _filter64(guide, cost.double(), case["sigma_i"], case["sigma_s"]), "guide": None}


# --- the differentiable sweep in 64 bits ----------------------------------------------------------

def _intrinsics(c):
    fl, pp = c.fl * c.matching_scale, c.principal * c.matching_scale
    return [float(fl[0]), float(fl[1]), float(pp[0]), float(pp[1]), float(c.xi), float(c.alpha)]


def _rays(c, cols, rows):
    fx, fy, cx, cy, xi, al = _intrinsics(c)
    v, u = torch.meshgrid(torch.arange(rows, device=DEV, dtype=torch.float64),
                          torch.arange(cols, device=DEV, dtype=torch.float64), indexing="ij")
    mx, my = (u - cx) / fx, (v - cy) / fy
    r2 = mx * mx + my * my
    disc = 1 - (2 * al - 1) * r2
    mz = (1 - al * al * r2) / (al * disc.clamp(min=0).sqrt() + 1 - al)
    s = (mz * xi + (mz * mz + (1 - xi * xi) * r2).sqrt()) / (mz * mz + r2)
    return torch.stack([s * mx, s * my, s * mz - xi], -1), disc >= 0


def _project(p, k):
    fx, fy, cx, cy, xi, al = k
    d1 = p.norm(dim=-1)
    c = xi * d1 + p[..., 2]
    d2 = (p[..., 0] ** 2 + p[..., 1] ** 2 + c * c).sqrt()
    n = al * d2 + (1 - al) * c
    w1 = (1 - al) / al if al > 0.5 else al / (1 - al)
    w2 = (w1 + xi) / math.sqrt(2 * w1 * xi + xi * xi + 1)
    return fx * p[..., 0] / n + cx, fy * p[..., 1] / n + cy, p[..., 2] > -w2 * d1


def _largest_displacement(cal, r, cols, rows):
    """Per pixel of camera r, the other camera that sees its nearest and farthest candidate
    furthest apart (more than a pixel), or -1."""
    ray, valid = _rays(cal[r], cols, rows)
    best = torch.ones(rows, cols, dtype=torch.float64, device=DEV)
    selected = torch.full((rows, cols), -1, dtype=torch.int8, device=DEV)
    for c, cam in enumerate(cal):
        rel = (torch.linalg.inv(cam.rt.double()) @ cal[r].rt.double()).to(DEV)
        ends = [_project((d * ray) @ rel[:3, :3].T + rel[:3, 3], _intrinsics(cam)) for d in (MIN_DIST, MAX_DIST)]
        (u0, v0, ok0), (u1, v1, ok1) = ends
        inside = [(u >= 0) & (u <= cols - 1) & (v >= 0) & (v <= rows - 1) for u, v in ((u0, v0), (u1, v1))]
        disp = torch.hypot(u0 - u1, v0 - v1)
        take = (disp > best) & valid & ok0 & ok1 & inside[0] & inside[1]
        best = torch.where(take, disp, best)
        selected = torch.where(take, torch.full_like(selected, c), selected)
    return selected


def _sample(image, u, v):
    """Bilinear, zero outside; two horizontal interpolations and a vertical one."""
    rows, cols = image.shape[:2]
    x0, y0 = u.detach().floor(), v.detach().floor()
    fx, fy = (u - x0)[..., None], (v - y0)[..., None]
    t = []
    for dx, dy in ((0, 0), (1, 0), (0, 1), (1, 1)):
        xs, ys = x0 + dx, y0 + dy
        inside = (xs >= 0) & (xs < cols) & (ys >= 0) & (ys < rows)
        t.append(image[ys.clamp(0, rows - 1).long(), xs.clamp(0, cols - 1).long()] * inside[..., None])
    top, bottom = t[0] + fx * (t[1] - t[0]), t[2] + fx * (t[3] - t[2])
    return top + fy * (bottom - top)


def _perturbed(rt, delta):
    """rt [Exp(omega), v] to first order in delta = 0, where value and gradient are exact."""
    z = torch.zeros((), dtype=torch.float64, device=DEV)
    w, v = delta[:3], delta[3:]
    turn = torch.stack([torch.stack([z, -w[2], w[1], v[0]]), torch.stack([w[2], z, -w[0], v[1]]),
                        torch.stack([-w[1], w[0], z, v[2]]), torch.stack([z, z, z, z])])
    return rt.double().to(DEV) @ (torch.eye(4, dtype=torch.float64, device=DEV) + turn)


def _exact_refine(case, seed):
    cal, refs, images, target, selected = _refine_inputs(case, seed)
    cols, rows, n = case["cols"], case["rows"], case["candidates"]
    guides = [_guide(images[r]) for r in refs]
    images = images.double().requires_grad_()
    deltas = torch.zeros(len(cal), 6, dtype=torch.float64, device=DEV, requires_grad=True)
    distance = (1 / torch.linspace(1 / MIN_DIST, 1 / MAX_DIST, n)).double().to(DEV)[:, None, None]
    out, grads = [], [torch.zeros_like(images), torch.zeros_like(deltas)]
    for slot, r in enumerate(refs):
        poses = [_perturbed(c.rt, d) for c, d in zip(cal, deltas)]
        ray = _rays(cal[r], cols, rows)[0]
        sample = torch.zeros(n, rows, cols, 3, dtype=torch.float64, device=DEV)
        for c, cam in enumerate(cal):
            if not bool((selected[slot] == c).any()):
                continue
            rel = torch.linalg.inv(poses[c]) @ poses[r]
            u, v, _ = _project((distance[..., None] * ray) @ rel[:3, :3].T + rel[:3, 3], _intrinsics(cam))
            sample = torch.where((selected[slot] == c)[None, ..., None], _sample(images[c], u, v), sample)
        cost = (sample - images[r]).abs().sum(-1).clamp(max=500)
        f = _filter64(guides[slot], cost, case["sigma_i"], case["sigma_s"])
        q = (torch.softmax(-f / 2.0, 0) / distance).sum(0)
        out.append(q.detach())
        loss = (q - target[slot].double()).abs().sum() / target.numel()
        for total, g in zip(grads, torch.autograd.grad(loss, [images, deltas])):
            total += g
    return {"inverse_distance": torch.stack(out), "grad_images": grads[0], "grad_poses": grads[1]}
