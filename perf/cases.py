"""The work a user has this framework do, as cases that can be timed and compared.

Every case goes through a public entry point: `GaussianRasterizer` (views and training
steps), `cfgs.pose` and `cfgs.batch.BatchSolver` (relative-pose solves),
`cfgs.pose.photometric_loss` (L1 + SSIM), `cfgs.pointcloud` (a frame's initial
Gaussians) and `cfgs.densify.GaussianOptimizer` (Adam, densification). Sizes and value
distributions are those of `cfgs.scenes`, the tests and `bench.py`.

`exact` restates each path in float64 PyTorch, without this repository's code.
"""
from __future__ import annotations

import math
import os
import sys

import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_ROOT, "cf-3dgs_gb300"))

import diff_gaussian_rasterization as dgr  # noqa: E402
from cfgs import batch, densify, loss, pointcloud, pose, scenes  # noqa: E402

DEV = "cuda"
F64 = torch.float64
LAMBDA_DSSIM = 0.2  # weight of 1 - SSIM in the photometric loss
EPOCH = 25          # iterations the server advances its pose solves by at a time
LRS = {"xyz": 1.6e-4 * 3.2, "f_dc": 2.5e-3, "f_rest": 2.5e-3 / 20, "opacity": 0.05, "scaling": 5e-3, "rotation": 1e-3}
DENSIFY = {"max_grad": 2e-4, "min_opacity": 0.005, "extent": 3.0, "max_screen_size": 20, "percent_dense": 0.01}
POSE_RESOLUTIONS = [(320, 180), (640, 360), (960, 540)]


def listed():
    return [
        # one view of a small scene, as an interactive viewer or an evaluation loop asks for it
        {"name": "view_256", "kind": "view", "cloud": "room", "n": 16384, "width": 256, "height": 256, "sh_degree": 3},
        # one novel view of a full scene
        {"name": "view_1080p", "kind": "view", "cloud": "field", "n": 1_000_000, "width": 1920, "height": 1080,
         "sh_degree": 3},
        # the training step of a small scene: render, RGB L1, all gradients
        {"name": "train_256", "kind": "train", "cloud": "room", "n": 16384, "width": 256, "height": 256, "sh_degree": 3,
         "precomputed": False, "geometry": False},
        # a step with colours and covariances computed outside and depth and alpha in the loss, ragged sizes
        {"name": "train_odd_geometry", "kind": "train", "cloud": "field", "n": 250_007, "width": 977, "height": 545,
         "sh_degree": 0, "precomputed": True, "geometry": True},
        # the training step of a full scene at full resolution
        {"name": "train_1080p", "kind": "train", "cloud": "field", "n": 1_000_000, "width": 1920, "height": 1080,
         "sh_degree": 3, "precomputed": False, "geometry": False},
        # one iteration of a relative-pose solve on the full photometric loss, written as a loop of PyTorch calls
        {"name": "pose_step_360p", "kind": "pose_step", "n": 640 * 360, "width": 640, "height": 360},
        # a single pose solve on the solve engine, one epoch of the server
        {"name": "pose_epoch_1", "kind": "pose_epoch", "solves": 1, "n": 640 * 360, "width": 640, "height": 360},
        # the server's continuous batch: solves of mixed sizes advanced together, one epoch
        {"name": "pose_epoch_16", "kind": "pose_epoch", "solves": 16, "n": 0, "width": 0, "height": 0},
        # the photometric loss of a rendered frame and its image gradient
        {"name": "loss_1080p", "kind": "loss", "width": 1920, "height": 1080},
        # a new frame's Gaussians from its depth map: unproject, voxel grid, neighbour scales
        {"name": "frame_360p", "kind": "frame", "width": 640, "height": 360},
        # the optimiser step of a full model with its densification statistics
        {"name": "optimise_1m", "kind": "optimise", "n": 1_000_000},
        # clone, split and prune a full model
        {"name": "densify_1m", "kind": "densify", "n": 1_000_000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["view", "view", "train", "train", "train", "pose_step", "pose_epoch", "loss", "frame", "optimise",
                       "densify"])
    if kind in ("view", "train"):
        n = _log_int(rng, 4000, 1_000_000)
        room = n <= 65536
        width = _log_int(rng, 130, 640) if room else _log_int(rng, 320, 1920)
        case = {"kind": kind, "cloud": "room" if room else "field", "n": n, "width": width,
                "height": max(64, int(width * rng.uniform(0.5, 0.75 if not room else 1.0))), "sh_degree": rng.randint(0, 3)}
        case["height"] = min(case["height"], 1080)
        if kind == "train":
            case["precomputed"] = rng.random() < 0.25
            case["geometry"] = rng.random() < 0.25
        return case
    if kind == "pose_step":
        width = _log_int(rng, 200, 960)
        height = int(width * 9 / 16) + rng.randint(0, 3)
        return {"kind": kind, "n": _log_int(rng, 0.3 * width * height, 1.0 * width * height), "width": width,
                "height": height}
    if kind == "pose_epoch":
        if rng.random() < 0.5:
            width, height = rng.choice(POSE_RESOLUTIONS)
            return {"kind": kind, "solves": 1, "n": _log_int(rng, 50_000, 500_000), "width": width, "height": height}
        return {"kind": kind, "solves": rng.randint(2, 15), "n": 0, "width": 0, "height": 0}
    if kind in ("loss", "frame"):
        width = _log_int(rng, 200, 1920 if kind == "loss" else 1280)
        return {"kind": kind, "width": width, "height": int(width * rng.uniform(0.5, 0.7))}
    return {"kind": kind, "n": _log_int(rng, 30_000, 1_000_000)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) & 0x7FFFFFFF)


def _rand(g, *shape, lo=0.0, hi=1.0):
    return lo + (hi - lo) * torch.rand(*shape, device=DEV, generator=g)


def _randn(g, *shape, mean=0.0, std=1.0):
    return mean + std * torch.randn(*shape, device=DEV, generator=g)


def _unit_quats(g, n):
    q = _randn(g, n, 4)
    return q / q.norm(dim=1, keepdim=True)


def _cloud(case, seed):
    """Activated Gaussians of a scene: "room" (uniform in a box in front of the camera) or
    "field" (a wide normal cloud), a camera and a target image."""
    g, n, width, height = _gen(seed), case["n"], case["width"], case["height"]
    degree = case["sh_degree"]
    if case["cloud"] == "room":
        means = torch.cat([_rand(g, n, 2, lo=-1, hi=1), _rand(g, n, 1, lo=2, hi=6)], 1)
        log_scale, logit, focal = (-3.5, 0.5), (0.0, 1.0), float(width)
    else:
        means = _randn(g, n, 3, std=math.sqrt(2.0))
        means[:, 2] = (means[:, 2] + 8.0).clamp_min(0.21)
        log_scale, logit, focal = (-4.5, 1.0), (-1.0, 1.5), 1400.0 * width / 1920.0
    sh = _randn(g, n, (degree + 1) ** 2, 3, std=0.05)
    sh[:, 0] *= 10.0
    out = {"means3D": means, "opacities": torch.sigmoid(_randn(g, n, 1, mean=logit[0], std=logit[1])), "shs": sh,
           "scales": torch.exp(_randn(g, n, 3, mean=log_scale[0], std=log_scale[1])), "rotations": _unit_quats(g, n)}
    if case.get("precomputed"):
        out["colors_precomp"] = (0.28209479177387814 * out.pop("shs")[:, 0] + 0.5).clamp_min(0.0)
        out["cov3D_precomp"] = _covariance(out.pop("scales").double(), out.pop("rotations").double()).float()
    images = {"color": _rand(g, 3, height, width), "depth": _rand(g, 1, height, width, lo=2, hi=10),
              "alpha": _rand(g, 1, height, width)}
    return out, images, scenes.make_camera(width, height, focal, focal).to(DEV)


def _settings(cam, sh_degree):
    return dgr.GaussianRasterizationSettings(cam.height, cam.width, cam.tanfovx, cam.tanfovy,
                                             torch.zeros(3, device=DEV), 1.0, cam.viewmatrix, cam.projmatrix, sh_degree,
                                             cam.campos, False, False)


def _field(g, u, v, waves):
    """A smooth random field: a sum of 2D sinusoids at the normalised coordinates (u, v)."""
    k, phase, amp = _rand(g, waves, 2, lo=-6, hi=6).double(), _rand(g, waves, hi=2 * math.pi).double(), \
        _rand(g, waves, lo=0.5).double()
    return lambda du=0.0, dv=0.0: sum(amp[i] * torch.sin(2 * math.pi * (k[i, 0] * (u + du) + k[i, 1] * (v + dv))
                                                         + phase[i]) for i in range(waves))


def _pose_inputs(n, width, height, seed):
    """One pose solve: Gaussians back-projected from a smooth depth field in [1, 10] (one per
    pixel, or n at random sub-pixel positions), coloured by a smooth field; the target
    frame shows the colour field displaced by a few pixels."""
    g = _gen(seed)
    fx = 500.0 * width / 640.0
    if n == width * height:
        vv, uu = torch.meshgrid(torch.arange(height, device=DEV, dtype=F64), torch.arange(width, device=DEV, dtype=F64),
                                indexing="ij")
        uu, vv, widen = uu.reshape(-1), vv.reshape(-1), 1.0
    else:
        uu, vv = _rand(g, n, hi=width).double() - 0.5, _rand(g, n, hi=height).double() - 0.5
        widen = math.sqrt(width * height / n)
    f = _field(g, (uu + 0.5) / width, (vv + 0.5) / height, 8)()
    depth = 1.0 + 9.0 * (f - f.min()) / (f.max() - f.min())
    means = torch.stack([(uu + 0.5 - width / 2) * depth / fx, (vv + 0.5 - height / 2) * depth / fx, depth], 1)
    pv, pu = torch.meshgrid((torch.arange(height, device=DEV, dtype=F64) + 0.5) / height,
                            (torch.arange(width, device=DEV, dtype=F64) + 0.5) / width, indexing="ij")
    shift = _rand(g, 2, lo=-4, hi=4).double()
    rgb, target = [], []
    for c in range(3):
        colour_seed = int(seed) * 3 + c + 1
        a = _field(_gen(colour_seed), (uu + 0.5) / width, (vv + 0.5) / height, 4)()
        lo, hi = a.min(), a.max()
        rgb.append(0.1 + 0.8 * (a - lo) / (hi - lo))
        b = _field(_gen(colour_seed), pu, pv, 4)(shift[0] / width, shift[1] / height)
        target.append((0.1 + 0.8 * (b - lo) / (hi - lo)).clamp(0, 1))
    scales = (depth / fx * widen)[:, None].repeat(1, 3)
    rots = torch.zeros(means.shape[0], 4, device=DEV)
    rots[:, 0] = 1.0
    cam = scenes.make_camera(width, height, fx, fx).to(DEV)
    sh = ((torch.stack(rgb, 1) - 0.5) / 0.28209479177387814)[:, None, :]
    opacity = torch.full((means.shape[0], 1), 1.0 / (1.0 + math.exp(-2.0)), device=DEV)
    return pose.PoseProblem(means.float(), opacity, sh.float().contiguous(), scales.float(), rots, 0,
                            _settings(cam, 0), torch.stack(target).float().contiguous()), cam


def _pose_specs(case, seed):
    """(n, width, height, seed) of the case's solves; a batch mixes resolutions and counts."""
    if case["solves"] == 1:
        return [(case["n"], case["width"], case["height"], seed)]
    g = torch.Generator().manual_seed(3 + case["solves"])  # the mix is the case's, the contents the seed's
    out = []
    for s in range(case["solves"]):
        n = int(round(math.exp(math.log(5e4) + torch.rand((), generator=g).item() * math.log(10.0))))
        width, height = POSE_RESOLUTIONS[int(torch.randint(0, 3, (), generator=g))]
        out.append((n, width, height, int(seed) * 64 + s))
    return out


def _frame_inputs(case, seed):
    """A depth map, its colours, the intrinsics and the voxel size. Monocular depth has no unit: a
    seed draws the scale (a power of two, so that the same voxels are occupied at any of
    them) and the colours; the surface is the case's."""
    width, height = case["width"], case["height"]
    g, scale = _gen(width), 2.0 ** (int(seed) % 7 - 3)
    v, u = torch.meshgrid(torch.arange(height, device=DEV) * (360.0 / height),
                          torch.arange(width, device=DEV) * (640.0 / width), indexing="ij")
    phase = _rand(g, 2, hi=2 * math.pi)
    depth = 2.0 + 0.5 * torch.sin(u / 37.0 + phase[0]) + 0.3 * torch.cos(v / 23.0 + phase[1])
    depth = depth + 0.02 * _randn(g, height, width)
    f = 500.0 * width / 640.0
    K = [[f, 0.0, width / 2.0], [0.0, f, height / 2.0], [0.0, 0.0, 1.0]]
    return depth * scale, _rand(_gen(seed), height * width, 3), K, 0.01 * scale


def _model(case, seed):
    """Raw parameters of a model, its Adam moments and its accumulated statistics. What
    decides how many Gaussians are cloned, split and pruned is the case's; which ones they
    are is the seed's."""
    g, n = _gen(seed), case["n"]
    own, order = _gen(n), torch.randperm(n, device=DEV, generator=g)
    p = {"xyz": _randn(g, n, 3), "f_dc": _randn(g, n, 1, 3), "f_rest": _randn(g, n, 15, 3, std=0.1),
         "opacity": _randn(own, n, 1, std=2.0)[order], "scaling": _randn(own, n, 3, mean=-4.0)[order],
         "rotation": _randn(g, n, 4)}
    m = {k: _randn(g, *v.shape, std=0.01) for k, v in p.items()}
    s = {k: _rand(g, *v.shape, lo=1e-6, hi=1e-3) for k, v in p.items()}
    grads = {k: _randn(g, *v.shape, std=0.01) for k, v in p.items()}
    denom = torch.randint(0, 40, (n,), device=DEV, generator=own).float()[order]
    accum = denom * torch.exp(_randn(own, n, mean=math.log(1e-4), std=0.8))[order]
    radii = (torch.randint(-60, 140, (n,), device=DEV, generator=g)).clamp_min(0).int()
    z = _randn(g, 2, n, 3)
    return {"params": p, "exp_avg": m, "exp_avg_sq": s, "grads": grads, "accum": accum, "denom": denom, "radii": radii,
            "grad2D": _randn(g, n, 3, std=1e-4), "z": z}


def _splits(model):
    """Points densification splits: large and with a large accumulated gradient."""
    grad = (model["accum"] / model["denom"]).nan_to_num(0.0)
    big = model["params"]["scaling"].exp().max(1).values > DENSIFY["percent_dense"] * DENSIFY["extent"]
    return (grad >= DENSIFY["max_grad"]) & big


def prepare(case, seed):
    kind = case["kind"]
    state = {"kind": kind, "case": dict(case)}
    if kind in ("view", "train"):
        inputs, images, cam = _cloud(case, seed)
        state["rasterizer"] = dgr.GaussianRasterizer(_settings(cam, case["sh_degree"]))
        inputs["means2D"] = torch.zeros_like(inputs["means3D"])
        if kind == "train":
            inputs = {k: v.requires_grad_(True) for k, v in inputs.items()}
            state["images"] = images
        state["inputs"] = inputs
    elif kind == "pose_step":
        state["problem"], _ = _pose_inputs(case["n"], case["width"], case["height"], seed)
        state["xi"] = _randn(_gen(int(seed) + 77), 6, std=0.004)
        state["optimizer"] = pose.FusedAdam(state["xi"])
    elif kind == "pose_epoch":
        state["solver"] = batch.BatchSolver([_pose_inputs(*spec)[0] for spec in _pose_specs(case, seed)])
    elif kind == "loss":
        g = _gen(seed)
        target = _rand(g, 3, case["height"], case["width"])
        state["target"] = target
        state["image"] = (target + _randn(g, *target.shape, std=0.1)).requires_grad_(True)
    elif kind == "frame":
        state["depth"], state["rgb"], state["K"], state["voxel"] = _frame_inputs(case, seed)
    elif kind in ("optimise", "densify"):
        model = _model(case, seed)
        opt = densify.GaussianOptimizer(model["params"], LRS)
        opt.exp_avg, opt.exp_avg_sq = model["exp_avg"], model["exp_avg_sq"]
        opt.grad_accum, opt.denom = model["accum"], model["denom"]
        opt.step_count = 500
        state["optimizer"] = opt
        if kind == "optimise":
            state.update(grads=model["grads"], grad2D=model["grad2D"], radii=model["radii"])
        else:
            count = int(_splits(model).sum())
            state.update(model=dict(opt.params), exp_avg=dict(opt.exp_avg), exp_avg_sq=dict(opt.exp_avg_sq),
                         accum=opt.grad_accum, denom=opt.denom, z=model["z"][:, :count].contiguous())
    else:
        raise ValueError(kind)
    return state


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind == "view":
        with torch.no_grad():
            color, radii, depth, alpha = state["rasterizer"](**state["inputs"])
        return {"color": color, "radii": radii, "depth": depth, "alpha": alpha}
    if kind == "train":
        inputs, images = state["inputs"], state["images"]
        color, radii, depth, alpha = state["rasterizer"](**inputs)
        value = loss.l1_loss(color, images["color"], clamp=True)
        if state["case"]["geometry"]:
            value = value + 0.05 * loss.l1_loss(depth, images["depth"]) + 0.05 * loss.l1_loss(alpha, images["alpha"])
        names = sorted(inputs)
        grads = torch.autograd.grad(value, [inputs[k] for k in names])
        return {"color": color, "radii": radii, "depth": depth, "alpha": alpha, "loss": value,
                "grads": dict(zip(names, grads))}
    if kind == "pose_step":
        problem, opt = state["problem"], state["optimizer"]
        xi = state["xi"].detach().requires_grad_(True)
        image = pose.render(problem, pose.pose_apply(xi, problem.xyz))
        value = pose.photometric_loss(image, problem.target, LAMBDA_DSSIM, fused=True)
        value.backward()
        opt.step(xi.grad)
        return {"image": image, "loss": value, "grad": xi.grad, "xi": opt.xi, "adam": opt.state}
    if kind == "pose_epoch":
        solver = state["solver"]
        solver.reset()
        solver.run(EPOCH)
        return {"xi": solver.xi, "adam": solver.adam, "color": solver.color}
    if kind == "loss":
        value = pose.photometric_loss(state["image"], state["target"], LAMBDA_DSSIM, fused=True)
        return {"loss": value, "grad": torch.autograd.grad(value, state["image"])[0]}
    if kind == "frame":
        points = pointcloud.depth_to_points(state["depth"], state["K"])
        xyz, rgb = pointcloud.voxel_down_sample(points, state["rgb"], state["voxel"])
        return {"points": points, "rgb": rgb, "gaussians": pointcloud.gaussians_from_points(xyz, rgb)}
    opt = state["optimizer"]
    if kind == "optimise":
        opt.step(state["grads"])
        opt.add_densification_stats(state["grad2D"], state["radii"])
        return {"params": opt.params, "exp_avg": opt.exp_avg, "exp_avg_sq": opt.exp_avg_sq, "accum": opt.grad_accum,
                "denom": opt.denom, "max_radii2D": opt.max_radii2D}
    # densification replaces the optimiser's arrays by new ones: the same model is handed to it again
    opt.params, opt.exp_avg, opt.exp_avg_sq = dict(state["model"]), dict(state["exp_avg"]), dict(state["exp_avg_sq"])
    opt.grad_accum, opt.denom = state["accum"], state["denom"]
    counts = opt.densify_and_prune(z=state["z"], **DENSIFY)
    return {"params": opt.params, "exp_avg": opt.exp_avg, "exp_avg_sq": opt.exp_avg_sq, "counts": counts}


def work(case):
    """Each input read once and each output written once. The rasteriser's operations depend on
    the view (how many Gaussians reach a pixel before it is opaque); counted here: the
    projection per Gaussian, and 30 Gaussians per pixel at 25 operations (75 with the
    backward)."""
    kind = case["kind"]

    def raster(n, pixels, floats, backward):
        flops = n * (300 + 6 * floats) + pixels * 30 * 25
        nbytes = 4 * n * floats + 4 * n + 20 * pixels
        if backward:
            nbytes += 4 * n * floats + 12 * n + 12 * pixels
            flops += n * (600 + 12 * floats) + pixels * 30 * 50
        return nbytes, flops

    if kind in ("view", "train"):
        floats = 13 if case.get("precomputed") else 11 + 3 * (case["sh_degree"] + 1) ** 2
        nbytes, flops = raster(case["n"], case["width"] * case["height"], floats, kind == "train")
        if case.get("geometry"):
            nbytes += 8 * case["width"] * case["height"]
    elif kind in ("pose_step", "pose_epoch"):
        specs = [(case["n"], case["width"], case["height"])] if kind == "pose_step" else \
            [s[:3] for s in _pose_specs(case, 0)]
        nbytes = flops = 0
        for n, width, height in specs:
            b, f = raster(n, width * height, 14, False)
            nbytes, flops = nbytes + b + 12 * width * height, flops + 3 * f
            if kind == "pose_step":
                flops += 3 * width * height * 450
        flops *= 1 if kind == "pose_step" else EPOCH
    elif kind == "loss":
        elements = 3 * case["width"] * case["height"]
        nbytes, flops = 12 * elements, 450 * elements
    elif kind == "frame":
        points = case["width"] * case["height"]
        nbytes, flops = points * (4 + 12 + 12 + 24 + 4 * 59), points * 600
    else:
        n = case["n"]
        nbytes = n * (59 * 4 * 7 + 4 * 13) if kind == "optimise" else n * (59 * 4 * 6)
        flops = n * 59 * (12 if kind == "optimise" else 1)
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------
# the same results in float64 PyTorch
# ---------------------------------------------------------------------------
def _rotation(q):
    r, x, y, z = q.unbind(1)
    return torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - r * z), 2 * (x * z + r * y),
                        2 * (x * y + r * z), 1 - 2 * (x * x + z * z), 2 * (y * z - r * x),
                        2 * (x * z - r * y), 2 * (y * z + r * x), 1 - 2 * (x * x + y * y)], 1).reshape(-1, 3, 3)


def _covariance(scales, rotations):
    m = _rotation(rotations) * scales[:, None, :]
    s = m @ m.transpose(1, 2)
    return torch.stack([s[:, 0, 0], s[:, 0, 1], s[:, 0, 2], s[:, 1, 1], s[:, 1, 2], s[:, 2, 2]], 1)


def _sh_colour(degree, sh, direction):
    x, y, z = direction.unbind(1)
    xx, yy, zz = x * x, y * y, z * z
    b = [torch.full_like(x, math.sqrt(1 / (4 * math.pi)))]
    if degree > 0:
        c = math.sqrt(3 / (4 * math.pi))
        b += [-c * y, c * z, -c * x]
    if degree > 1:
        c, c0 = math.sqrt(15 / (4 * math.pi)), math.sqrt(5 / (16 * math.pi))
        b += [c * x * y, -c * y * z, c0 * (2 * zz - xx - yy), -c * x * z, 0.5 * c * (xx - yy)]
    if degree > 2:
        c3, c2 = math.sqrt(35 / (32 * math.pi)), math.sqrt(105 / (4 * math.pi))
        c1, c0 = math.sqrt(21 / (32 * math.pi)), math.sqrt(7 / (16 * math.pi))
        b += [-c3 * y * (3 * xx - yy), c2 * x * y * z, -c1 * y * (4 * zz - xx - yy), c0 * z * (2 * zz - 3 * xx - 3 * yy),
              -c1 * x * (4 * zz - xx - yy), 0.5 * c2 * z * (xx - yy), -c3 * x * (xx - 3 * yy)]
    return (torch.stack(b, 1)[:, :, None] * sh).sum(1) + 0.5


class _Exact:
    """A view by the published 3DGS algorithm in float64: forward() gives (color, depth,
    alpha); backward(dcolor, ddepth, dalpha) the gradients of the given leaves."""
    TILE, BUDGET = 16, 1 << 25  # (instance, pixel) pairs evaluated at a time

    def __init__(self, cam, inputs, sh_degree):
        self.leaves, W, H = inputs, cam.width, cam.height
        self.W, self.H = W, H
        p, V, P = inputs["means3D"], cam.viewmatrix.double(), cam.projmatrix.double()
        ph = torch.cat([p, torch.ones_like(p[:, :1])], 1)
        t, hom = (ph @ V)[:, :3], ph @ P
        ndc = hom[:, :2] / (hom[:, 3:] + 1e-7) + inputs["means2D"][:, :2]
        xy = ((ndc + 1) * torch.tensor([W, H], dtype=F64, device=DEV) - 1) * 0.5
        cov = inputs["cov3D_precomp"] if "cov3D_precomp" in inputs else _covariance(inputs["scales"], inputs["rotations"])
        tz = t[:, 2]
        jac = []
        for axis, (size, tan) in enumerate(((W, cam.tanfovx), (H, cam.tanfovy))):
            f, lim = size / (2.0 * tan), 1.3 * tan
            ratio = (t[:, axis] / tz).detach()
            inside = (ratio >= -lim) & (ratio <= lim)
            ta = torch.where(inside, t[:, axis], ratio.clamp(-lim, lim) * tz.detach())
            jac.append((f / tz)[:, None] * V[:3, axis] + (-f * ta / (tz * tz))[:, None] * V[:3, 2])
        S = torch.stack([cov[:, 0], cov[:, 1], cov[:, 2], cov[:, 1], cov[:, 3], cov[:, 4], cov[:, 2], cov[:, 4],
                         cov[:, 5]], 1).reshape(-1, 3, 3)
        u, v = (S @ jac[0][:, :, None])[:, :, 0], (S @ jac[1][:, :, None])[:, :, 0]
        a, b, c = (jac[0] * u).sum(1) + 0.3, (jac[0] * v).sum(1), (jac[1] * v).sum(1) + 0.3
        det = a * c - b * b
        if "colors_precomp" in inputs:
            rgb = inputs["colors_precomp"]
        else:
            d = p - cam.campos.double()
            rgb = _sh_colour(sh_degree, inputs["shs"], d / d.norm(dim=1, keepdim=True)).clamp_min(0.0)
        self.graph = torch.cat([xy, torch.stack([c / det, -b / det, a / det], 1), inputs["opacities"].reshape(-1, 1), rgb,
                                tz[:, None]], 1)
        self.feat = self.graph.detach()
        with torch.no_grad():
            mid = 0.5 * (a + c)
            radius = torch.ceil(3.0 * torch.sqrt(mid + torch.sqrt((mid * mid - det).clamp_min(0.1))))
            grid = [-(-W // self.TILE), -(-H // self.TILE)]
            lo, hi = [], []
            for axis in range(2):
                lo.append(torch.trunc((xy[:, axis] - radius) / self.TILE).clamp(0, grid[axis]).long())
                hi.append(torch.trunc((xy[:, axis] + radius + self.TILE - 1) / self.TILE).clamp(0, grid[axis]).long())
            w, h = hi[0] - lo[0], hi[1] - lo[1]
            touched = torch.where((tz > 0.2) & (det != 0), w * h, torch.zeros_like(w))
            order = torch.argsort(tz, stable=True)
            gid = torch.repeat_interleave(order, touched[order])
            first = torch.cumsum(touched[order], 0) - touched[order]
            j = torch.arange(gid.numel(), device=DEV) - torch.repeat_interleave(first, touched[order])
            tile = (lo[1][gid] + j // w[gid]) * grid[0] + lo[0][gid] + j % w[gid]
            tile, by = torch.sort(tile, stable=True)
            self.gid = gid[by]
            count = torch.bincount(tile, minlength=grid[0] * grid[1])
            self.start, self.count, self.grid = torch.cumsum(count, 0) - count, count, grid
            sizes, self.by_size = torch.sort(count, descending=True)
            self.sizes = sizes.tolist()

    def _chunks(self):
        k = 0
        while k < len(self.sizes):
            longest = max(self.sizes[k], 1)
            tiles = self.by_size[k:k + max(1, self.BUDGET // (longest * self.TILE ** 2))]
            k += tiles.numel()
            at = torch.arange(longest, device=DEV)[None, :]
            there = at < self.count[tiles][:, None]
            gid = self.gid[(self.start[tiles][:, None] + at).clamp_max(max(self.gid.numel() - 1, 0))] if self.gid.numel() \
                else torch.zeros_like(at).expand(tiles.numel(), 1)
            pix = torch.arange(self.TILE ** 2, device=DEV)
            x = (tiles % self.grid[0])[:, None] * self.TILE + pix % self.TILE
            y = (tiles // self.grid[0])[:, None] * self.TILE + pix // self.TILE
            yield gid, there, x, y, (x < self.W) & (y < self.H)

    def _tiles(self, feat, gid, there, x, y):
        """color [B,P,3], depth [B,P] and alpha [B,P] of a chunk of tiles."""
        f = feat[gid]
        dx, dy = f[:, :, None, 0] - x[:, None, :], f[:, :, None, 1] - y[:, None, :]
        power = -0.5 * (f[:, :, None, 2] * dx * dx + f[:, :, None, 4] * dy * dy) - f[:, :, None, 3] * dx * dy
        raw = f[:, :, None, 5] * torch.exp(power.clamp_max(0.0))
        alpha = raw - (raw - 0.99).clamp_min(0.0).detach()
        alpha = alpha * ((power <= 0) & (alpha >= 1.0 / 255.0) & there[:, :, None])
        after = torch.cumsum(torch.log1p(-alpha.detach()), 1)
        alpha = alpha * (after >= math.log(1e-4))
        log_t = torch.log1p(-alpha)
        after = torch.cumsum(log_t, 1)
        weight = alpha * torch.exp(after - log_t)
        return torch.einsum("blp,blc->bpc", weight, f[:, :, 6:10]), 1.0 - torch.exp(after[:, -1])

    @torch.no_grad()
    def forward(self):
        out = torch.zeros(5, self.H * self.W, dtype=F64, device=DEV)
        for gid, there, x, y, inside in self._chunks():
            rgbd, alpha = self._tiles(self.feat, gid, there, x, y)
            out[:, (y * self.W + x)[inside]] = torch.cat([rgbd, alpha[:, :, None]], 2)[inside].t()
        out = out.reshape(5, self.H, self.W)
        return out[:3], out[3:4], out[4:5]

    def backward(self, dcolor, ddepth=None, dalpha=None):
        total = torch.zeros_like(self.feat)
        zero = torch.zeros(1, self.H, self.W, dtype=F64, device=DEV)
        image = torch.cat([dcolor, zero if ddepth is None else ddepth, zero if dalpha is None else dalpha]).reshape(5, -1)
        for gid, there, x, y, inside in self._chunks():
            feat = self.feat.clone().requires_grad_(True)
            rgbd, alpha = self._tiles(feat, gid, there, x, y)
            g = image[:, (y * self.W + x).clamp_max(self.H * self.W - 1)].permute(1, 2, 0) * inside[:, :, None]
            total += torch.autograd.grad([rgbd, alpha], feat, [g[:, :, :4], g[:, :, 4]])[0]
        names = [k for k in sorted(self.leaves) if self.leaves[k].requires_grad]
        return dict(zip(names, torch.autograd.grad(self.graph, [self.leaves[k] for k in names], total)))


def _ssim(x, y):
    w = torch.exp(-((torch.arange(11, dtype=F64, device=DEV) - 5) ** 2) / (2 * 1.5 ** 2))
    w = w / w.sum()

    def blur(a):
        a = torch.nn.functional.conv2d(a[:, None], w.reshape(1, 1, 1, 11), padding=(0, 5))
        return torch.nn.functional.conv2d(a, w.reshape(1, 1, 11, 1), padding=(5, 0))[:, 0]

    m1, m2 = blur(x), blur(y)
    s11, s22, s12 = blur(x * x) - m1 * m1, blur(y * y) - m2 * m2, blur(x * y) - m1 * m2
    c1, c2 = 0.01 ** 2, 0.03 ** 2
    return (((2 * m1 * m2 + c1) * (2 * s12 + c2)) / ((m1 * m1 + m2 * m2 + c1) * (s11 + s22 + c2))).mean()


def _photometric(image, target, weight):
    c = image.clamp(0, 1)
    value = (1 - weight) * (c - target).abs().mean()
    return value + weight * (1 - _ssim(c, target)) if weight else value


def _posed(xi, xyz):
    """exp(xi) applied to positions, xi = (rho, phi)."""
    rho, phi = xi[:3], xi[3:]
    zero = torch.zeros((), dtype=F64, device=DEV)
    hat = torch.stack([zero, -phi[2], phi[1], phi[2], zero, -phi[0], -phi[1], phi[0], zero]).reshape(3, 3)
    eye = torch.eye(3, dtype=F64, device=DEV)
    rot, left, term = eye, eye, eye
    for k in range(1, 16):  # the exponential series and that of its left Jacobian
        term = term @ hat / k
        rot, left = rot + term, left + term / (k + 1)
    return xyz @ rot.t() + left @ rho


def _pose_gradient(problem, cam, xi, weight):
    """(image, loss, dL/dxi) of one pose iteration."""
    xi = xi.detach().requires_grad_(True)
    means = _posed(xi, problem.xyz.double())
    leaf = means.detach().requires_grad_(True)
    inputs = {"means3D": leaf, "means2D": torch.zeros_like(leaf).detach(), "opacities": problem.opacities.double(),
              "shs": problem.shs.double(), "scales": problem.scales.double(), "rotations": problem.rotations.double()}
    view = _Exact(cam, inputs, problem.sh_degree)
    image = view.forward()[0].requires_grad_(True)
    value = _photometric(image, problem.target.double(), weight)
    d_means = view.backward(torch.autograd.grad(value, image)[0])["means3D"]
    return image.detach(), value.detach(), torch.autograd.grad(means, xi, d_means)[0]


def _adam6(xi, m, v, grad, step):
    m = 0.9 * m + 0.1 * grad
    v = 0.999 * v + 0.001 * grad * grad
    return xi - 1e-3 / (1 - 0.9 ** step) * m / (v.sqrt() / math.sqrt(1 - 0.999 ** step) + 1e-15), m, v


def _adam_row(m, v, step):
    tail = torch.tensor([float(step), 0.0, 0.0, 0.0], dtype=F64, device=DEV)
    return torch.cat([m, v, tail])[None]


def _exact_raster(case, seed):
    inputs, images, cam = _cloud(case, seed)
    train = case["kind"] == "train"
    leaves = {k: v.double().requires_grad_(train) for k, v in inputs.items()}
    leaves["means2D"] = torch.zeros_like(leaves["means3D"]).detach().requires_grad_(train)
    with torch.set_grad_enabled(train):
        view = _Exact(cam, leaves, case["sh_degree"])
    color, depth, alpha = view.forward()
    out = {"color": color, "radii": None, "depth": depth, "alpha": alpha}
    if train:
        parts = [x.clone().requires_grad_(True) for x in (color, depth, alpha)]
        value = (parts[0].clamp(0, 1) - images["color"].double()).abs().mean()
        if case["geometry"]:
            value = value + 0.05 * (parts[1] - images["depth"].double()).abs().mean() + \
                0.05 * (parts[2] - images["alpha"].double()).abs().mean()
        out["loss"] = value.detach()
        out["grads"] = view.backward(*torch.autograd.grad(value, parts, allow_unused=True))
    return out


def _nearest3(points):
    """Mean squared distance of each point to its three nearest others."""
    out = torch.empty(points.shape[0], dtype=F64, device=DEV)
    rows = max(1, (1 << 28) // points.shape[0])
    for k in range(0, points.shape[0], rows):
        q = points[k:k + rows]
        d = sum((q[:, None, a] - points[None, :, a]) ** 2 for a in range(3))
        d[torch.arange(q.shape[0], device=DEV), torch.arange(k, k + q.shape[0], device=DEV)] = math.inf
        out[k:k + rows] = torch.topk(d, 3, dim=1, largest=False).values.mean(1)
    return out


def _exact_frame(case, seed):
    depth, rgb, K, voxel = _frame_inputs(case, seed)
    v, u = torch.meshgrid(torch.arange(case["height"], device=DEV), torch.arange(case["width"], device=DEV), indexing="ij")

    def unproject(d, dtype):
        fx, fy, cx, cy = (torch.tensor(x, dtype=dtype, device=DEV) for x in (K[0][0], K[1][1], K[0][2], K[1][2]))
        return torch.stack([(u.to(dtype) - cx) / fx * d, (v.to(dtype) - cy) / fy * d, d], -1).reshape(-1, 3)

    p = unproject(depth, torch.float32).double()  # the grid is laid over the points as the program holds them
    cell = torch.floor((p - (p.min(0).values - 0.5 * voxel)) / voxel).long()
    dim = cell.max(0).values + 1
    _, inverse, count = torch.unique((cell[:, 0] * dim[1] + cell[:, 1]) * dim[2] + cell[:, 2], return_inverse=True,
                                     return_counts=True)
    n = count.numel()
    if n > 250_000:
        return None
    mean = torch.zeros(n, 6, dtype=F64, device=DEV).index_add_(0, inverse, torch.cat([p, rgb.double()], 1))
    mean /= count[:, None]
    xyz, rgb = mean[:, :3], mean[:, 3:]
    rotation = torch.zeros(n, 4, dtype=F64, device=DEV)
    rotation[:, 0] = 1
    scaling = torch.log(torch.sqrt(_nearest3(xyz).clamp_min(1e-7)))[:, None].repeat(1, 3)
    return {"points": unproject(depth.double(), F64), "rgb": rgb, "gaussians": {
        "xyz": xyz, "features_dc": rgb[:, None, :], "features_rest": torch.zeros(n, 15, 3, dtype=F64, device=DEV),
        "scaling": scaling, "rotation": rotation,
        "opacity": torch.full((n, 1), math.log(0.1 / 0.9), dtype=F64, device=DEV)}}


def _exact_optimise(case, seed):
    model = _model(case, seed)
    out = {"params": {}, "exp_avg": {}, "exp_avg_sq": {}}
    for k in LRS:
        g = model["grads"][k].double()
        m = 0.9 * model["exp_avg"][k].double() + 0.1 * g
        v = 0.999 * model["exp_avg_sq"][k].double() + 0.001 * g * g
        denom = v.sqrt() / math.sqrt(1 - 0.999 ** 501) + 1e-15
        out["params"][k] = model["params"][k].double() - LRS[k] / (1 - 0.9 ** 501) * m / denom
        out["exp_avg"][k], out["exp_avg_sq"][k] = m, v
    seen = model["radii"] > 0
    out["accum"] = model["accum"].double() + seen * model["grad2D"][:, :2].double().norm(dim=1)
    out["denom"] = model["denom"].double() + seen
    out["max_radii2D"] = model["radii"].double()
    return out


def _exact_densify(case, seed):
    model = _model(case, seed)
    p = {k: v.double() for k, v in model["params"].items()}
    split = _splits(model)
    grad = (model["accum"].double() / model["denom"].double()).nan_to_num(0.0)
    biggest = p["scaling"].exp().max(1).values
    low = torch.sigmoid(p["opacity"][:, 0]) < DENSIFY["min_opacity"]
    big = biggest > 0.1 * DENSIFY["extent"]
    clone = (grad >= DENSIFY["max_grad"]) & ~split
    child = split & ~(low | (biggest / 1.6 > 0.1 * DENSIFY["extent"]))
    keep = ~split & ~(low | big)
    source = torch.cat([torch.nonzero(x)[:, 0] for x in (keep, clone & ~(low | big), child, child)])
    fresh = torch.arange(source.numel(), device=DEV) >= int(keep.sum())
    out = {"params": {k: v[source] for k, v in p.items()}, "counts": {}}
    for name in ("exp_avg", "exp_avg_sq"):
        out[name] = {k: v.double()[source] * ~fresh.reshape(-1, *[1] * (v.dim() - 1)) for k, v in model[name].items()}
    at = torch.nonzero(child)[:, 0]
    rank = (torch.cumsum(split, 0) - 1)[at]
    q = p["rotation"][at]
    rot = _rotation(q / q.norm(dim=1, keepdim=True))
    z = model["z"][:, :int(split.sum())].double()
    rows = 2 * at.numel()
    moved = [p["xyz"][at] + (rot @ (p["scaling"][at].exp() * z[c][rank])[:, :, None])[:, :, 0] for c in range(2)]
    out["params"]["xyz"][source.numel() - rows:] = torch.cat(moved)
    out["params"]["scaling"][source.numel() - rows:] = (p["scaling"][at] - math.log(1.6)).repeat(2, 1)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("view", "train"):
        return _exact_raster(case, seed)
    if kind == "pose_step":
        problem, cam = _pose_inputs(case["n"], case["width"], case["height"], seed)
        xi = _randn(_gen(int(seed) + 77), 6, std=0.004).double()
        image, value, grad = _pose_gradient(problem, cam, xi, LAMBDA_DSSIM)
        zero = torch.zeros(6, dtype=F64, device=DEV)
        moved, m, v = _adam6(xi, zero, zero, grad, 1)
        return {"image": image, "loss": value, "grad": grad, "xi": moved, "adam": _adam_row(m, v, 1)}
    if kind == "pose_epoch":
        if case["solves"] > 1:
            return None  # minutes of dense float64 rendering
        problem, cam = _pose_inputs(*_pose_specs(case, seed)[0])
        xi = m = v = torch.zeros(6, dtype=F64, device=DEV)
        for step in range(1, EPOCH + 1):
            image, _, grad = _pose_gradient(problem, cam, xi, 0.0)
            xi, m, v = _adam6(xi, m, v, grad, step)
        return {"xi": xi[None], "adam": _adam_row(m, v, EPOCH), "color": image.reshape(-1)}
    if kind == "loss":
        g = _gen(seed)
        target = _rand(g, 3, case["height"], case["width"])
        image = (target + _randn(g, *target.shape, std=0.1)).double().requires_grad_(True)
        value = _photometric(image, target.double(), LAMBDA_DSSIM)
        return {"loss": value.detach(), "grad": torch.autograd.grad(value, image)[0]}
    if kind == "frame":
        return _exact_frame(case, seed)
    return _exact_optimise(case, seed) if kind == "optimise" else _exact_densify(case, seed)
