"""Workloads of the point-splatting rasterizer: what a training program and a viewer ask of it in one pass.

Two kinds of pass, both through PointRenderModule:
  render  the module in eval mode: views of a scene -> image pyramids (viewer frames, evaluation batches)
  train   the module in train mode, the gradient of the pyramid that the network behind the rasterizer hands back,
          and MyAdam over all point parameters

Scenes are drawn on the GPU from a seed with the value distributions of trips_b200/scenes.py; points come in random order.
"""
import math

import numpy as np
import torch

from trips_b200.modules import IntrinsicsModule, NeuralPointCloudCuda, NeuralPointTexture, NeuralScene, PointRenderModule, PoseModule
from trips_b200.optim import MyAdam
from trips_b200.renderer import PointRendererCache, ReducedImageInfo, RenderParams
from trips_b200.scenes import layer_sizes, look_at_pose, num_pyramid_pixels


def _case(kind, scene, points, width, height, layers, views, keep=16, channels=4, raw=False, cameras=False):
    """scene: which distribution of points and cameras.  keep: fragments kept per pixel.  raw: confidences and descriptors
    are the raw parameters (sigmoid and abs inside the rasterizer).  cameras: pose and intrinsics gradients as well."""
    return {"kind": kind, "scene": scene, "points": points, "width": width, "height": height, "layers": layers, "views": views,
            "keep": keep, "channels": channels, "raw": raw, "cameras": cameras}


def listed():
    cases = {
        # the smallest step anybody runs (a toy or a unit test): launches and host time
        "train_4k_96x64": _case("train", "cube", 4_000, 96, 64, 4, 2),
        # a preview of a small object
        "render_200k_640x480": _case("render", "sphere", 200_000, 640, 480, 4, 1, keep=8),
        # one frame of a viewer
        "render_6m_1080p_frame": _case("render", "surfaces", 6_000_000, 1920, 1080, 8, 1),
        # an evaluation pass over the test views of a scene; the largest call
        "render_10m_1080p_64_views": _case("render", "surfaces", 10_000_000, 1920, 1080, 8, 64),
        # training on crops of odd sizes, raw parameters, cameras refined with the points
        "train_1m_crops_cameras": _case("train", "surfaces", 1_234_567, 511, 509, 5, 4, raw=True, cameras=True),
        # wider descriptors on a ragged image
        "train_800k_8_channels": _case("train", "surfaces", 777_777, 1001, 563, 6, 2, channels=8),
        # a room at 720p
        "train_2m_720p": _case("train", "surfaces", 2_000_000, 1280, 720, 6, 4),
        # one view per step, as a single image is fitted or a batch is split over many GPUs
        "train_6m_1080p_1_view": _case("train", "surfaces", 6_000_000, 1920, 1080, 8, 1, raw=True),
        # the benchmark's training step
        "train_6m_1080p": _case("train", "surfaces", 6_000_000, 1920, 1080, 8, 8),
        # a large outdoor scene: ground and clusters, uneven density, heavy-tailed sizes
        "train_20m_1440p": _case("train", "ground", 20_000_000, 2560, 1440, 8, 2),
        # an object far away: all points inside 64x64 pixels, lists of thousands of fragments
        "train_3m_crowded": _case("train", "blob", 3_000_000, 1920, 1080, 8, 4),
    }
    return [dict(c, name=n) for n, c in cases.items()]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["train", "train", "render"])
    scene = rng.choice(["surfaces", "surfaces", "surfaces", "ground", "sphere", "cube", "blob"])
    width = log_int(64, 2560)
    height = max(48, min(1440, int(width * rng.uniform(0.5, 1.1))))
    points = log_int(2_000, {"cube": 300_000, "sphere": 2_000_000, "blob": 2_000_000}.get(scene, 12_000_000))
    most = min(12, 48_000_000 // points, 16_000_000 // (width * height))  # no more than the largest listed cases
    views = rng.randint(1, max(1, most))
    deepest = max(2, min(8, int(math.log2(min(width, height))) - 1))
    layers = rng.randint(max(1, deepest - 3), deepest)
    return _case(kind, scene, points, width, height, layers, views, keep=rng.choice([16, 16, 8]), channels=rng.choice([4, 4, 4, 3, 8]),
                 raw=rng.random() < 0.5, cameras=kind == "train" and rng.random() < 0.25)


def _points(case, gen, dev):
    """Positions [N, 3] (double), world-space sizes [N], and the scene's cameras: (eye, target) per view and focal length."""
    n, views = case["points"], case["views"]

    def uniform(lo, hi, *shape):
        return torch.rand(shape, generator=gen, device=dev, dtype=torch.float64) * (hi - lo) + lo

    def normal(*shape):
        return torch.randn(shape, generator=gen, device=dev, dtype=torch.float64)

    def log_uniform(lo, hi):
        return torch.exp(uniform(math.log(lo), math.log(hi), n))

    def choose(k):
        return torch.randint(0, k, (n,), generator=gen, device=dev)

    turn = float(uniform(0, 2 * math.pi, 1))
    ring = [turn + 2 * math.pi * i / views for i in range(views)]

    def around(radius, y, target_y=0.0):
        return [((radius * math.cos(a), y, radius * math.sin(a)), (0.0, target_y, 0.0)) for a in ring]

    def unit(v):
        return v / v.norm(dim=1, keepdim=True)

    if case["scene"] == "cube":
        return uniform(-1.5, 1.5, n, 3), log_uniform(5e-3, 0.4), around(4.0, -0.5), 0.94 * case["width"]
    if case["scene"] == "sphere":
        return unit(normal(n, 3)) + 0.01 * normal(n, 3), log_uniform(1e-3, 1e-1), around(3.0, 0.0), 0.78 * case["width"]
    if case["scene"] == "blob":
        far = [((0.0, 0.0, -30.0), (0.0, 0.0, 0.0))] * views
        return uniform(-0.6, 0.6, n, 3), log_uniform(1e-3, 5e-2), far, 0.78 * case["width"]
    if case["scene"] == "ground":
        flat = torch.stack([uniform(-100, 100, n), 0.02 * normal(n), uniform(-100, 100, n)], 1)
        centre = torch.stack([uniform(-90, 90, 48), uniform(-6, -0.5, 48), uniform(-90, 90, 48)], 1)
        cluster = centre[choose(48)] + 1.5 * normal(n, 3)
        sizes = 2e-3 * uniform(1e-9, 1, n).pow(-1 / 1.5)  # Pareto(1.5)
        return torch.where(uniform(0, 1, n, 1) < 0.7, flat, cluster), sizes.clamp(max=2.0), around(60.0, -1.7, -1.0), 0.78 * case["width"]
    # random square patches and spheres in a box; cameras on a ring, or scattered around the box for an evaluation batch
    count, box = 64, 20.0
    centre, extent, normals = uniform(-0.4 * box, 0.4 * box, count, 3), uniform(0.1 * box, 0.35 * box, count), unit(normal(count, 3))
    a = unit(torch.linalg.cross(normals, torch.tensor([[0.3, 0.5, 0.8]], device=dev, dtype=torch.float64).expand(count, 3)))
    b = torch.linalg.cross(normals, a)
    which = choose(count)
    patch = centre[which] + (uniform(-1, 1, n, 1) * a[which] + uniform(-1, 1, n, 1) * b[which]) * extent[which, None]
    ball = centre[which] + unit(normal(n, 3)) * (0.5 * extent[which, None])
    flat = uniform(0, 1, count) < 0.5
    pts = torch.where(flat[which, None], patch, ball).clamp(-0.5 * box, 0.5 * box)
    if views <= 8:
        cameras = around(13.0, -3.0)
    else:
        eyes = (unit(normal(views, 3)) * uniform(11.0, 16.0, views, 1)).tolist()
        cameras = list(zip(eyes, uniform(-3.0, 3.0, views, 3).tolist()))
    return pts, log_uniform(1e-3, 5e-2), cameras, 0.78 * case["width"]


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    n, c, views, w, h = (case[k] for k in ("points", "channels", "views", "width", "height"))
    pts, sizes, cameras, focal = _points(case, gen, dev)
    position = torch.cat([pts, sizes[:, None]], 1).float()
    size_raw = torch.where(sizes > 20, sizes, torch.log(torch.expm1(sizes.clamp(max=20)))).float()
    del pts, sizes
    texture = torch.rand((c, n), generator=gen, device=dev)
    confidence = torch.rand((1, n), generator=gen, device=dev)
    if case["raw"]:
        texture = texture * torch.where(torch.rand((c, n), generator=gen, device=dev) < 0.1, -1.0, 1.0)
        confidence = torch.logit(confidence.clamp(1e-4, 1 - 1e-4)) / 10.0
    poses = torch.from_numpy(np.stack([look_at_pose(eye, target) for eye, target in cameras])).to(dev)
    intrinsics = torch.zeros((views, 13), device=dev)
    intrinsics[:, 0:2] = focal
    intrinsics[:, 2] = w / 2
    intrinsics[:, 3] = h / 2
    scene = NeuralScene(NeuralPointCloudCuda(position, point_size_raw=size_raw),
                        NeuralPointTexture(c, n, texture=texture, confidence_raw=confidence, device=dev), PoseModule(poses),
                        IntrinsicsModule(intrinsics))
    params = RenderParams(num_texture_channels=c, k_keep=case["keep"], confidence_is_raw=case["raw"], texture_abs=case["raw"])
    module = PointRenderModule(params, num_layers=case["layers"])
    module.cache = PointRendererCache(dev)
    images = [ReducedImageInfo(w=w, h=h, image_index=v, camera_index=v) for v in range(views)]
    state = {"scene": scene, "module": module, "images": images}
    if case["kind"] == "render":
        module.eval()
        return state
    module.train()
    if case["cameras"]:
        scene.poses.tangent_poses.requires_grad_(True)
        scene.intrinsics.intrinsics.requires_grad_(True)
    # what an L1 loss behind the rasterizer gives: +-1 / number of values
    numel = c * num_pyramid_pixels(w, h, case["layers"])
    state["image_grads"] = [(torch.randint(0, 2, (views, c, lh, lw), generator=gen, device=dev).float() * 2 - 1) / numel
                            for lw, lh in layer_sizes(w, h, case["layers"])]
    cloud, tex = scene.point_cloud_cuda, scene.texture
    state["weights"] = [tex.texture_raw, tex.confidence_raw, cloud.t_position, cloud.t_point_size, tex.background_color_raw]
    # the rate at the end of a decaying schedule: many passes on one state leave the scene as it is
    state["optimizer"] = MyAdam(state["weights"], lr=1e-7, betas=(0.9, 0.999), cache=module.cache)
    return state


def run(state):
    scene, module = state["scene"], state["module"]
    if not module.training:
        with torch.no_grad():
            return {"pyramid": module(scene, state["images"])[0]}
    optimizer, weights = state["optimizer"], state["weights"]
    optimizer.zero_grad(set_to_none=True)
    cameras = [p for p in (scene.poses.tangent_poses, scene.intrinsics.intrinsics) if p.requires_grad]
    for p in cameras:
        p.grad = None
    pyramid = module(scene, state["images"])[0]
    torch.autograd.backward(pyramid, state["image_grads"])
    optimizer.step()
    return {"pyramid": [p.detach() for p in pyramid], "gradients": [p.grad for p in weights + cameras], "weights": [p.detach() for p in weights]}


def work(case):
    n, c = case["points"], case["channels"]
    pyramid = 4 * c * num_pyramid_pixels(case["width"], case["height"], case["layers"]) * case["views"]
    scene = n * (16 + 4 + 4 + 4 * c + 4)  # position, size, index, descriptor, confidence
    if case["kind"] == "render":
        return {"bytes": scene + pyramid, "flops": 0}
    # the pyramid out and its gradient in; gradients of position, size, descriptor and confidence out; MyAdam reads them and
    # the weights again, and reads and writes two moments and a step counter
    values = n * (c + 6)
    return {"bytes": scene + 2 * pyramid + 4 * values + (4 + 8 + 24) * values, "flops": 0}


def tolerance(case):
    # Rendered twice the pyramid is the same to the bit; its sums of 16 products in another order move it by 1e-7.  Gradients
    # are sums of thousands of 32-bit terms of both signs, added by atomics in any order: 1e-7 apart between two runs
    # (single values up to 1e-5 of the tensor's root mean square), several times that with another recurrence over a list.
    return {"rel": 1e-6} if case["kind"] == "render" else {"rel": 2e-6, "max": 2e-4}
