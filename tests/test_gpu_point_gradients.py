"""The gather of per-entry gradient rows into per-point gradients (point_grad_kernel) at the sizes where it can go wrong:
view counts around the rows requested at a time (4) and above the cameras held in shared memory (32), clouds that take the
aggregating binning kernels (they note the entry of a point in their own code), a dropout mask, and points that change or
are gone by the time of the backward pass (their gradients are those of the points that were rendered).

Gradients are fp32 sums over fragments of both signs in another order than the oracle's: the bound of 1e-4 on elements
above 1 % of the tensor's largest magnitude is the one of the parity tests (thousands of terms x 6e-8)."""
import numpy as np
import pytest

import oracle
from trips_b200 import scenes
from util import gpu_render, oracle_frames, rel_err

pytestmark = pytest.mark.gpu


def _check(s, dropout=None, between=None, **kw):
    import torch
    if dropout is None:
        sa, op, frames = oracle_frames(s, train=True, **kw)
    else:
        op = oracle.make_params(s.num_layers, s.k_keep, True, **kw)
        sa = [oracle.SceneArrays.from_scene(s, dropout=mask) for mask in dropout]
        frames = [oracle.forward(a, oracle.make_view(s.width, s.height, s.poses[b], s.intrinsics[b]), op) for b, a in enumerate(sa)]
    ns, info, blend = gpu_render(s, train=True, **kw)
    params = dict(texture=ns.texture.texture_raw, confidence=ns.texture.confidence_raw, position=ns.point_cloud_cuda.t_position,
                  point_size=ns.point_cloud_cuda.t_point_size)
    for t in params.values():
        t.requires_grad_(True)
    grads = [scenes.target_gradient(s, b) for b in range(s.n_views)]
    sizes = scenes.layer_sizes(s.width, s.height, s.num_layers)

    def backward():
        outs = blend(info)
        loss, base = 0, 0
        for l, (w, h) in enumerate(sizes):
            g = np.stack([grads[b][s.channels * base:s.channels * (base + w * h)].reshape(s.channels, h, w) for b in range(s.n_views)])
            loss = loss + (outs[l] * torch.from_numpy(g).cuda()).sum()
            base += w * h
        if between is not None:
            between(info, ns.point_cloud_cuda)
        loss.backward()
        torch.cuda.synchronize()
        assert info.cache.last_status() == 0
        got = {k: t.grad.cpu().numpy().copy() for k, t in params.items()}
        for t in params.values():
            t.grad = None
        return got

    if dropout is not None:
        info.cache.dropout_points = torch.from_numpy(dropout).cuda()
    ref = {k: 0.0 for k in params}
    for b, f in enumerate(frames):
        r = f.backward(grads[b])
        for k in ref:
            ref[k] = ref[k] + r[k]
    for call in range(2 if between is None else 1):  # a sized call, then one in the steady state
        got = backward()
        for k in ref:
            assert rel_err(got[k].reshape(ref[k].shape), ref[k]) <= 1e-4, f"{k}, call {call}"
    return got


@pytest.mark.parametrize("n_views", [1, 3, 4, 5, 33])
def test_view_counts(oracle_lib, cuda_lib, n_views):
    _check(scenes.tiny(seed=60 + n_views, n_points=1531, n_views=n_views, width=61, height=43, num_layers=3))


@pytest.mark.parametrize("n_views", [2, 17])
def test_crowded_cloud(oracle_lib, cuda_lib, n_views):
    s = scenes.tiny(seed=80 + n_views, n_points=12000, n_views=n_views, width=64, height=48, num_layers=3)
    s.position[:, :3] *= 0.02  # all points inside a few pixels: more than 4096 in one screen tile
    _check(s)


@pytest.mark.parametrize("crowded", [False, True])
def test_dropout_mask(oracle_lib, cuda_lib, crowded):
    """Points dropped in some views, and 30 % of them in all: those receive nothing (the oracle's gradients are exactly 0)."""
    n = 12000 if crowded else 3000
    s = scenes.tiny(seed=90, n_points=n, n_views=3)
    if crowded:
        s.position[:, :3] *= 0.02
    rng = np.random.default_rng(1)
    mask = (rng.random((3, n)) < 0.5) | (rng.random(n) < 0.2)
    got = _check(s, dropout=mask.astype(np.float32))
    hidden = mask.all(axis=0)
    assert not got["position"][hidden].any() and not got["point_size"].reshape(-1)[hidden].any()
    assert not got["texture"][:, hidden].any() and not got["confidence"].reshape(-1)[hidden].any()


def _move(info, cloud):
    import torch
    with torch.no_grad():
        cloud.t_position[:, :3] += 0.3 * torch.randn_like(cloud.t_position[:, :3])
        cloud.t_point_size -= 1.0


def _take_away(info, cloud):
    with_points = info.cache._scene_struct

    def without_points(*args):
        scene = with_points(*args)
        scene.position = scene.point_size = None
        return scene

    info.cache._scene_struct = without_points


@pytest.mark.parametrize("between", [_move, _take_away])
@pytest.mark.parametrize("crowded", [False, True])
@pytest.mark.parametrize("n_views", [2, 17])
def test_points_are_those_of_the_forward_pass(oracle_lib, cuda_lib, between, crowded, n_views):
    s = scenes.tiny(seed=95, n_points=12000 if crowded else 1500, n_views=n_views, width=64, height=48, num_layers=3)
    if crowded:
        s.position[:, :3] *= 0.02
    _check(s, between=between)


@pytest.mark.parametrize("indexed", [False, True])
def test_entry_table_in_groups_of_views(cuda_lib, indexed):
    """11 M points x 100 views: the table of a point's entries would exceed its limit of 4 GB and is filled for 97 views at a time.
    The gradients are those of two calls with half of the views each, whose tables hold all of theirs."""
    import torch
    n, shown = 11_000_000, 4000
    s = scenes.tiny(seed=96, n_points=n, n_views=100, width=61, height=43, num_layers=3)
    s.position[shown // 2:n - shown // 2, 1] += 1000.0  # out of every view
    index = np.random.default_rng(3).permutation(n).astype(np.int32) if indexed else None
    ns, info, blend = gpu_render(s, train=True, index=index)
    params = dict(texture=ns.texture.texture_raw, confidence=ns.texture.confidence_raw, position=ns.point_cloud_cuda.t_position,
                  point_size=ns.point_cloud_cuda.t_point_size)
    for t in params.values():
        t.requires_grad_(True)
    images, gen = info.images, torch.Generator(device="cuda")
    gen.manual_seed(1)
    targets = [torch.randn((100, s.channels, h, w), generator=gen, device="cuda") for w, h in scenes.layer_sizes(s.width, s.height, s.num_layers)]

    def gradients(first, last):
        info.images = images[first:last]
        torch.autograd.backward(blend(info), [t[first:last] for t in targets])
        assert info.cache.last_status() == 0
        got = {k: t.grad.double() for k, t in params.items()}
        for t in params.values():
            t.grad = None
        return got

    whole, a, b = gradients(0, 100), gradients(0, 50), gradients(50, 100)
    for k in params:
        ref = a[k] + b[k]
        scale = ref.abs().max()
        assert scale > 0 and float(((whole[k] - ref).abs() / ref.abs().clamp(min=1e-2 * scale)).max()) <= 1e-4, k
