"""Selection of the nearest fragments where the per-pixel sort can go wrong: list lengths around its chunks of 16 (the
shorter networks for 8 and 12, the comparators for up to 4), many fragments of the same depth inside and across the end of the selection, and lists around
the length at which a block of its own pre-selects them.  Kept points, their order and the pyramid must be the oracle's:
ids bit for bit, alphas and colours to 1e-5 (16 products in 32 bits, 16 x 6e-8)."""
import ctypes as C

import numpy as np
import pytest

from trips_b200 import scenes
from util import gpu_render, oracle_frames, rel_err

pytestmark = pytest.mark.gpu


def _check(s, views=None, min_length=0):
    sa, op, frames = oracle_frames(s, train=True, views=views)
    ns, info, blend = gpu_render(s, train=True)
    outs = blend(info)
    assert info.cache.last_status() == 0 and info.cache.stats()["max_list_length"] >= min_length
    for b, f in zip(range(s.n_views) if views is None else views, frames):
        nrec, pid, alpha = info.cache.debug_records(b, f.P)
        onrec, opid, oalpha = f.records()
        assert np.array_equal(nrec, onrec)
        assert np.array_equal(pid, opid)
        assert rel_err(alpha, oalpha, floor=1e-6) <= 1e-5
        for l, ref in enumerate(f.pyramid()):
            got = outs[l][b].detach().cpu().numpy()
            assert np.max(np.abs(got - ref) / np.maximum(np.abs(ref), 1e-3)) <= 1e-5
    return info


def _stack(n, copies, k_keep, seed):
    """`n` distinct points, `copies` of each (ids i, i + n, ...): every copy has the same depth on the same pixels."""
    s = scenes.tiny(seed=seed, n_points=n * copies, width=72, height=40, num_layers=3, k_keep=k_keep, n_views=2)
    for c in range(1, copies):
        s.position[c * n:(c + 1) * n] = s.position[:n]
        s.point_size[c * n:(c + 1) * n] = s.point_size[:n]
    s.confidence[:] = np.minimum(s.confidence, 0.1)  # the transmittance stays above the cut-off for all kept fragments
    return s


@pytest.mark.parametrize("k_keep", [1, 8, 16])
@pytest.mark.parametrize("n,copies", [(40, 1), (12, 2), (12, 3), (12, 4), (12, 5), (12, 8), (12, 9), (12, 16), (12, 17), (200, 15), (12, 33), (300, 20), (3, 512), (3, 513), (2, 700)])
def test_kept_fragments(oracle_lib, cuda_lib, n, copies, k_keep):
    s = _stack(n, copies, k_keep, seed=200 + copies)
    _check(s)


@pytest.mark.parametrize("order", ["random", "near_first", "far_first"])
def test_long_lists_in_any_order(oracle_lib, cuda_lib, order):
    """Lists far above the pre-selection length of points numbered at random, nearest first and farthest first.  (The order inside
    a list is left to the passes that write it; test_selection_in_a_given_order fixes it.)"""
    s = scenes.tiny(seed=300, n_points=6000, width=32, height=24, num_layers=2, n_views=1)
    s.position[:, 0:3:2] *= 0.02
    s.position[:, 1] *= 0.02
    pose = s.poses[0]
    q, t = np.asarray(pose[:4], np.float64), np.asarray(pose[4:7], np.float64)
    x, y, z, w = q
    forward = np.array([2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)])  # third row of the rotation
    rng = np.random.default_rng(5)
    along = rng.uniform(-0.5, 0.5, s.n_points)
    along = {"random": along, "near_first": np.sort(along), "far_first": np.sort(along)[::-1]}[order]
    s.position[:, :3] = (s.position[:, :3].astype(np.float64) + along[:, None] * forward).astype(np.float32)
    _check(s, min_length=600)


@pytest.mark.parametrize("k_keep", [5, 16])
@pytest.mark.parametrize("n_points", [900, 9000, 60_000])
def test_wall_facing_the_camera(oracle_lib, cuda_lib, n_points, k_keep):
    """All fragments of all lists at one depth or at one of three: ids alone decide, within the selection and across its end."""
    s = scenes.tiny(seed=320, n_points=n_points, width=72, height=40, num_layers=3, k_keep=k_keep, n_views=2)
    s.poses[:] = 0.0
    s.poses[:, 3] = 1.0  # no rotation: depth = z + 4, exactly
    s.poses[:, 6] = 4.0
    s.position[:, 2] = 0.0
    s.position[::5, 2] = -0.25
    s.position[::7, 2] = 0.25
    s.position[: n_points // 2, 2] = 0.0
    s.confidence[:] = np.minimum(s.confidence, 0.1)
    _check(s, min_length=16 * (n_points // 3000))


def _order(order, n, rng):
    keys = (rng.choice(2 * n, n, replace=False).astype(np.uint64) << 32) | rng.permutation(n).astype(np.uint64)
    if order in ("ascending", "descending"):
        return np.sort(keys) if order == "ascending" else np.sort(keys)[::-1].copy()
    if order == "one_depth":
        return (np.uint64(0x41f00000) << np.uint64(32)) | rng.permutation(n).astype(np.uint64)
    if order != "random":  # all near fragments in the shares of 15 of the 64 groups, so that the first bound is of no use
        few = np.arange(n) % 256 < 60
        keys[~few] += np.uint64(4 * n) << np.uint64(32)
        keys[few] = np.sort(keys[few]) if order == "few_groups_ascending" else np.sort(keys[few])[::-1]
    return keys


@pytest.mark.parametrize("order", ["random", "ascending", "descending", "one_depth", "few_groups_ascending", "few_groups_descending"])
def test_selection_in_a_given_order(cuda_lib, order):
    """The pre-selection on keys in a given order: the 16 smallest, ascending, in few gatherings whatever the order."""
    import torch
    from trips_b200 import _lib
    rng = np.random.default_rng(11)
    ctx = C.c_void_p()
    _lib.check(cuda_lib.trips_context_create(C.byref(ctx), torch.cuda.current_device()))
    try:
        for n in (16, 17, 32, 63, 255, 256, 257, 513, 2048, 8193, 300_007):
            keys = _order(order, n, rng)
            pos, walks = np.zeros(16, np.uint32), C.c_int()
            _lib.check(cuda_lib.trips_debug_nearest(ctx, keys.ctypes.data, n, pos.ctypes.data, C.byref(walks), None), ctx)
            assert np.array_equal(pos, np.argsort(keys)[:16]), n
            assert walks.value <= 67
            if not order.startswith("few_groups") and n >= 513:
                assert walks.value == 1  # at most 64 keys within the first bound in order, more than 128 of a random order never
            elif n >= 8193:
                assert walks.value > 1
    finally:
        cuda_lib.trips_context_destroy(ctx)


@pytest.mark.parametrize("n_points,n_views", [(8692, 1), (8693, 1), (40_000, 3), (400_000, 1)])
def test_lists_shared_by_blocks(oracle_lib, cuda_lib, n_points, n_views):
    """Lists around and far above the length from which several blocks share one, in the same call as short ones."""
    s = scenes.tiny(seed=310, n_points=n_points, width=32, height=24, num_layers=2, n_views=n_views)
    s.position[:-500, :3] *= 0.001
    s.confidence[:] = np.minimum(s.confidence, 0.1)
    _check(s, min_length=8192)


def test_more_long_lists_than_the_preselection_takes(oracle_lib, cuda_lib):
    """Above 131 072 long lists in a call nothing is pre-selected and the blend walks them itself."""
    s = scenes.tiny(seed=330, n_points=1_500_000, width=96, height=80, num_layers=3, n_views=34, size_range=(1e-3, 2e-2))
    s.confidence[:] = np.minimum(s.confidence, 0.1)
    info = _check(s, views=[0, 13, 33], min_length=1000)
    P = scenes.num_pyramid_pixels(s.width, s.height, s.num_layers)
    assert sum(int((info.cache.debug_lists(v, P)[0] > 512).sum()) for v in range(s.n_views)) > 131_072
