"""Selection of the nearest fragments where the per-pixel sort can go wrong: list lengths around its chunks of 16 (and the
shorter network for 8), many fragments of the same depth inside and across the end of the selection, and lists around
the length at which a block of its own pre-selects them.  Kept points, their order and the pyramid must be the oracle's:
ids bit for bit, alphas and colours to 1e-5 (16 products in 32 bits, 16 x 6e-8)."""
import numpy as np
import pytest

from trips_b200 import scenes
from util import gpu_render, oracle_frames, rel_err

pytestmark = pytest.mark.gpu


def _stack(n, copies, k_keep, seed):
    """`n` distinct points, `copies` of each (ids i, i + n, ...): every copy has the same depth on the same pixels."""
    s = scenes.tiny(seed=seed, n_points=n * copies, width=72, height=40, num_layers=3, k_keep=k_keep, n_views=2)
    for c in range(1, copies):
        s.position[c * n:(c + 1) * n] = s.position[:n]
        s.point_size[c * n:(c + 1) * n] = s.point_size[:n]
    s.confidence[:] = np.minimum(s.confidence, 0.1)  # the transmittance stays above the cut-off for all kept fragments
    return s


@pytest.mark.parametrize("k_keep", [1, 8, 16])
@pytest.mark.parametrize("n,copies", [(40, 1), (12, 8), (12, 9), (12, 16), (12, 17), (200, 15), (12, 33), (300, 20), (3, 512), (3, 513), (2, 700)])
def test_kept_fragments(oracle_lib, cuda_lib, n, copies, k_keep):
    s = _stack(n, copies, k_keep, seed=200 + copies)
    sa, op, frames = oracle_frames(s, train=True)
    ns, info, blend = gpu_render(s, train=True)
    outs = blend(info)
    assert info.cache.last_status() == 0
    for b, f in enumerate(frames):
        nrec, pid, alpha = info.cache.debug_records(b, f.P)
        onrec, opid, oalpha = f.records()
        assert np.array_equal(nrec, onrec)
        assert np.array_equal(pid, opid)
        assert rel_err(alpha, oalpha, floor=1e-6) <= 1e-5
        for l, ref in enumerate(f.pyramid()):
            got = outs[l][b].detach().cpu().numpy()
            assert np.max(np.abs(got - ref) / np.maximum(np.abs(ref), 1e-3)) <= 1e-5


@pytest.mark.parametrize("order", ["random", "near_first", "far_first"])
def test_long_lists_in_any_order(oracle_lib, cuda_lib, order):
    """Lists far above the pre-selection length whose fragments come in random order, nearest first and farthest first (the
    order of the points): the bound that the pre-selection starts from lets about 50, or more than fit its table, pass."""
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
    sa, op, frames = oracle_frames(s, train=True)
    ns, info, blend = gpu_render(s, train=True)
    outs = blend(info)
    assert info.cache.last_status() == 0 and info.cache.stats()["max_list_length"] > 600
    f = frames[0]
    nrec, pid, alpha = info.cache.debug_records(0, f.P)
    onrec, opid, oalpha = f.records()
    assert np.array_equal(nrec, onrec) and np.array_equal(pid, opid)
    for l, ref in enumerate(f.pyramid()):
        got = outs[l][0].detach().cpu().numpy()
        assert np.max(np.abs(got - ref) / np.maximum(np.abs(ref), 1e-3)) <= 1e-5
