"""Inference calls launch the binning and window kernels that suit the pass before.  A pass that calls for others (points crowded into
few pixels after a spread cloud and the other way round, many more points than before) goes on with its own; its points are counted
once, it takes two more launches of the binning stage, and it gives the pyramid and the statistics of a context of its own, to the bit."""
import pytest

from trips_b200 import scenes
from util import gpu_render

pytestmark = pytest.mark.gpu


def _scene(n_points, n_views, spread, width=160, height=120):
    s = scenes.tiny(seed=950, n_points=n_points, n_views=n_views, width=width, height=height, num_layers=2, size_range=(0.001, 0.002), fx=0.9 * width)
    s.position[:, :3] *= spread
    return s


@pytest.mark.parametrize("points,views", [(20_000, 1), (20_000, 8), (36_000, 11)])
def test_crowded_and_spread(cuda_lib, points, views):
    import torch
    scene = {"crowded": _scene(points, views, 0.01), "spread": _scene(points, views, 1.0)}
    _check(torch, scene, ["crowded", "crowded", "spread", "spread", "crowded", "spread", "spread"])


def test_many_more_points(cuda_lib):
    import torch
    scene = {"many": _scene(400_000, 8, 1.0, 640, 480), "few": _scene(20_000, 1, 1.0, 640, 480)}  # 139 and 12 points in the fullest 8x4 pixels
    stats = _check(torch, scene, ["many", "many", "few", "many", "many"], other=[("few", "many")])
    assert stats["many"]["visible_points"] > max(8 * stats["few"]["visible_points"], 2 << 20)


def _check(torch, scene, order, other=None):
    """other: the changes from one scene to the next after which the pass calls for other kernels (None: all changes)."""
    with torch.no_grad():
        made, alone, stats, plain = {}, {}, {}, {}
        for name, s in scene.items():
            _, info, blend = gpu_render(s, train=False)
            alone[name], made[name] = [t.clone() for t in blend(info)], info
            stats[name] = info.cache.stats()
            info.cache.stage_times(reset=True)
            blend(info)
            plain[name] = info.cache.stage_times(reset=True)["bin_points"][2]
        cache = made[order[0]].cache
        for before, name in zip([order[0]] + order, order):
            made[name].cache = cache
            cache.stage_times(reset=True)
            together = blend(made[name])
            times = cache.stage_times(reset=True)
            passes = (scene[name].n_views + 7) // 8
            changed = before != name and (other is None or (before, name) in other)
            assert times["setup_cams"][2] == passes and times["bin_points"][2] == plain[name] + (2 if changed else 0)
            assert cache.last_status() == 0 and cache.stats() == stats[name]
            for a, b in zip(alone[name], together):
                assert torch.equal(a, b)
    return stats
