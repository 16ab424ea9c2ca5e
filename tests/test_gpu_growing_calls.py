"""Inference calls that outgrow the buffers of the call before: by entries, by fragments, by both, with long lists and under the rules of
the second pipeline.  The pass is taken up where it stopped (its views are set up and its points counted once), and gives the pyramid,
the statistics and the status of a context of its own, to the bit."""
import pytest

from trips_b200 import scenes
from util import gpu_render

pytestmark = pytest.mark.gpu


def _scene(n_points, n_views, size, spread=1.0, channels=4):
    s = scenes.tiny(seed=900, n_points=n_points, n_views=n_views, width=96, height=64, num_layers=4, size_range=(0.5 * size, size), channels=channels)
    s.position[:, :3] *= spread
    return s


GROWTH = {
    "entries": lambda: (_scene(300, 1, 0.01), _scene(9000, 2, 0.01)),
    "fragments": lambda: (_scene(40_000, 8, 0.001, 0.4), _scene(40_000, 8, 1.0, 0.4)),
    "both": lambda: (_scene(300, 1, 0.01), _scene(40_000, 8, 1.0)),
    "some_views_fit": lambda: (_scene(40_000, 5, 0.3), _scene(40_000, 8, 0.3)),
    "second_batch": lambda: (_scene(40_000, 3, 0.3), _scene(40_000, 11, 0.3)),
    "long_lists": lambda: (_scene(60_000, 4, 0.3, 1.0), _scene(60_000, 4, 0.3, 0.05)),
    "nothing_to_all": lambda: (_scene(1, 1, 0.01), _scene(40_000, 8, 1.0)),
    "8_channels": lambda: (_scene(300, 1, 0.01, channels=8), _scene(40_000, 8, 1.0, channels=8)),
}


@pytest.mark.parametrize("combine", [False, True])
@pytest.mark.parametrize("growth", sorted(GROWTH))
def test_growing_calls(cuda_lib, growth, combine):
    import torch
    if combine and growth == "long_lists":
        pytest.skip("one thread walks each list there")
    small, large = GROWTH[growth]()
    kw = dict(combine_lists=True) if combine else {}
    _, info, blend = gpu_render(large, train=False, **kw)
    with torch.no_grad():
        alone = [t.clone() for t in blend(info)]
        stats = info.cache.stats()
        _, before, _ = gpu_render(small, train=False, **kw)
        blend(before), blend(before)
        cache = info.cache = before.cache
        for _ in range(2):  # the call that grows, then one that fits
            cache.stage_times(reset=True)
            together = blend(info)
            times = cache.stage_times(reset=True)
            assert times["setup_cams"][2] == (large.n_views + 7) // 8
            assert cache.last_status() == 0 and cache.stats() == stats
            for a, b in zip(alone, together):
                assert torch.equal(a, b)
