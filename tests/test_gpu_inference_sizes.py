"""Inference calls launch everything with the buffers of earlier calls and look at the sizes afterwards.  Calls that need more entries,
more fragments or other shapes than the one before give the pyramid, the statistics and the status of a context of their own, to
the bit."""
import pytest

from trips_b200 import scenes
from util import gpu_render

pytestmark = pytest.mark.gpu


def _scene(n_points, n_views, size, channels=4):
    return scenes.tiny(seed=800, n_points=n_points, n_views=n_views, width=96, height=64, num_layers=3, size_range=(0.5 * size, size), channels=channels)


@pytest.mark.parametrize("order", ["grow", "shrink", "channels"])
def test_calls_of_changing_sizes(cuda_lib, order):
    import torch
    calls = [_scene(300, 1, 0.01), _scene(300, 1, 1.0), _scene(9000, 2, 0.05), _scene(40_000, 11, 0.3), _scene(40_000, 3, 0.01)]
    if order == "shrink":
        calls = calls[::-1]
    if order == "channels":
        calls = [_scene(9000, 2, 0.05, c) for c in (4, 8, 3, 4)]
    shared = None
    for s in calls * 2:
        ns, info, blend = gpu_render(s, train=False)
        with torch.no_grad():
            alone = [t.clone() for t in blend(info)]
            stats = info.cache.stats()
            shared = shared or info.cache.__class__()
            info.cache = shared
            together = blend(info)
        assert shared.last_status() == 0
        assert shared.stats() == stats
        for a, b in zip(alone, together):
            assert torch.equal(a, b)


def test_training_after_inference(cuda_lib):
    """A training call on a context that rendered before is sized by its own counts."""
    import torch
    small, large = _scene(300, 1, 0.01), _scene(9000, 2, 0.3)
    _, info, blend = gpu_render(small, train=False)
    cache = info.cache
    with torch.no_grad():
        blend(info), blend(info)
    _, info, blend = gpu_render(large, train=True)
    alone = [t.detach().clone() for t in blend(info)]
    info.cache = cache
    for _ in range(2):
        for a, b in zip(alone, blend(info)):
            assert torch.equal(a, b.detach())
        assert cache.last_status() == 0
