"""The two variants of the backward tile kernel: it is chosen by the visible points per pixel of layer 0, at 1.75.  Clouds on both
sides of the line, in one and several views, with the channel counts that have one or both variants; bounds as in
test_gpu_point_gradients (sums of thousands of 32-bit terms in another order than the oracle's)."""
import numpy as np
import pytest

from test_gpu_point_gradients import _check
from trips_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("channels", [3, 4, 8])
@pytest.mark.parametrize("per_pixel,n_views", [(0.3, 1), (1.6, 2), (1.9, 2), (6.0, 1)])
def test_point_gradients_at_densities(oracle_lib, cuda_lib, per_pixel, n_views, channels):
    w, h = 61, 43
    s = scenes.tiny(seed=500 + channels, n_points=int(per_pixel * w * h), n_views=n_views, width=w, height=h, num_layers=3, channels=channels)
    # all points in front of the cameras, so that nearly all are visible
    s.position[:, :3] *= 0.35
    _check(s)
