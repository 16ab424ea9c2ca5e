"""Where the device places the lists (list_starts_kernel): together they fill the view's part of the list buffer exactly, and the
lists of the 16384 pixels of a block follow one another in pixel order.  Whole numbers, compared exactly."""
import numpy as np
import pytest

from trips_b200 import scenes
from util import gpu_render

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,layers", [(16, 32, 1), (19, 27, 1), (127, 129, 1), (128, 128, 1), (145, 113, 1), (300, 220, 4)])
def test_starts_of_ragged_pyramids(cuda_lib, w, h, layers):
    s = scenes.tiny(seed=600 + w, n_points=4000, width=w, height=h, num_layers=layers, n_views=3)
    _, info, blend = gpu_render(s, train=True)
    blend(info)
    P = scenes.num_pyramid_pixels(w, h, layers)
    for v in range(s.n_views):
        counts, _, frags = info.cache.debug_lists(v, P)  # (fails where the lists do not fill the view's part of the buffer)
        starts = info.cache.debug_list_starts(v, P)
        used = np.flatnonzero(counts)
        used = used[np.argsort(starts[used])]
        assert np.array_equal(starts[used], np.concatenate([[0], np.cumsum(counts[used])[:-1]])) and frags.size == counts.sum()
        for first in range(0, P, 16384):  # the pixels of a block: one list behind the other
            c, at = counts[first:first + 16384], starts[first:first + 16384]
            assert np.array_equal(at, at[0] + np.concatenate([[0], np.cumsum(c)[:-1]]))
