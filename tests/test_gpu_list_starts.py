"""Placing the lists (a warp takes 512 pixels, a block 16384) and handing out entries to the window passes (the bin that holds a
chunk's first entry is found by 32 lanes at a time), at the pixel and bin counts where they can go wrong.  Kept points must be the
oracle's, ids bit for bit (test_gpu_list_selection)."""
import numpy as np
import pytest

from test_gpu_list_selection import _check
from trips_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,layers", [(16, 32, 1), (19, 27, 1), (127, 129, 1), (128, 128, 1), (145, 113, 1), (300, 220, 4)])
def test_lists_of_ragged_pyramids(oracle_lib, cuda_lib, w, h, layers):
    s = scenes.tiny(seed=600 + w, n_points=4000, width=w, height=h, num_layers=layers, n_views=3)
    info = _check(s)
    P = scenes.num_pyramid_pixels(w, h, layers)
    for v in range(s.n_views):
        counts, offsets, frags = info.cache.debug_lists(v, P)
        assert np.array_equal(offsets, np.concatenate([[0], np.cumsum(counts)[:-1]])) and frags.size == counts.sum()


@pytest.mark.parametrize("bins_x,bins_y", [(1, 1), (8, 4), (11, 3), (33, 1), (41, 25)])
def test_chunks_over_bins(oracle_lib, cuda_lib, bins_x, bins_y):
    """Half of the cloud in a few bins (more than 512 entries each), the rest scattered."""
    s = scenes.tiny(seed=700 + bins_x, n_points=9000, width=32 * bins_x, height=32 * bins_y, num_layers=3, n_views=2)
    s.position[: s.n_points // 2, :3] *= 0.1
    s.confidence[:] = np.minimum(s.confidence, 0.1)
    _check(s)
