"""The binning passes at the sizes where they can go wrong: point counts around a block's 256 threads, a ticket's 1024 points and a
bounding box's 8192, view counts around the sweeps of 4 and the groups of 16, with and without the radius drop-out (the only
reader of the projected radius).  Kept points and their order must be the oracle's, ids bit for bit, alphas to 1e-5 (a handful of
32-bit products)."""
import numpy as np
import pytest

from trips_b200 import scenes
from util import gpu_render, oracle_frames, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radius", [None, 1.5])
@pytest.mark.parametrize("n_points,n_views", [(1, 1), (255, 4), (257, 5), (1023, 3), (1025, 1), (2049, 17), (8193, 2)])
def test_entries_of_ragged_clouds(oracle_lib, cuda_lib, n_points, n_views, radius):
    s = scenes.tiny(seed=400 + n_points, n_points=n_points, n_views=n_views, width=61, height=43, num_layers=3)
    kw = {} if radius is None else dict(drop_out_points_by_radius=True, drop_out_radius_threshold=radius)
    _, _, frames = oracle_frames(s, train=True, **kw)
    _, info, blend = gpu_render(s, train=True, **kw)
    for call in range(2):  # a sized call, then one in the steady state
        blend(info)
        assert info.cache.last_status() == 0
        for b, f in enumerate(frames):
            nrec, pid, alpha = info.cache.debug_records(b, f.P)
            onrec, opid, oalpha = f.records()
            assert np.array_equal(nrec, onrec) and np.array_equal(pid, opid)
            assert rel_err(alpha, oalpha, floor=1e-6) <= 1e-5


@pytest.mark.parametrize("w,h,layers", [(61, 43, 6), (64, 48, 7), (97, 65, 8), (2, 2, 2), (33, 3, 4)])
def test_layers_at_the_far_border(oracle_lib, cuda_lib, w, h, layers):
    """Large points around the right and lower border, where the footprint leaves some layer before the last one."""
    s = scenes.tiny(seed=450 + w, n_points=1500, n_views=2, width=w, height=h, num_layers=layers, size_range=(0.05, 3.0), fx=0.9 * w)
    s.intrinsics[:, 2] = 0.85 * w
    s.intrinsics[:, 3] = 0.85 * h
    _, _, frames = oracle_frames(s, train=True)
    _, info, blend = gpu_render(s, train=True)
    blend(info)
    assert info.cache.last_status() == 0
    for b, f in enumerate(frames):
        nrec, pid, alpha = info.cache.debug_records(b, f.P)
        onrec, opid, oalpha = f.records()
        assert np.array_equal(nrec, onrec) and np.array_equal(pid, opid)
        assert rel_err(alpha, oalpha, floor=1e-6) <= 1e-5
