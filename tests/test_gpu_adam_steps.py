"""Adam at the ends of the step counter, which counts in 32 bits without sign: the first element of every thread meets an empty
cache of the learning rate, whatever its count.  Weights and moments must be those of the scalar restatement: 1e-6 relative for a
handful of 32-bit operations, and for the step that the weight takes what powf (4 ulp) leaves of 1 - beta^t."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("n", [3, 4096 + 5])
@pytest.mark.parametrize("steps", [0, 1, 2**31 - 2, 2**31 - 1, 2**32 - 3, 2**32 - 2])
def test_adam_at_step_counts(oracle_lib, cuda_lib, steps, n, fused):
    import torch
    from trips_b200 import _lib
    rng = np.random.default_rng(steps % 1000 + n)
    w, g, m, v = (rng.normal(size=n).astype(np.float32) for _ in range(4))
    v = np.abs(v)
    rule = dict(lr=1e-2, beta1=0.9, beta2=0.999, eps=1e-8, rel_decay=0.1, abs_decay=0.05)
    dw, dg, dm, dv = (torch.from_numpy(a.copy()).cuda() for a in (w, g, m, v))
    ds = torch.from_numpy(np.full(n, steps, np.uint32).view(np.int32)).cuda()
    flt_max = float(np.finfo(np.float32).max)
    hyper = (rule["lr"], rule["beta1"], rule["beta2"], rule["eps"], rule["rel_decay"], rule["abs_decay"], 0.0, 0.0, flt_max)
    ctx = C.c_void_p()
    _lib.check(cuda_lib.trips_context_create(C.byref(ctx), torch.cuda.current_device()))
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    try:
        if fused:
            gp, pp = (C.c_void_p * 1)(dg.data_ptr()), (C.c_void_p * 1)(dw.data_ptr())
            seg = (_lib.TripsAdamSegment * 1)(_lib.TripsAdamSegment(0, *hyper))
            _lib.check(cuda_lib.trips_fused_reduce_adam(ctx, gp, pp, 1, 0, seg, 1, 0, n, dm.data_ptr(), dv.data_ptr(), ds.data_ptr(), stream), ctx)
        else:
            row = (_lib.TripsAdamTensor * 1)(_lib.TripsAdamTensor(dw.data_ptr(), dg.data_ptr(), dm.data_ptr(), dv.data_ptr(), ds.data_ptr(), n, *hyper))
            _lib.check(cuda_lib.trips_adam_step(ctx, row, 1, stream), ctx)
        torch.cuda.synchronize()
    finally:
        cuda_lib.trips_context_destroy(ctx)
    count, w0 = np.full(n, steps, np.int64), w.copy()
    oracle_lib.adam(w, g, m, v, count, **rule)
    assert np.array_equal(ds.cpu().numpy().view(np.uint32), (count % 2**32).astype(np.uint32))
    t, ulps = float(count[0]), 4 * 2.0**-24
    rel = ulps * (0.5 / (1 - 0.999**t) + 1 / (1 - 0.9**t)) + 1e-6
    assert np.all(np.abs(dw.cpu().numpy() - w) <= 1e-6 * np.abs(w0) + rel * np.abs(w - w0))
    for got, want in ((dm, m), (dv, v)):
        assert np.allclose(got.cpu().numpy(), want, rtol=1e-6, atol=1e-7)
