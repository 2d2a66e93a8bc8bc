"""Images and results in pageable memory: below and above the size from which the copies go through the thread pool, with
ragged chunks, tails shorter than a cache line and buffers at odd addresses; results that come back with the run and longer ones."""
import numpy as np
import pytest

from msnhnet_b200 import _ffi as ffi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c,h,w,batch", [(3, 11, 13, 2), (3, 208, 209, 1), (3, 209, 209, 1), (5, 300, 177, 1), (3, 333, 331, 3)])
@pytest.mark.parametrize("offset", [0, 1])
def test_pageable_images_and_results(c, h, w, batch, offset):
    rng = np.random.default_rng(2)
    ctx = ffi.Context(0)
    plan = ffi.Plan(ctx, [ffi.make_op(ffi.OP_CLIP, [ffi.INPUT], const_val=-10.0, scale=10.0, is_output=1)], (c, h, w), batch, ffi.F32)
    try:
        plan.finalize()
        n = batch * c * h * w
        for _ in range(3):                                   # the staging is used again
            x = np.empty(n + offset, np.float32)[offset:]
            x[:] = rng.standard_normal(n, dtype=np.float32)
            plan.run(x.reshape(batch, c, h, w))
            out = np.empty(n + offset, np.float32)[offset:]
            ctx.check(plan.lib.msnh_b200_plan_read_output(plan.h, 0, out.ctypes.data_as(ffi.C.POINTER(ffi.C.c_float)), n))
            assert np.array_equal(out, x)
    finally:
        plan.close()
        ctx.close()
