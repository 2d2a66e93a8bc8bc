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


@pytest.mark.parametrize("c,h,w,batch", [(3, 11, 13, 2), (1, 512, 512, 1), (1, 512, 513, 1), (5, 300, 177, 3)])
def test_streamed_results(c, h, w, batch):
    rng = np.random.default_rng(3)
    ctx = ffi.Context(0)
    plan = ffi.Plan(ctx, [ffi.make_op(ffi.OP_CLIP, [ffi.INPUT], const_val=-10.0, scale=10.0, is_output=1)], (c, h, w), batch, ffi.F32)
    try:
        plan.finalize()
        sent = []
        for k in (batch, 1, batch, batch):
            if len(sent) == 2:
                pop(plan, sent.pop(0))
            x = rng.standard_normal((k, c, h, w), dtype=np.float32)
            ctx.check(plan.lib.msnh_b200_plan_stream_push(plan.h, 0, x.ctypes.data, k))
            sent.append(x)
        for x in sent:
            pop(plan, x)
    finally:
        plan.close()
        ctx.close()


def pop(plan, want):
    out, n = np.empty_like(want), ffi.C.c_int()
    plan.ctx.check(plan.lib.msnh_b200_plan_stream_pop(plan.h, out.ctypes.data_as(ffi.C.POINTER(ffi.C.c_float)), out.size, 0, None, ffi.C.byref(n)))
    assert n.value == len(want) and np.array_equal(out, want)


def clip_plan(ctx, c, h, w, batch):
    plan = ffi.Plan(ctx, [ffi.make_op(ffi.OP_CLIP, [ffi.INPUT], const_val=-10.0, scale=10.0, is_output=1)], (c, h, w), batch, ffi.F32)
    plan.finalize()
    return plan


# (the pinned staging is a ring of 16 MB: just below it, at it, just above, several times round)
@pytest.mark.parametrize("floats", [4193792, 4194304, 4194305, 4200000, 8388608, 10000001, 33000003])
def test_copies_that_go_round_the_staging(floats):
    rng = np.random.default_rng(4)
    ctx = ffi.Context(0)
    plan = clip_plan(ctx, 1, 1, floats, 1)
    try:
        for _ in range(3):
            x = rng.standard_normal(floats, dtype=np.float32)
            plan.run(x.reshape(1, 1, 1, floats))
            assert np.array_equal(plan.read_output(0, 1).ravel(), x)
    finally:
        plan.close()
        ctx.close()


def address_space_mb():
    return [int(line.split()[1]) for line in open("/proc/self/status") if line.startswith("VmSize")][0] / 1024


def test_staging_does_not_grow_with_the_images():
    ctx = ffi.Context(0)
    x = np.zeros((1, 1, 1, 64 << 20), np.float32)            # 256 MB
    out = np.empty_like(x)
    small, plan = clip_plan(ctx, 1, 1, 1 << 20, 1), clip_plan(ctx, 1, 1, x.size, 1)
    try:
        small.run(x[..., :1 << 20])                           # starts the threads
        plan.run_device(None, 1)
        before = address_space_mb()
        plan.run(x)
        ctx.check(plan.lib.msnh_b200_plan_read_output(plan.h, 0, out.ctypes.data_as(ffi.C.POINTER(ffi.C.c_float)), out.size))
        assert address_space_mb() - before < 300              # (the read-back's device buffer of 256 MB may be counted; the staging was as much again)
    finally:
        small.close()
        plan.close()
        ctx.close()
