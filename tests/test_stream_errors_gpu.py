"""Streaming: an error a batch's kernels report belongs to the pop of that batch, although the next one already runs. The error code
is left by the host (no kernel waits in vain)."""
import time

import numpy as np
import pytest

from msnhnet_b200 import _ffi as ffi

pytestmark = pytest.mark.gpu

BATCH, SIZE = 2, 24
CODE = 3


@pytest.fixture(params=[(ffi.F16, 0), (ffi.F32, 0), (ffi.F16, ffi.PLAN_NO_GRAPH)], ids=["fp16", "fp32", "no graph"])
def plan(request):
    dtype, flags = request.param
    rng = np.random.default_rng(1)
    ctx = ffi.Context(0)
    p = ffi.Plan(ctx, [ffi.make_op(ffi.OP_CONV, [ffi.INPUT], filters=40, k_h=3, k_w=3, pad_h=1, pad_w=1), ffi.make_op(ffi.OP_CONV, [0], filters=24, is_output=1)],
                 (3, SIZE, SIZE), BATCH, dtype, flags)
    p.set_weights(0, ffi.W_WEIGHTS, rng.standard_normal((40, 3, 3, 3)).astype(np.float32))
    p.set_weights(1, ffi.W_WEIGHTS, rng.standard_normal((24, 40, 1, 1)).astype(np.float32))
    p.finalize()
    yield p
    p.close()
    ctx.close()


def push(p, images):
    if images.dtype == np.uint8:
        rc = p.lib.msnh_b200_plan_stream_push_u8(p.h, 1, images.ctypes.data, SIZE, SIZE, len(images), ffi.PREP_UNIT, 1, None, None)
    else:
        rc = p.lib.msnh_b200_plan_stream_push(p.h, 1, images.ctypes.data, len(images))
    p.ctx.check(rc)


def pop(p):
    out, n = np.empty((BATCH, 24, SIZE, SIZE), np.float32), ffi.C.c_int()
    rc = p.lib.msnh_b200_plan_stream_pop(p.h, out.ctypes.data_as(ffi.C.POINTER(ffi.C.c_float)), out.size, 0, None, ffi.C.byref(n))
    return rc, out[:n.value]


def images(kind, seed):
    rng = np.random.default_rng(seed)
    if kind == "u8":
        return rng.integers(0, 256, (BATCH, SIZE, SIZE, 3), dtype=np.uint8)
    return rng.random((BATCH, 3, SIZE, SIZE), dtype=np.float32)


def alone(p, x):
    if x.dtype != np.uint8:
        p.run(x)
    else:
        for i, img in enumerate(x):
            p.preprocess_u8(img, i, ffi.PREP_UNIT, 1)
        p.run_device(None, BATCH)
    return p.read_output(1, BATCH)


@pytest.mark.parametrize("kinds", [("float", "float"), ("u8", "u8"), ("float", "u8"), ("u8", "float")])
def test_the_batch_that_failed_is_the_one_whose_pop_says_so(plan, kinds):
    a, b = images(kinds[0], 2), images(kinds[1], 3)
    want = [alone(plan, x) for x in (a, b)]
    for _ in range(2):                                  # the second time through: the error is gone with its batch
        push(plan, a)
        push(plan, b)
        time.sleep(0.05)                                # both have run
        plan.ctx.check(plan.lib.msnh_b200_plan_stream_set_error(plan.h, CODE))
        rc, got = pop(plan)
        assert rc == ffi.OK and np.array_equal(got, want[0])
        rc, got = pop(plan)
        assert rc == 5 and np.array_equal(got, want[1])            # MSNH_B200_ERR_DEVICE_TIMEOUT
        assert f"code {CODE}" in plan.ctx.error()
    assert plan.lib.msnh_b200_plan_stream_set_error(plan.h, CODE) == 4          # nothing in flight (MSNH_B200_ERR_STATE)
    assert np.array_equal(alone(plan, a), want[0])


def test_a_reset_drops_the_error_with_the_batch(plan):
    x = images("float", 4)
    push(plan, x)
    plan.ctx.check(plan.lib.msnh_b200_plan_stream_set_error(plan.h, CODE))
    plan.ctx.check(plan.lib.msnh_b200_plan_stream_reset(plan.h))
    want = alone(plan, x)                               # (a synchronous run reports its own errors only)
    for _ in range(3):
        push(plan, x)
        rc, got = pop(plan)
        assert rc == ffi.OK and np.array_equal(got, want)
