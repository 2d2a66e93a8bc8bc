"""The tensor-core conv's epilogue where it can go wrong: residuals fetched in boxes that hang over the last pixel and
channel, store units of every width, several tiles per CTA, each
activation in layers of one wave and of several."""
import numpy as np
import pytest

import helpers as H
from msnhnet_b200 import _ffi as ffi
from oracle import msnh_oracle as mo

pytestmark = pytest.mark.gpu


def run(ops, weights, chw, x, dtype):
    ctx = ffi.Context(0)
    plan = ffi.Plan(ctx, ops, chw, x.shape[0], dtype)
    try:
        for op, slot, data in weights:
            plan.set_weights(op, slot, data)
        plan.finalize()
        plan.run(x)
        return plan.read_output(len(ops) - 1, x.shape[0])
    finally:
        plan.close()
        ctx.close()


@pytest.mark.parametrize("dtype", [ffi.F32, ffi.F16])
@pytest.mark.parametrize("cout,h,w,batch", [(16, 5, 7, 1), (24, 9, 15, 1), (72, 13, 13, 2), (136, 31, 33, 1), (64, 101, 67, 4), (320, 37, 41, 9)])
def test_residual_boxes(dtype, cout, h, w, batch):
    rng = np.random.default_rng(9)
    x = (rng.random((batch, 32, h, w), dtype=np.float32) - 0.4).astype(np.float16).astype(np.float32)
    w1 = (rng.standard_normal((cout, 32, 1, 1)) * 0.2).astype(np.float16).astype(np.float32)
    w2 = (rng.standard_normal((cout, cout, 3, 3)) * np.sqrt(2.0 / (9 * cout))).astype(np.float16).astype(np.float32)
    ops = [ffi.make_op(ffi.OP_CONV, [ffi.INPUT], filters=cout),
           ffi.make_op(ffi.OP_CONV, [0], filters=cout, k_h=3, k_w=3, pad_h=1, pad_w=1, act=ffi.ACT_LEAKY, act_param=0.1),
           ffi.make_op(ffi.OP_ADD, [0, 1], act=ffi.ACT_RELU, is_output=1)]
    got = run(ops, [(0, ffi.W_WEIGHTS, w1), (1, ffi.W_WEIGHTS, w2)], (32, h, w), x, dtype)
    for i in {0, batch - 1}:
        a = mo.conv2d(x[i], w1, 1, 1, 1, 1, 0, 0, 1, 1, 1)
        if dtype == ffi.F16:
            a = a.astype(np.float16).astype(np.float32)
        b = mo.activate(mo.conv2d(a, w2, 3, 3, 1, 1, 1, 1, 1, 1, 1), "leaky", [0.1])
        assert H.rel_err(got[i], np.maximum(a + b, 0)) < (2e-3 if dtype == ffi.F16 else H.TOL_F32)


@pytest.mark.parametrize("dtype", [ffi.F32, ffi.F16])
@pytest.mark.parametrize("h,w,batch", [(13, 13, 1), (151, 149, 2)])
@pytest.mark.parametrize("act,name", [(ffi.ACT_NONE, "none"), (ffi.ACT_RELU, "relu"), (ffi.ACT_RELU6, "relu6"),
                                      (ffi.ACT_HARD_SWISH, "hardswish"), (ffi.ACT_MISH, "mish")])
def test_activations_by_waves(dtype, h, w, batch, act, name):
    rng = np.random.default_rng(4)
    x = ((rng.random((batch, 32, h, w), dtype=np.float32) - 0.5) * 4).astype(np.float16).astype(np.float32)
    wt = (rng.standard_normal((72, 32, 1, 1)) * 0.5).astype(np.float16).astype(np.float32)
    ops = [ffi.make_op(ffi.OP_CONV, [ffi.INPUT], filters=72, act=act, is_output=1)]
    got = run(ops, [(0, ffi.W_WEIGHTS, wt)], (32, h, w), x, dtype)
    for i in {0, batch - 1}:
        want = mo.conv2d(x[i], wt, 1, 1, 1, 1, 0, 0, 1, 1, 1)
        if name != "none":
            want = mo.activate(want, name, [])
        assert H.rel_err(got[i], want) < (2e-3 if dtype == ffi.F16 else H.TOL_F32)
