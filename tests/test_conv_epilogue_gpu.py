"""The tensor-core conv's epilogue where it can go wrong: mish far out on both sides (four values share a reciprocal), residuals
fetched in boxes that hang over the last pixel and channel, store units of every width, several tiles per CTA."""
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


def test_mish_far_out():
    values = np.array([-6e4, -90, -50, -20, -9.9, -5, -1, -1e-3, 0, 1e-3, 1, 5, 9.9, 10.1, 20, 44, 88, 120, 3e4, 6e4], np.float32)
    x = np.zeros((1, 16, 20, 20), np.float32)
    for c in range(16):                                        # neighbours in every combination of sizes
        x[0, c] = values[(np.arange(400) * (2 * c + 1) + c) % len(values)].reshape(20, 20)
    got = run([ffi.make_op(ffi.OP_CONV, [ffi.INPUT], filters=16, act=ffi.ACT_MISH, is_output=1)],
              [(0, ffi.W_WEIGHTS, np.eye(16, dtype=np.float32).reshape(16, 16, 1, 1))], (16, 20, 20), x, ffi.F16)
    v = x.astype(np.float16).astype(np.float64)
    want = v * np.tanh(np.logaddexp(0, v))
    assert np.all(np.abs(got - want) <= 1e-3 * np.abs(want) + 1e-6)


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
