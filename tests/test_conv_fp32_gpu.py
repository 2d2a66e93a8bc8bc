"""The CUDA-core fp32 convolution at the edges of its tiles: ragged pixel and channel tiles, pad channels, filter taps that
share a k-step, every number of CTAs that may split a tile's sums (including more CTAs than k-steps)."""
import numpy as np
import pytest

import helpers as H
from msnhnet_b200 import _ffi as ffi
from oracle import msnh_oracle as mo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("split", [1, 2, 3, 5, 8])
@pytest.mark.parametrize("cin,cout,h,w,k,stride", [(3, 16, 9, 7, 3, 1), (6, 255, 8, 8, 1, 1), (20, 64, 13, 13, 3, 2), (96, 70, 5, 27, 3, 1), (65, 130, 1, 1, 1, 1)])
def test_fp32_conv_against_the_oracle(split, cin, cout, h, w, k, stride, monkeypatch):
    monkeypatch.setenv("MSNH_B200_FP32_SPLIT", str(split))
    rng = np.random.default_rng(5)
    batch, pad = 3, k // 2
    x = rng.random((batch, cin, h, w), dtype=np.float32) - np.float32(0.4)
    w0 = (rng.standard_normal((cin, cin, 1, 1)) / np.sqrt(cin)).astype(np.float32)       # first layer: the conv under test reads a channels-last tensor
    wt = (rng.standard_normal((cout, cin, k, k)) * np.sqrt(2.0 / (cin * k * k))).astype(np.float32)
    bias = rng.standard_normal(cout).astype(np.float32)
    ops = [ffi.make_op(ffi.OP_CONV, [ffi.INPUT], filters=cin),
           ffi.make_op(ffi.OP_CONV, [0], filters=cout, k_h=k, k_w=k, stride_h=stride, stride_w=stride, pad_h=pad, pad_w=pad, has_bias=1,
                       act=ffi.ACT_LEAKY, act_param=0.1, is_output=1)]
    ctx = ffi.Context(0)
    plan = ffi.Plan(ctx, ops, (cin, h, w), batch, ffi.F32, ffi.PLAN_NO_TENSOR_CORE)
    try:
        plan.set_weights(0, ffi.W_WEIGHTS, w0)
        plan.set_weights(1, ffi.W_WEIGHTS, wt)
        plan.set_weights(1, ffi.W_BIAS, bias)
        plan.finalize()
        assert f"k over {split} CTAs" in plan.describe()
        plan.run(x)
        got = plan.read_output(1, batch)
        plan.run(x)
        assert np.array_equal(got, plan.read_output(1, batch))      # the order of the sums does not depend on timing
    finally:
        plan.close()
        ctx.close()
    for i in range(batch):
        a = mo.conv2d(x[i], w0, 1, 1, 1, 1, 0, 0, 1, 1, 1)
        ref = mo.activate(mo.conv2d(a, wt, k, k, stride, stride, pad, pad, 1, 1, 1) + bias[:, None, None], "leaky", [0.1])
        assert H.rel_err(got[i], ref) < 2e-6
