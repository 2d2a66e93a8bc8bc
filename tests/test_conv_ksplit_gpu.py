"""The tensor-core conv with the k of a tile shared by a cluster: every cluster size, ragged pixel and channel tiles, fewer rows
than CTAs, shares of unequal length, residuals, channel counts that are no multiple of four."""
import numpy as np
import pytest

import helpers as H
from msnhnet_b200 import _ffi as ffi
from oracle import msnh_oracle as mo

pytestmark = pytest.mark.gpu


def f16(a):                    # (tf32 represents these exactly)
    return a.astype(np.float16).astype(np.float32)


@pytest.mark.parametrize("split", [2, 4, 8])
@pytest.mark.parametrize("residual", [False, True])
@pytest.mark.parametrize("cin,cout,h,w,k,stride,batch", [(32, 16, 9, 7, 3, 1, 1), (64, 70, 13, 13, 3, 2, 2), (96, 255, 8, 8, 3, 1, 1), (576, 48, 1, 1, 1, 1, 3),
                                                        (40, 130, 12, 11, 3, 1, 4)])
def test_shared_k_against_the_oracle(split, residual, cin, cout, h, w, k, stride, batch, monkeypatch):
    monkeypatch.setenv("MSNH_B200_K_SPLIT", str(split))
    rng = np.random.default_rng(6)
    pad = k // 2
    x = f16(rng.random((batch, cin, h, w), dtype=np.float32) - np.float32(0.4))
    w0 = f16(rng.standard_normal((cin, cin, 1, 1)) / np.sqrt(cin))
    wt = f16(rng.standard_normal((cout, cin, k, k)) * np.sqrt(2.0 / (cin * k * k)))
    ws = f16(rng.standard_normal((cout, cin, 1, 1)) / np.sqrt(cin))
    bias = rng.standard_normal(cout).astype(np.float32)
    ops = [ffi.make_op(ffi.OP_CONV, [ffi.INPUT], filters=cin),
           ffi.make_op(ffi.OP_CONV, [0], filters=cout, stride_h=stride, stride_w=stride),
           ffi.make_op(ffi.OP_CONV, [0], filters=cout, k_h=k, k_w=k, stride_h=stride, stride_w=stride, pad_h=pad, pad_w=pad, has_bias=1,
                       act=ffi.ACT_LEAKY, act_param=0.1, is_output=0 if residual else 1)]
    if residual:
        ops.append(ffi.make_op(ffi.OP_ADD, [1, 2], act=ffi.ACT_RELU, is_output=1))
    ctx = ffi.Context(0)
    plan = ffi.Plan(ctx, ops, (cin, h, w), batch, ffi.F32)
    try:
        for op, wi in ((0, w0), (1, ws), (2, wt)):
            plan.set_weights(op, ffi.W_WEIGHTS, wi)
        plan.set_weights(2, ffi.W_BIAS, bias)
        plan.finalize()
        assert f"k over {split} CTAs" in plan.describe()
        plan.run(x)
        got = plan.read_output(len(ops) - 1, batch)
        plan.run(x)
        assert np.array_equal(got, plan.read_output(len(ops) - 1, batch))      # the order of the sums does not depend on timing
    finally:
        plan.close()
        ctx.close()
    for i in range(batch):
        a = mo.conv2d(x[i], w0, 1, 1, 1, 1, 0, 0, 1, 1, 1)
        ref = mo.activate(mo.conv2d(a, wt, k, k, stride, stride, pad, pad, 1, 1, 1) + bias[:, None, None], "leaky", [0.1])
        if residual:
            s = mo.conv2d(a, ws, 1, 1, stride, stride, 0, 0, 1, 1, 1)
            ref = np.maximum(ref + s, 0)
        assert H.rel_err(got[i], ref) < H.TOL_F32
