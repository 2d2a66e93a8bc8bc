"""Stems too large for a patch matrix: the image as rows of patches, the conv as kh x 1 over them."""
import numpy as np
import pytest

import helpers as H
from msnhnet_b200 import _ffi as ffi
from oracle import msnh_oracle as mo

pytestmark = pytest.mark.gpu


# odd widths, strides that leave columns over, strides beyond what TMA walks (the conv then runs on the CUDA cores), padding of its own on every side, a filter wider than the plane, one row, one channel and four
@pytest.mark.parametrize("cin,cout,h,w,kh,kw,sh,sw,ph,pw", [
    (3, 64, 64, 64, 7, 7, 2, 2, 3, 3), (3, 20, 33, 37, 7, 7, 2, 2, 3, 3), (3, 17, 21, 50, 5, 5, 1, 3, 2, 0), (4, 16, 19, 23, 5, 7, 3, 1, 0, 5),
    (1, 40, 9, 70, 3, 31, 1, 4, 1, 15), (3, 24, 70, 60, 7, 7, 9, 9, 3, 3), (3, 8, 12, 5, 7, 9, 1, 1, 3, 4), (4, 33, 18, 40, 8, 16, 2, 2, 0, 0)])
@pytest.mark.parametrize("dtype", [ffi.F16, ffi.F32])
@pytest.mark.parametrize("batch", [1, 3])
def test_row_patch_stem(batch, dtype, cin, cout, h, w, kh, kw, sh, sw, ph, pw):
    rng = np.random.default_rng(2)
    x = rng.random((batch, cin, h, w), dtype=np.float32) - np.float32(0.4)
    wt = (rng.standard_normal((cout, cin, kh, kw)) / np.sqrt(cin * kh * kw)).astype(np.float32)
    bias = rng.standard_normal(cout).astype(np.float32)
    ctx = ffi.Context(0)
    plan = ffi.Plan(ctx, [ffi.make_op(ffi.OP_CONV, [ffi.INPUT], filters=cout, k_h=kh, k_w=kw, stride_h=sh, stride_w=sw, pad_h=ph, pad_w=pw, has_bias=1,
                                      act=ffi.ACT_RELU, is_output=1)], (cin, h, w), batch, dtype, 0)
    try:
        plan.set_weights(0, ffi.W_WEIGHTS, wt)
        plan.set_weights(0, ffi.W_BIAS, bias)
        plan.finalize()
        assert "input_nchw_to_row_patches" in plan.describe() and "row patches" in plan.describe()
        plan.run(x)
        got = plan.read_output(0, batch)
    finally:
        plan.close()
        ctx.close()
    for i in range(batch):
        ref = mo.activate(mo.conv2d(x[i], wt, kw, kh, sw, sh, pw, ph, 1, 1, 1) + bias[:, None, None], "relu", [])
        assert H.rel_err(got[i], ref) < H.TOL_F32 * (2 if dtype == ffi.F16 else 1)       # one layer of 11-bit operands: 2^-11 and the store's 2^-11
