"""Small kernels at the edges of what they take: pooling rows (windows over the border, channel counts that are no power of two
of vectors, planes narrower than a CTA), patch stems (odd widths, strides, tiles that end inside a row)."""
import numpy as np
import pytest

import helpers as H
from msnhnet_b200 import _ffi as ffi
from oracle import msnh_oracle as mo

pytestmark = pytest.mark.gpu


def run(ops, weights, chw, x, dtype):
    ctx = ffi.Context(0)
    ops[-1].is_output = 1
    plan = ffi.Plan(ctx, ops, chw, x.shape[0], dtype)
    try:
        for o, slot, data in weights:
            plan.set_weights(o, slot, data)
        plan.finalize()
        plan.run(x)
        return plan.read_output(len(ops) - 1, x.shape[0]), plan.describe()
    finally:
        plan.close()
        ctx.close()


def half(x):
    return x.astype(np.float16).astype(np.float32)


@pytest.mark.parametrize("dtype", [ffi.F32, ffi.F16])
@pytest.mark.parametrize("c,h,w,k,s,p", [(8, 2, 2, 2, 2, 0), (24, 7, 9, 2, 1, 0), (64, 30, 31, 2, 2, 0), (40, 17, 300, 2, 2, 1), (8, 1, 5, 2, 1, 1), (520, 5, 4, 2, 2, 1), (40, 17, 30, 3, 2, 1)])
def test_pool_rows(dtype, c, h, w, k, s, p):
    rng = np.random.default_rng(1)
    x = half(rng.standard_normal((3, c, h, w)).astype(np.float32) - np.float32(3.0))       # mostly negative: padding must not win
    got, _ = run([ffi.make_op(ffi.OP_MAXPOOL, [ffi.INPUT], k_h=k, k_w=k, stride_h=s, stride_w=s, pad_h=p, pad_w=p)], [], (c, h, w), x, dtype)
    oh, ow = got.shape[2:]
    want = np.full(got.shape, -np.inf, np.float32)
    for r in range(k):
        for q in range(k):
            for y in range(oh):
                iy = y * s - p + r
                if not 0 <= iy < h:
                    continue
                for z in range(ow):
                    ix = z * s - p + q
                    if 0 <= ix < w:
                        want[:, :, y, z] = np.maximum(want[:, :, y, z], x[:, :, iy, ix])
    assert np.array_equal(got, want)


@pytest.mark.parametrize("h,w,stride,pad", [(1, 1, 1, 1), (5, 129, 1, 1), (33, 128, 1, 1), (18, 127, 1, 0), (41, 300, 2, 1), (16, 258, 2, 1), (9, 65, 2, 0)])
def test_patch_stem(h, w, stride, pad):
    rng = np.random.default_rng(2)
    x = rng.random((2, 3, h, w), dtype=np.float32)
    wt = half((rng.standard_normal((16, 3, 3, 3)) * 0.3).astype(np.float32))
    got, desc = run([ffi.make_op(ffi.OP_CONV, [ffi.INPUT], filters=16, k_h=3, k_w=3, stride_h=stride, stride_w=stride, pad_h=pad, pad_w=pad)],
                    [(0, ffi.W_WEIGHTS, wt)], (3, h, w), x, ffi.F16)
    assert "patch" in desc
    for i in range(2):
        ref = mo.conv2d(half(x[i]), wt, 3, 3, stride, stride, pad, pad, 1, 1, 1)
        assert H.rel_err(got[i], ref) < 1e-3


@pytest.mark.parametrize("dtype", [ffi.F32, ffi.F16])
@pytest.mark.parametrize("c,h,w,k,s,p", [(1280, 7, 7, 7, 1, 0), (3, 4, 2, 2, 2, 0), (40, 9, 11, 3, 1, 1), (5, 8, 8, 8, 1, 0), (64, 61, 67, 3, 2, 1)])
def test_average_pool(dtype, c, h, w, k, s, p):
    rng = np.random.default_rng(3)
    x = half(rng.standard_normal((4, c, h, w)).astype(np.float32))
    got, _ = run([ffi.make_op(ffi.OP_AVGPOOL, [ffi.INPUT], k_h=k, k_w=k, stride_h=s, stride_w=s, pad_h=p, pad_w=p)], [], (c, h, w), x, dtype)
    for i in range(4):
        want = mo.avgpool(x[i], k, k, s, s, p, p, False)[:, :got.shape[2], :got.shape[3]]
        assert got[i].shape == want.shape and H.rel_err(got[i], want) < (1e-3 if dtype == ffi.F16 else 1e-6)
