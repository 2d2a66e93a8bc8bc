"""The fp32 convolution on split operands (four bf16 parts of every fp32 value, ten tensor-core products, k-blocks added up in fp32):
edges of its tiles and k-blocks, several tiles a CTA, shares of k on a cluster and in one CTA, values that are not finite."""
import numpy as np
import pytest
import torch

from msnhnet_b200 import _ffi as ffi

pytestmark = pytest.mark.gpu

ACTS = [ffi.ACT_NONE, ffi.ACT_LEAKY, ffi.ACT_HARD_SWISH, ffi.ACT_MISH]


def conv(x, wt, bias, stride, shares, monkeypatch, act=ffi.ACT_NONE, residual=None, pad=None):
    """The images through one conv (+ a 1x1 conv of the input added to it): output, description of its launch. shares: see
    MSNH_B200_CONV_SPLIT; None: fp32 FMAs on the CUDA cores."""
    if shares is None:
        monkeypatch.delenv("MSNH_B200_CONV_SPLIT", raising=False)
    else:
        monkeypatch.setenv("MSNH_B200_CONV_SPLIT", str(shares))
    batch, cin, h, w = x.shape
    cout, _, k, _ = wt.shape
    pad = k // 2 if pad is None else pad
    ops = [ffi.make_op(ffi.OP_CONV, [ffi.INPUT], filters=cout, stride_h=stride, stride_w=stride)] if residual is not None else []
    at = len(ops)
    ops.append(ffi.make_op(ffi.OP_CONV, [ffi.INPUT], filters=cout, k_h=k, k_w=k, stride_h=stride, stride_w=stride, pad_h=pad, pad_w=pad, has_bias=1,
                           act=act, act_param=0.1, is_output=0 if residual is not None else 1))
    if residual is not None:
        ops.append(ffi.make_op(ffi.OP_ADD, [0, at], act=act, act_param=0.1, is_output=1))
    ctx = ffi.Context(0)
    plan = ffi.Plan(ctx, ops, (cin, h, w), batch, ffi.F32, ffi.PLAN_NO_TENSOR_CORE if shares is None else 0)
    try:
        plan.set_weights(at, ffi.W_WEIGHTS, wt)
        plan.set_weights(at, ffi.W_BIAS, bias)
        if residual is not None:
            plan.set_weights(0, ffi.W_WEIGHTS, residual)
        plan.finalize()
        plan.run(x)
        out = plan.read_output(len(ops) - 1, batch)
        plan.run(x)
        assert np.array_equal(out, plan.read_output(len(ops) - 1, batch), equal_nan=True)      # the order of the sums does not depend on timing
        return out, [line for line in plan.describe().splitlines() if f" op={at} " in line][-1]
    finally:
        plan.close()
        ctx.close()


def tensors(cin, cout, h, w, k, batch, seed=3):
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((batch, cin, h, w), dtype=np.float32)
    wt = (rng.standard_normal((cout, cin, k, k)) / np.sqrt(cin * k * k)).astype(np.float32)
    return x, wt, rng.standard_normal(cout).astype(np.float32)


def reference(x, wt, bias, stride, pad):
    """The conv in 64 bits, and the sum of the absolute products: what a rounding of the sums is relative to."""
    x, wt = torch.from_numpy(x).double(), torch.from_numpy(wt).double()
    y = torch.nn.functional.conv2d(x, wt, stride=stride, padding=pad).numpy()
    size = torch.nn.functional.conv2d(x.abs(), wt.abs(), stride=stride, padding=pad).numpy()
    return y + bias[:, None, None].astype(np.float64), size + np.abs(bias)[:, None, None]


# channels at the edges of a k-block and of its tensor-core steps, ragged channel tiles of every width, planes smaller than a tile and a few
# pixels larger, a tile more than the SMs, k too short for a k-block of 32
@pytest.mark.parametrize("cin,cout,h,w,k,stride,batch", [
    (1, 1, 1, 1, 1, 1, 1), (3, 16, 19, 21, 3, 1, 2), (27, 33, 13, 10, 1, 1, 1), (32, 64, 8, 16, 1, 1, 1), (33, 47, 9, 15, 1, 1, 2), (40, 255, 13, 13, 1, 1, 1),
    (12, 48, 21, 21, 3, 2, 1), (65, 130, 1, 1, 1, 1, 3), (64, 70, 5, 27, 3, 1, 3), (8, 17, 139, 137, 3, 1, 1), (96, 300, 26, 27, 5, 1, 1)])
@pytest.mark.parametrize("shares", [1, -3, 2, 8])
def test_split_conv_is_an_fp32_conv(shares, cin, cout, h, w, k, stride, batch, monkeypatch):
    x, wt, bias = tensors(cin, cout, h, w, k, batch)
    got, desc = conv(x, wt, bias, stride, shares, monkeypatch)
    assert "conv_split " in desc
    want, size = reference(x, wt, bias, stride, k // 2)
    # In units of 2^-24, all of sums no larger than `size`: 1 for the products left out; an ulp (2) for each of a k-block's two accumulations of the large
    # products and a quarter of that for its four of the middle ones, 2^-3 of them (5, the k-blocks' sums being parts of `size`); half an ulp for every addition
    # of k-blocks (1 each, the middle ones' 1/8), of what goes to shared memory (every eighth), of shares and bias; an ulp for each of the fourteen accumulations
    # of a k-block's other products, 2^-7 of the sum (1/4 each)
    blocks = k * k * ((cin + 31) // 32)
    assert np.all(np.abs(got - want) <= size * 2.0 ** -24 * (1 + 5 + 1.5 * blocks + abs(shares) + 2))


@pytest.mark.parametrize("act", ACTS)
@pytest.mark.parametrize("shares", [2, 5, 8])
@pytest.mark.parametrize("add", [False, True])
def test_a_cluster_and_one_cta_sum_the_same_shares(act, shares, add, monkeypatch):
    x, wt, bias = tensors(72, 130, 9, 11, 3, 4)                     # 27 k-blocks: unequal shares; ragged pixel and channel tiles
    res = tensors(72, 130, 9, 11, 1, 1, seed=4)[1] if add else None
    want, desc = conv(x, wt, bias, 1, shares, monkeypatch, act, res)
    assert f"k over {shares} CTAs" in desc
    got, desc = conv(x, wt, bias, 1, -shares, monkeypatch, act, res)
    assert f"k over 1 CTAs in {shares} shares" in desc
    assert np.array_equal(got, want)
    plain, _ = conv(x, wt, bias, 1, None, monkeypatch, act, res)    # fp32 FMAs and the same epilogue
    assert np.abs(got - plain).max() <= 1e-5 * np.abs(plain).max()  # (both within 2^-24 x 60 of sums that are some 30 times a value)


@pytest.mark.parametrize("shares", [1, 2])
def test_values_that_are_not_finite_go_where_fp32_takes_them(shares, monkeypatch):
    x, wt, bias = tensors(40, 48, 12, 12, 3, 1)
    x[0, 3, 2, 2], x[0, 7, 2, 9], x[0, 39, 9, 3] = np.inf, -np.inf, np.nan
    x[0, 5, 9, 9], x[0, 6, 10, 9] = 3e38, 1e-42
    wt[:, 3, 1, 1] = 1e-3
    want, _ = conv(x, wt, bias, 1, None, monkeypatch)
    got, _ = conv(x, wt, bias, 1, shares, monkeypatch)
    assert np.isinf(want).any() and np.isnan(want).any()
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isposinf(got), np.isposinf(want)) and np.array_equal(np.isneginf(got), np.isneginf(want))
    fine = np.isfinite(want)
    assert np.all(np.abs(got[fine] - want[fine]) <= 1e-5 * np.maximum(np.abs(want[fine]), 1))


@pytest.mark.parametrize("shares", [1, 2])
def test_nan_beside_an_infinity_and_the_largest_numbers(shares, monkeypatch):
    """The NaN of all ones, which CUDA's own operations give, in the window of an infinity; values that six, four or eight bits round up to infinity."""
    x, wt, bias = tensors(40, 48, 12, 12, 3, 1)
    x[0, 3, 2, 2] = np.inf
    x[0, 7, 3, 3] = np.array([0x7fffffff], np.uint32).view(np.float32)[0]
    x[0, 8, 9, 3] = np.array([0xff800001], np.uint32).view(np.float32)[0]           # (a NaN whose low bits alone tell it from an infinity)
    x[0, 5, 9, 9] = np.finfo(np.float32).max
    wt[:, 5] *= 1e-2                                                             # (products of the largest number that fp32 holds, alone in their sums)
    wt[3, 7, 1, 1] = np.inf
    want, _ = conv(x, wt, bias, 1, None, monkeypatch)
    got, _ = conv(x, wt, bias, 1, shares, monkeypatch)
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isposinf(got), np.isposinf(want)) and np.array_equal(np.isneginf(got), np.isneginf(want))
    fine = np.isfinite(want)
    assert np.abs(want[fine]).max() > 1e35
    assert np.all(np.abs(got[fine] - want[fine]) <= 1e-5 * np.maximum(np.abs(want[fine]), 1))


@pytest.mark.parametrize("ca,cb", [(48, 48), (96, 33), (64, 255), (192, 192)])
def test_two_1x1_convs_over_one_input_in_one_launch(ca, cb, monkeypatch):
    x, wa, bias = tensors(40, ca, 13, 17, 1, 3)
    wb = tensors(40, cb, 1, 1, 1, 1, seed=9)[1]
    out = {}
    for merge in (True, False):
        monkeypatch.setenv("MSNH_B200_CONV_SPLIT", "1")
        if merge:
            monkeypatch.delenv("MSNH_B200_NO_MERGE", raising=False)
        else:
            monkeypatch.setenv("MSNH_B200_NO_MERGE", "1")
        ctx = ffi.Context(0)
        plan = ffi.Plan(ctx, [ffi.make_op(ffi.OP_CONV, [ffi.INPUT], filters=ca, act=ffi.ACT_LEAKY, act_param=0.1, is_output=1),
                              ffi.make_op(ffi.OP_CONV, [ffi.INPUT], filters=cb, act=ffi.ACT_HARD_SWISH, is_output=1)], (40, 13, 17), 3, ffi.F32, 0)
        try:
            plan.set_weights(0, ffi.W_WEIGHTS, wa)
            plan.set_weights(1, ffi.W_WEIGHTS, wb)
            plan.finalize()
            assert ("with the 1x1 conv of op 1" in plan.describe()) == merge
            plan.run(x)
            out[merge] = [plan.read_output(i, 3) for i in (0, 1)]
        finally:
            plan.close()
            ctx.close()
    for a, b in zip(out[True], out[False]):
        assert np.array_equal(a, b)


def test_runs_of_many_layers_agree_bit_for_bit(monkeypatch):
    """A chain of convs of every tile width, run again and again: what one warp hands another must not depend on timing."""
    monkeypatch.setenv("MSNH_B200_CONV_SPLIT", "3")
    rng = np.random.default_rng(7)
    widths = [16, 24, 48, 64, 32, 96, 255]
    ops, cin = [], 3
    for i, cout in enumerate(widths):
        ops.append(ffi.make_op(ffi.OP_CONV, [i - 1 if i else ffi.INPUT], filters=cout, k_h=3, k_w=3, pad_h=1, pad_w=1, act=ffi.ACT_LEAKY, act_param=0.1, is_output=1))
    ctx = ffi.Context(0)
    plan = ffi.Plan(ctx, ops, (3, 52, 52), 2, ffi.F32, 0)
    try:
        for i, cout in enumerate(widths):
            plan.set_weights(i, ffi.W_WEIGHTS, (rng.standard_normal((cout, cin, 3, 3)) / np.sqrt(4.5 * cin)).astype(np.float32))
            cin = cout
        plan.finalize()
        x = rng.random((2, 3, 52, 52), dtype=np.float32)
        want = None
        for _ in range(40):
            plan.run(x)
            got = [plan.read_output(i, 2) for i in range(len(widths))]
            want = want or got
            for i, (a, b) in enumerate(zip(got, want)):
                assert np.array_equal(a, b), f"layer {i}"
    finally:
        plan.close()
        ctx.close()


def test_a_plan_without_tensor_cores_stays_without(monkeypatch):
    monkeypatch.setenv("MSNH_B200_CONV_SPLIT", "2")
    ctx = ffi.Context(0)
    plan = ffi.Plan(ctx, [ffi.make_op(ffi.OP_CONV, [ffi.INPUT], filters=16, is_output=1)], (40, 5, 5), 1, ffi.F32, ffi.PLAN_NO_TENSOR_CORE)
    try:
        plan.set_weights(0, ffi.W_WEIGHTS, np.zeros((16, 40, 1, 1), np.float32))
        plan.finalize()
        launch = [line for line in plan.describe().splitlines() if " op=0 " in line][-1]
        assert "conv_direct " in launch
    finally:
        plan.close()
        ctx.close()


# a dilated filter, and a fully connected layer, that just fits the box of an im2col tensor map and that just does not
@pytest.mark.parametrize("k,dil,h,w,fits", [(3, 64, 131, 130, True), (3, 65, 133, 134, False), (3, 80, 170, 163, False), (0, 1, 129, 3, True), (0, 1, 130, 3, False), (0, 1, 2, 200, False)])
@pytest.mark.parametrize("flags", [0, ffi.PLAN_NO_TENSOR_CORE])
def test_layers_that_an_im2col_map_cannot_walk_run_on_the_cuda_cores(flags, k, dil, h, w, fits, monkeypatch):
    if not flags:
        monkeypatch.setenv("MSNH_B200_CONV_SPLIT", "1")
    rng = np.random.default_rng(4)
    x = rng.standard_normal((2, 8, h, w), dtype=np.float32)
    conv_op = dict(filters=20, k_h=k, k_w=k, dil_h=dil, dil_w=dil) if k else dict(filters=20)
    wt = (rng.standard_normal((20, 8, k or h, k or w)) / 50).astype(np.float32)
    ctx = ffi.Context(0)
    plan = ffi.Plan(ctx, [ffi.make_op(ffi.OP_CONV if k else ffi.OP_CONNECTED, [ffi.INPUT], is_output=1, **conv_op)], (8, h, w), 2, ffi.F32, flags)
    try:
        plan.set_weights(0, ffi.W_WEIGHTS, wt)
        plan.finalize()
        launch = [line for line in plan.describe().splitlines() if " op=0 " in line][-1]
        assert ("conv_split " in launch) == (fits and not flags)
        plan.run(x)
        got = plan.read_output(0, 2)
    finally:
        plan.close()
        ctx.close()
    X, W = torch.from_numpy(x).double(), torch.from_numpy(wt).double()
    want = torch.nn.functional.conv2d(X, W, dilation=dil).numpy()
    size = torch.nn.functional.conv2d(X.abs(), W.abs(), dilation=dil).numpy()
    terms = 8 * wt.shape[2] * wt.shape[3]
    assert np.all(np.abs(got - want) <= size * 2.0 ** -24 * (terms + 8))         # (a chain of as many roundings of sums no larger than `size`)
