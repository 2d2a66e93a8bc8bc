"""An image has the same bits in a plan of any batch size, in fp32 plans too: the shares in which a layer's sums over k are added
come from the layer and one image, and whether a cluster or a single CTA sums them does not show."""
import numpy as np
import pytest

import helpers as H
from msnhnet_b200 import _ffi as ffi
from msnhnet_b200 import synth

pytestmark = pytest.mark.gpu


def conv_plan(ctx, x, wt, stride, flags, act=ffi.ACT_LEAKY, residual=None):
    """The images x through one conv (with a bias; + a 1x1 conv of the input added to it) in a plan of their number: output, description."""
    batch, cin, h, w = x.shape
    cout, _, k, _ = wt.shape
    ops = [ffi.make_op(ffi.OP_CONV, [ffi.INPUT], filters=cin)]            # (the layer under test reads a channels-last tensor)
    if residual is not None:
        ops.append(ffi.make_op(ffi.OP_CONV, [0], filters=cout, stride_h=stride, stride_w=stride))
    conv = len(ops)
    ops.append(ffi.make_op(ffi.OP_CONV, [0], filters=cout, k_h=k, k_w=k, stride_h=stride, stride_w=stride, pad_h=k // 2, pad_w=k // 2, has_bias=1,
                           act=act, act_param=0.1, is_output=0 if conv == 2 else 1))
    if residual is not None:
        ops.append(ffi.make_op(ffi.OP_ADD, [1, 2], act=act, act_param=0.1, is_output=1))
    plan = ffi.Plan(ctx, ops, (cin, h, w), batch, ffi.F32, flags)
    try:
        plan.set_weights(0, ffi.W_WEIGHTS, np.eye(cin, dtype=np.float32)[:, :, None, None])
        plan.set_weights(conv, ffi.W_WEIGHTS, wt)
        plan.set_weights(conv, ffi.W_BIAS, np.linspace(-1, 1, cout, dtype=np.float32))
        if residual is not None:
            plan.set_weights(1, ffi.W_WEIGHTS, residual)
        plan.finalize()
        plan.run(x)
        return plan.read_output(len(ops) - 1, batch), plan.describe()
    finally:
        plan.close()


def tensors(cin, cout, h, w, k, batch):
    rng = np.random.default_rng(11)
    return (rng.standard_normal((batch, cin, h, w), dtype=np.float32), (rng.standard_normal((cout, cin, k, k)) / np.sqrt(cin * k * k)).astype(np.float32),
            (rng.standard_normal((cout, cin, 1, 1)) / np.sqrt(cin)).astype(np.float32))


@pytest.mark.parametrize("flags", [0, ffi.PLAN_NO_TENSOR_CORE])
@pytest.mark.parametrize("cin,cout,h,w,k,stride", [(512, 512, 7, 7, 3, 1), (256, 256, 14, 14, 3, 1), (256, 512, 14, 14, 3, 2), (1280, 1000, 1, 1, 1, 1), (96, 70, 13, 11, 3, 1), (512, 255, 13, 13, 1, 1)])
def test_a_layer_gives_an_image_the_same_bits_at_any_batch_size(flags, cin, cout, h, w, k, stride):
    x, wt, _ = tensors(cin, cout, h, w, k, 40)
    ctx = ffi.Context(0)
    try:
        want = np.concatenate([conv_plan(ctx, x[i:i + 1], wt, stride, flags)[0] for i in (0, 1, 39)])
        for batch in (2, 7, 40):
            got, _ = conv_plan(ctx, x[:batch], wt, stride, flags)
            assert np.array_equal(got[:2], want[:2]), batch
        assert np.array_equal(got[39], want[2])
    finally:
        ctx.close()


@pytest.mark.parametrize("name,size,batches", [("resnet18", 224, (3, 32)), ("mobilenetv2", 160, (5, 24)), ("yolov3_tiny", 416, (2, 6)), ("yolov5m", 160, (3, 9))])
def test_a_net_gives_an_image_the_same_bits_at_any_batch_size(name, size, batches):
    text = H.net_text(name, size, **({"conf": 0.02} if name.startswith("yolo") else {}))
    blob = H.net_blob(name, text)
    imgs = synth.make_images(max(batches), 3, size, size)

    def first(batch):
        g = H.GpuNet(text, blob, fp16=False, batch=batch)
        try:
            if g.is_yolo:
                g.yolo(imgs[:batch])
                return H.sort_rows(g.candidates(batch, 60000)[0])
            return g.classify(imgs[:batch])[0]
        finally:
            g.close()

    want = first(1)
    assert want.size
    for batch in batches:
        assert np.array_equal(first(batch), want), batch


# the share counts; activations with cases of their own in both epilogues, and one both take from the slow path
@pytest.mark.parametrize("shares", [2, 4, 8])
@pytest.mark.parametrize("act", [ffi.ACT_NONE, ffi.ACT_LEAKY, ffi.ACT_RELU6, ffi.ACT_MISH, ffi.ACT_SWISH, ffi.ACT_LOGISTIC, ffi.ACT_HARD_SWISH, ffi.ACT_TANH])
@pytest.mark.parametrize("add", [False, True])
def test_a_cluster_and_one_cta_sum_the_same_shares(shares, act, add, monkeypatch):
    cin, cout, h, w = 72, 130, 9, 11                                      # 27 k-blocks: unequal shares; ragged pixel and channel tiles
    x, wt, ws = tensors(cin, cout, h, w, 3, 4)
    ctx = ffi.Context(0)
    try:
        monkeypatch.setenv("MSNH_B200_K_SPLIT", str(shares))
        want, desc = conv_plan(ctx, x, wt, 1, 0, act, ws if add else None)
        assert f"k over {shares} CTAs" in desc
        monkeypatch.setenv("MSNH_B200_K_SPLIT", str(-shares))
        got, desc = conv_plan(ctx, x, wt, 1, 0, act, ws if add else None)
        assert f"k in {shares} shares" in desc and "CTAs" not in desc
        assert np.array_equal(got, want)
    finally:
        ctx.close()


@pytest.mark.parametrize("shares", [1, 2, 3, 5, 8])
@pytest.mark.parametrize("cin,k", [(6, 1), (20, 3), (96, 3)])              # fewer k-steps than shares, unequal shares
def test_a_cluster_and_one_cta_sum_the_same_shares_in_fp32(shares, cin, k, monkeypatch):
    x, wt, _ = tensors(cin, 70, 9, 11, k, 3)
    ctx = ffi.Context(0)
    try:
        monkeypatch.setenv("MSNH_B200_FP32_SPLIT", str(shares))
        want, desc = conv_plan(ctx, x, wt, 1, ffi.PLAN_NO_TENSOR_CORE)
        assert f"k over {shares} CTAs" in desc
        monkeypatch.setenv("MSNH_B200_FP32_SPLIT", str(-shares))
        got, desc = conv_plan(ctx, x, wt, 1, ffi.PLAN_NO_TENSOR_CORE)
        assert "k over 1 CTAs" in desc
        assert np.array_equal(got, want)
    finally:
        ctx.close()


# several tiles a CTA, the shares in one, two and more accumulator stages
@pytest.mark.parametrize("shares", [2, 4, 8])
@pytest.mark.parametrize("cout", [16, 32, 100])
def test_shares_of_many_tiles(shares, cout, monkeypatch):
    x, wt, _ = tensors(40, cout, 65, 63, 3, 6)                            # 24570 pixels: more than one 128-pixel tile for each SM
    ctx = ffi.Context(0)
    try:
        monkeypatch.setenv("MSNH_B200_K_SPLIT", str(-shares))
        got, desc = conv_plan(ctx, x, wt, 1, 0)
        assert f"k in {shares} shares" in desc
        want = np.concatenate([conv_plan(ctx, x[i:i + 1], wt, 1, 0)[0] for i in range(6)])
        assert np.array_equal(got, want)
        monkeypatch.setenv("MSNH_B200_K_SPLIT", "1")
        assert H.rel_err(got, conv_plan(ctx, x, wt, 1, 0)[0]) < 2.0**-10   # (the result is rounded to tf32: 2^-11 apart where the sums' last bits differ)
    finally:
        ctx.close()


def test_an_output_is_not_rounded_for_a_conv_that_reads_another_tensor():
    """Outputs are stored as they are, tensors that a tensor-core conv reads rounded to tf32, whatever memory the two share over time:
    with one image the last tensor of this chain lies behind every conv's input, with 64 where one of them was."""
    ch = (252, 248, 4, 492, 300)
    rng = np.random.default_rng(5)
    x = rng.standard_normal((64, ch[0], 1, 1), dtype=np.float32)
    weights = [(rng.standard_normal((ch[i + 1], ch[i], 1, 1)) / np.sqrt(ch[i])).astype(np.float32) for i in range(4)]
    ctx = ffi.Context(0)
    try:
        out = {}
        for batch in (1, 64):
            plan = ffi.Plan(ctx, [ffi.make_op(ffi.OP_CONV, [ffi.INPUT if i == 0 else i - 1], filters=ch[i + 1], is_output=int(i == 3)) for i in range(4)], (ch[0], 1, 1), batch, ffi.F32)
            for i, w in enumerate(weights):
                plan.set_weights(i, ffi.W_WEIGHTS, w)
            plan.finalize()
            plan.run(x[:batch])
            out[batch] = plan.read_output(3, batch)
            plan.close()
        assert np.array_equal(out[1][0], out[64][0])
        assert (out[64].view(np.uint32) & 0x1FFF).any()                   # (more than tf32's ten bits of mantissa)
    finally:
        ctx.close()


def to_tf32(a):
    """Nearest tf32, ties away from zero (cvt.rna)."""
    u = np.ascontiguousarray(a, np.float32).view(np.uint32)
    return ((u + np.uint32(0x1000)) & np.uint32(0xFFFFE000)).view(np.float32)


COPIES = {"pool 2x2": (dict(kind=ffi.OP_MAXPOOL, k_h=2, k_w=2, stride_h=2, stride_w=2), 8, lambda x: x.reshape(x.shape[0], 8, 6, 2, 6, 2).max((3, 5))),
          "pool 3x3": (dict(kind=ffi.OP_MAXPOOL, k_h=3, k_w=3, stride_h=3, stride_w=3), 8, lambda x: x.reshape(x.shape[0], 8, 4, 3, 4, 3).max((3, 5))),
          "pool 5x5": (dict(kind=ffi.OP_MAXPOOL, k_h=5, k_w=5, pad_h=2, pad_w=2), 8, None),
          "upsample": (dict(kind=ffi.OP_UPSAMPLE, stride_h=2, stride_w=2), 8, lambda x: x.repeat(2, 2).repeat(2, 3)),
          "clip": (dict(kind=ffi.OP_CLIP, const_val=-0.7371, scale=0.9173), 8, lambda x: np.clip(x, np.float32(-0.7371), np.float32(0.9173))),
          "slice": (dict(kind=ffi.OP_SLICE, slice_start=(0, 1, 0), slice_step=(1, 2, 2)), 8, lambda x: x[:, :, 1::2, ::2])}


@pytest.mark.parametrize("name", sorted(COPIES))
def test_what_a_conv_reads_is_rounded_to_nearest_behind_layers_that_move_values(name):
    """The image goes through a layer that stores values as it finds them into a 1x1 conv with unit weights, whose products and sums
    are exact: out comes the layer's result, each value the tf32 nearest to it (the tensor cores by themselves would cut bits off)."""
    kw, c, want = COPIES[name]
    kw = dict(kw)
    rng = np.random.default_rng(6)
    x = rng.standard_normal((3, c, 12, 12), dtype=np.float32)
    ctx = ffi.Context(0)
    plan = ffi.Plan(ctx, [ffi.make_op(kw.pop("kind"), [ffi.INPUT], **kw), ffi.make_op(ffi.OP_CONV, [0], filters=c, is_output=1)], (c, 12, 12), 3, ffi.F32)
    try:
        plan.set_weights(1, ffi.W_WEIGHTS, np.eye(c, dtype=np.float32)[:, :, None, None])
        plan.finalize()
        assert "conv_umma" in plan.describe()
        plan.run(x)
        got = plan.read_output(1, 3)
    finally:
        plan.close()
        ctx.close()
    if want is None:
        pad = np.pad(x, ((0, 0), (0, 0), (2, 2), (2, 2)), constant_values=-np.inf)
        ref = np.max([pad[:, :, r:r + 12, s:s + 12] for r in range(5) for s in range(5)], axis=0)
    else:
        ref = want(x)
    assert np.array_equal(got, to_tf32(ref))
