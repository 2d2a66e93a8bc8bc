"""The fp32 convolution on split operands against fp32 FMAs on the CUDA cores, which it stands in for: no further from the sums in 64
bits whatever the data are like, and exact where those are."""
import numpy as np
import pytest
import torch

from msnhnet_b200 import _ffi as ffi

pytestmark = pytest.mark.gpu


def conv(x, wt, shares, monkeypatch):
    """shares: see MSNH_B200_CONV_SPLIT; None: fp32 FMAs on the CUDA cores."""
    if shares is None:
        monkeypatch.delenv("MSNH_B200_CONV_SPLIT", raising=False)
    else:
        monkeypatch.setenv("MSNH_B200_CONV_SPLIT", str(shares))
    cout, _, k, _ = wt.shape
    ctx = ffi.Context(0)
    plan = ffi.Plan(ctx, [ffi.make_op(ffi.OP_CONV, [ffi.INPUT], filters=cout, k_h=k, k_w=k, pad_h=k // 2, pad_w=k // 2, is_output=1)], x.shape[1:], 1, ffi.F32,
                    ffi.PLAN_NO_TENSOR_CORE if shares is None else 0)
    try:
        plan.set_weights(0, ffi.W_WEIGHTS, wt)
        plan.finalize()
        plan.run(x)
        return plan.read_output(0, 1).astype(np.float64).ravel()
    finally:
        plan.close()
        ctx.close()


def sums(x, wt):
    """The conv in 64 bits."""
    return torch.nn.functional.conv2d(torch.from_numpy(x).double(), torch.from_numpy(wt).double(), padding=wt.shape[2] // 2).numpy().ravel()


def tensors(kind, cin, cout, k, size=32):
    rng = np.random.default_rng(5)
    x = rng.standard_normal((1, cin, size, size), dtype=np.float32)
    wt = (rng.standard_normal((cout, cin, k, k)) / np.sqrt(cin * k * k)).astype(np.float32)
    if kind == "leaky":                  # activations behind a LeakyReLU
        x = np.where(x > 0, x, np.float32(0.1) * x)
    elif kind == "rectified":
        x = np.maximum(x, 0)
    elif kind == "image":
        x = rng.random(x.shape, dtype=np.float32)
    elif kind == "positive":             # no sum cancels: what an accumulator cuts off has one sign
        x, wt = rng.random(x.shape, dtype=np.float32), np.abs(wt)
    elif kind == "wide":                 # magnitudes over twelve binades either way
        x, wt = (x * np.exp(2 * rng.standard_normal(x.shape))).astype(np.float32), (wt * np.exp(2 * rng.standard_normal(wt.shape))).astype(np.float32)
    elif kind == "sparse":
        x = x * (rng.random(x.shape) < 0.05).astype(np.float32)
    elif kind == "dominated":            # one product of a sum a thousand times the others
        wt[np.arange(cout), rng.integers(0, cin, cout), k // 2, k // 2] *= 1000
    elif kind == "one-hot":
        wt[:] = 0
        wt[np.arange(cout), rng.integers(0, cin, cout), k // 2, k // 2] = 1
    elif kind == "integers":             # of more than six bits; sums below 2^24
        x, wt = rng.integers(-300, 301, x.shape).astype(np.float32), rng.integers(-10, 11, wt.shape).astype(np.float32)
    return x, wt


LAYERS = [(8, 1), (3, 3), (16, 3), (32, 1), (64, 1), (128, 1), (64, 3), (256, 3), (512, 3)]


@pytest.mark.parametrize("cin,k", LAYERS)
@pytest.mark.parametrize("kind", ["normal", "leaky", "rectified", "image", "positive", "wide", "sparse", "dominated"])
def test_no_further_from_the_sums_than_fp32_fmas(kind, cin, k, monkeypatch):
    x, wt = tensors(kind, cin, 64, k)
    want = sums(x, wt)
    plain = np.linalg.norm(conv(x, wt, None, monkeypatch) - want)
    for shares in (1, 3):
        got = np.linalg.norm(conv(x, wt, shares, monkeypatch) - want)
        # 65536 results: the norms of two errors of the same distribution differ by well under 2 %
        bound = plain * 1.02
        if kind == "wide":
            # Where one of a few products outweighs the rest fp32 FMAs round once or twice. A tensor core cuts off once (a remainder of up to an ulp) and
            # the k-blocks' sum is rounded (half an ulp): sqrt(1/3 + 1/12) ulp, 2^-23 * 0.72 of a value on average over its binade
            bound = max(bound, np.sqrt(5 / 12) * 0.72 * 2.0 ** -23 * np.linalg.norm(want))
        assert got <= bound, f"{shares} shares: {got / np.linalg.norm(want):.2e}, FMAs {plain / np.linalg.norm(want):.2e}"


@pytest.mark.parametrize("cin,k", LAYERS)
@pytest.mark.parametrize("kind", ["one-hot", "integers"])
@pytest.mark.parametrize("shares", [1, 3])
def test_sums_that_fp32_holds_come_out_exact(shares, kind, cin, k, monkeypatch):
    x, wt = tensors(kind, cin, 64, k)
    assert np.array_equal(conv(x, wt, shares, monkeypatch), sums(x, wt))
