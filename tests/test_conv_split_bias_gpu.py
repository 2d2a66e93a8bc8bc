"""The tensor core's accumulators truncate; the fp32 convs on split operands may not pass that on as a gain below one, which layers upon
layers would multiply."""
import numpy as np
import pytest
import torch

from msnhnet_b200 import _ffi as ffi

pytestmark = pytest.mark.gpu


# one to four tensor-core steps a k-block, mixed ones, one share and several
@pytest.mark.parametrize("cin,k", [(8, 3), (16, 3), (24, 3), (32, 3), (48, 3), (96, 1), (256, 3)])
@pytest.mark.parametrize("shares", ["1", "3"])
def test_results_are_no_smaller_than_the_sums(cin, k, shares, monkeypatch):
    monkeypatch.setenv("MSNH_B200_CONV_SPLIT", shares)
    rng = np.random.default_rng(1)
    cout, size = 64, 40
    x = rng.standard_normal((1, cin, size, size), dtype=np.float32)
    wt = (rng.standard_normal((cout, cin, k, k)) / np.sqrt(cin * k * k)).astype(np.float32)
    ctx = ffi.Context(0)
    plan = ffi.Plan(ctx, [ffi.make_op(ffi.OP_CONV, [ffi.INPUT], filters=cout, k_h=k, k_w=k, pad_h=k // 2, pad_w=k // 2, is_output=1)], (cin, size, size), 1, ffi.F32, 0)
    try:
        plan.set_weights(0, ffi.W_WEIGHTS, wt)
        plan.finalize()
        plan.run(x)
        got = plan.read_output(0, 1).astype(np.float64).ravel()
    finally:
        plan.close()
        ctx.close()
    want = torch.nn.functional.conv2d(torch.from_numpy(x).double(), torch.from_numpy(wt).double(), padding=k // 2).numpy().ravel()
    # 102400 results whose errors are some 1.3e-7 of their norm leave the slope uncertain by 4e-10; uncorrected it is -3.6e-8 to -8.9e-8
    assert abs((got @ want) / (want @ want) - 1) < 1.2e-8
