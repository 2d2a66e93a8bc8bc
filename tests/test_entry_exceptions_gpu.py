"""No C++ exception leaves a C entry point: where the host runs out of memory the entry returns a status. The allocation that fails is
made to fail in a process of its own (failing_new.cpp); nothing runs on the device meanwhile."""
import os
import subprocess
import sys

import pytest

from msnhnet_b200 import build

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))

CHILD = """
import ctypes as C
import numpy as np
from msnhnet_b200 import _ffi as ffi
fail = C.CDLL(None).fail_new_at
fail.argtypes, fail.restype = [C.c_long], C.c_long
ctx = ffi.Context(0)
lib = ctx.lib
ops = (ffi.Op * 2)(ffi.make_op(ffi.OP_CONV, [ffi.INPUT], filters=8, has_bias=1), ffi.make_op(ffi.OP_CONV, [0], filters=8, is_output=1))
weights = np.ones(3 * 8, np.float32)
ptr = weights.ctypes.data_as(C.POINTER(C.c_float))
ms = (C.c_float * 64)()

def at_every_allocation(call, ok, undo=lambda: None):
    # the entry with its first, second, ... allocation failing, until it gets through: statuses, and the context's text of each
    fail(-1)
    assert call() == ok
    undo()
    n = fail(-1)
    assert n > 0
    for k in range(n):
        fail(k)
        rc = call()
        fail(-1)
        assert rc == 6 or rc == ok, rc                    # MSNH_B200_ERR_NOMEM, or it did without
        if rc == 6: assert "memory" in ctx.error() or ctx.error() == "", ctx.error()
        if rc == ok: undo()
    assert call() == ok

h = C.c_void_p()
def create():
    return lib.msnh_b200_plan_create(ctx.h, ops, 2, 3, 8, 8, 1, ffi.F32, 0, C.byref(h))
at_every_allocation(create, 0, lambda: lib.msnh_b200_plan_destroy(h))
at_every_allocation(lambda: lib.msnh_b200_plan_set_weights(h, 0, ffi.W_WEIGHTS, ptr, weights.size), 0,
                    lambda: (lib.msnh_b200_plan_destroy(h), create()))
at_every_allocation(lambda: lib.msnh_b200_plan_set_weights(h, 0, ffi.W_WEIGHTS, ptr, 5), 1)      # (the text of the refusal allocates)
lib.msnh_b200_plan_set_weights(h, 0, ffi.W_BIAS, ptr, 8)
w1 = np.ones(64, np.float32)
lib.msnh_b200_plan_set_weights(h, 1, ffi.W_WEIGHTS, w1.ctypes.data_as(C.POINTER(C.c_float)), 64)
ctx.check(lib.msnh_b200_plan_finalize(h))
fail(0)
assert lib.msnh_b200_plan_run_instrumented(h, 1, 1, ms, 64) == 6
fail(-1)
ctx.check(lib.msnh_b200_plan_run_instrumented(h, 1, 1, ms, 64))
print("all returned")
"""


def test_entries_return_a_status_when_memory_runs_out(tmp_path):
    so = str(tmp_path / "failing_new.so")
    subprocess.run([build._host_cxx(), "-O1", "-std=c++17", "-fPIC", "-shared", "-o", so, os.path.join(HERE, "failing_new.cpp")], check=True)
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=os.path.dirname(HERE), env=dict(os.environ, LD_PRELOAD=so), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "all returned" in r.stdout, r.stdout + r.stderr
