"""The training step's shared-memory limit belongs to a device and context: a
process that trains in a second one gets the same gradients there. The second
context is one more of the same device, made with the driver API in a process of
its own. (Where the limit is missing the launch is refused on the host.)
"""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import ctypes
import numpy as np
from marigold_b200 import _lib, learned

cu = ctypes.CDLL("libcuda.so.1")
P = ctypes.c_void_p


def ok(rc):
    assert rc == 0, f"driver error {rc}"


def put(a):
    d = ctypes.c_uint64()
    ok(cu.cuMemAlloc_v2(ctypes.byref(d), ctypes.c_size_t(a.nbytes)))
    ok(cu.cuMemcpyHtoD_v2(d, a.ctypes.data_as(P), ctypes.c_size_t(a.nbytes)))
    return d


def step():
    B = 64
    rng = np.random.default_rng(2)
    x = rng.normal(scale=0.6, size=(B, 24)).astype(np.float32)
    label = rng.integers(0, 48, B).astype(np.uint32)
    gain = (rng.random(B) < 0.5).astype(np.float32)
    w = learned.to_bf16_bits(learned.init_params(21))
    grad, loss = np.zeros(learned.NPARAM, np.float32), np.zeros(2, np.float32)
    d = [put(a) for a in (x, label, gain, w, grad, loss)]
    p = [P(v.value) for v in d]
    rc = _lib.load().mgbvh_mlp_train_step_dev(p[0], p[1], p[2], B, p[3], p[4], p[5], None)
    assert rc == 0, f"train step: status {rc}"
    ok(cu.cuCtxSynchronize())
    ok(cu.cuMemcpyDtoH_v2(grad.ctypes.data_as(P), d[4], ctypes.c_size_t(grad.nbytes)))
    return grad


ok(cu.cuInit(0))
dev, primary, second = ctypes.c_int(), P(), P()
ok(cu.cuDeviceGet(ctypes.byref(dev), 0))
ok(cu.cuDevicePrimaryCtxRetain(ctypes.byref(primary), dev))
ok(cu.cuCtxSetCurrent(primary))
first = step()
ok(cu.cuCtxCreate_v2(ctypes.byref(second), 0, dev))
again = step()
# (two CTAs add to every gradient, in either order: a sum of two is the same)
assert np.abs(first).max() > 0 and np.array_equal(first, again)
print("CONTEXTS_OK")
"""


def test_train_step_in_a_second_context():
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert "CONTEXTS_OK" in r.stdout, r.stdout + r.stderr
