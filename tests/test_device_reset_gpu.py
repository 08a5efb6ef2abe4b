"""cudaDeviceReset ends the context and with it every attribute that was set on a kernel; a host program may go
on with new buffers afterwards.  Own process (the reset would take torch's memory with it)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROGRAM = r"""
import ctypes as C
import sys

import numpy as np

sys.path.insert(0, sys.argv[1])
from cssm_b200 import GatedCSSM, _lib
L = _lib.lib()                                  # brings the CUDA runtime with it
rt = C.CDLL("libcudart.so.12")

B, T, H, W, Cc = 1, 2, 56, 56, 128              # projections and plane kernel above 48 KB of shared memory
mod = GatedCSSM(channels=Cc, kernel_size=3, gate_type="factored")
p = mod.init(3, (B, T, H, W, Cc), bias_scale=0.1)["params"]
x = np.random.default_rng(0).standard_normal((B, T, H, W, Cc)).astype(np.float32)


def ok(rc):
    assert rc == 0, (rc, L.cssm_last_cuda_error())


def dev(n):
    q = C.c_void_p()
    ok(rt.cudaMalloc(C.byref(q), C.c_size_t(n)))
    return q.value


def put(a):
    a = np.ascontiguousarray(a, np.float32)
    q = dev(a.nbytes)
    ok(rt.cudaMemcpy(C.c_void_p(q), a.ctypes.data_as(C.c_void_p), C.c_size_t(a.nbytes), 1))
    return q


def forward():
    d, w = mod._desc(x.shape), _lib.GatedWeights()
    w.in_proj_kernel, w.in_proj_bias = put(p["in_proj"]["kernel"]), put(p["in_proj"]["bias"])
    w.out_proj_kernel, w.out_proj_bias = put(p["out_proj"]["kernel"]), put(p["out_proj"]["bias"])
    w.conv_sp_kernel, w.conv_sp_bias = put(p["short_conv_spatial"]["kernel"]), put(p["short_conv_spatial"]["bias"])
    w.conv_t_kernel, w.conv_t_bias = put(p["short_conv_temporal"]["kernel"]), put(p["short_conv_temporal"]["bias"])
    w.kernel = put(p["kernel"])
    for g, n in enumerate(("delta_proj", "B_proj", "C_proj")):
        for k, s in enumerate("hw"):
            w.gate_kernel[2 * g + k], w.gate_bias[2 * g + k] = put(p[f"{n}_{s}"]["kernel"]), put(p[f"{n}_{s}"]["bias"])
    plan, ws = dev(L.cssm_gated_plan_bytes(C.byref(d))), dev(L.cssm_gated_workspace_bytes(C.byref(d)))
    xd, yd = put(x), dev(x.nbytes)
    ok(L.cssm_gated_plan_init(C.byref(d), C.byref(w), plan, L.cssm_gated_plan_bytes(C.byref(d)), None))
    ok(L.cssm_gated_forward(C.byref(d), C.byref(w), plan, xd, yd, ws, L.cssm_gated_workspace_bytes(C.byref(d)), None))
    y = np.empty_like(x)
    ok(rt.cudaMemcpy(y.ctypes.data_as(C.c_void_p), C.c_void_p(yd), C.c_size_t(y.nbytes), 2))
    return y


first = forward()
for _ in range(2):
    ok(rt.cudaDeviceReset())
    assert np.array_equal(forward(), first)
print("same bits")
"""


def test_forward_after_a_device_reset():
    r = subprocess.run([sys.executable, "-c", PROGRAM, ROOT], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "same bits" in r.stdout, r.stdout + r.stderr
