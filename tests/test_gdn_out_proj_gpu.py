"""GDN's output projection at 64 channels on planes of whole 128-pixel tiles (csrc/gemm_tc.cu, the form with the RMS prologue) against
float64 of the very planes and gates that the call leaves in its workspace."""
import ctypes as C

import numpy as np
import pytest
import torch

from cssm_b200 import GatedDeltaNetCSSM, device_error

pytestmark = pytest.mark.gpu
f64 = lambda a: torch.from_numpy(np.asarray(a, np.float64)).cuda()


def planes(b, shape):
    """v planes (the readout) and gate planes of the workspace: [xdw: none][qkv: 3 C planes a frame][gate: C planes a frame]."""
    B, T, H, W, Cc = shape
    d = b.desc(shape)
    ws = b.buf.get("ws", b.L.cssm_gdn_workspace_bytes(C.byref(d))).view(torch.float32)
    n = B * T * Cc * H * W
    return ws[:3 * n].view(B * T, 3 * Cc, H * W)[:, 2 * Cc:].double(), ws[3 * n:4 * n].view(B * T, Cc, H * W).double()


def run(shape, edit=None, **kw):
    m = GatedDeltaNetCSSM(channels=64, kernel_size=3, qkv_conv_size=1, rope_mode="none", gate_type="factored", **kw)
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    x = torch.randn(shape, device="cuda", generator=g)
    v = m.init(5, shape, bias_scale=0.1)
    p = v["params"]
    p["rms_scale"] = (1 + 0.3 * np.random.default_rng(1).standard_normal(64)).astype(np.float32)
    if edit is not None:
        edit(p)
    b = m.bind(v)
    y = b(x).double().reshape(-1, shape[2] * shape[3], 64)
    torch.cuda.synchronize()
    assert device_error() == 0
    a, gate = planes(b, shape)
    a = a * torch.rsqrt((a * a).mean(1, keepdim=True) + 1e-6) * f64(p["rms_scale"])[None, :, None] * gate
    return y, a.permute(0, 2, 1) @ f64(p["output_proj"]["kernel"]) + f64(p["output_proj"]["bias"]), gate


@pytest.mark.parametrize("shape,dk", [((2, 3, 8, 16, 64), 4), ((4, 2, 32, 32, 64), 4), ((2, 2, 64, 64, 64), 4), ((8, 8, 32, 32, 64), 2),
                                      ((1, 1, 16, 8, 64), 1)])
def test_against_float64(shape, dk):
    """Three bf16 parts hold all 24 bits and what is dropped is below 2^-24.  The accumulator truncates at each of the four leading MMAs, half of
    2^-23 of the sum so far, which is 1, 2, 3 and 4 quarters of the last: at most 4 (0.625) 2^-24 = 1.5e-7 if all went one way.  Measured
    1.2e-7; two tf32 parts (22 bits, eight leading MMAs) 2.0e-7."""
    y, want, _ = run(shape, delta_key_dim=dk)
    assert float((y - want).norm() / want.norm()) < 1.6e-7


def test_products_beyond_float32():
    """The row factor comes after the products.  Planes near 1e17 and gates near 1e23 overflow there although the normalised rows do not: those
    outputs are taken again by FMAs (64 of them in order: below 64 / 2 roundings of 2^-24, some 1.5e-7 in practice)."""
    def edit(p):
        k = np.array(p["qkv_proj"]["kernel"])
        k[:, 128:] *= 1e17
        p["qkv_proj"] = {"kernel": k, "bias": p["qkv_proj"]["bias"]}
        p["gate_proj"] = {"kernel": np.array(p["gate_proj"]["kernel"]) * np.float32(1e23), "bias": p["gate_proj"]["bias"]}
    y, want, gate = run((2, 2, 16, 16, 64), edit, delta_key_dim=4, output_gate_act="silu", use_input_gates=False)
    assert float(gate.max()) > 1e22
    assert torch.isfinite(y).all()
    assert float((y - want).norm() / want.norm()) < 5e-7
