"""The float32 channel-projection GEMM (three-way bfloat16 split on the tensor cores) through the gated
block's projection stages, against float64: ragged row tiles, tiles that cross frames, channel counts
around the 16 / 32 / 64 steps of the K loop and of the column tiles, resident and streamed weights.

Tolerance: dropped partial products are below 2^-24 of |a||b|.  The accumulator is truncated (an error of
half of 2^-23 of the running sum on average, always toward zero) at every MMA of 16 k: 6 * 4 times for
K <= 64, K / 16 times for the leading products of K up to 384, at most 24 times either way.  The running sum
averages about half of the final one, so the error is below 24 * 2^-24 * 0.5 + 2^-24 = 0.8e-6 of the
result.  Larger K has several leading accumulators of at most 2 sqrt(K / 64) blocks of 64, four MMAs each; the
parts are added with rounding to nearest.  SiLU adds a few ulp."""
import ctypes as C

import numpy as np
import pytest
import torch

from cssm_b200 import GatedCSSM, device_error
from cssm_b200._lib import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,T,H,W,Cc", [
    (1, 1, 3, 3, 4), (2, 3, 5, 7, 12), (1, 2, 11, 13, 16), (3, 2, 9, 14, 20), (1, 1, 16, 8, 32), (2, 2, 14, 14, 48),
    (1, 3, 10, 13, 64), (5, 4, 32, 32, 64), (1, 2, 12, 11, 68), (2, 1, 14, 14, 96), (1, 1, 7, 7, 128),
    (3, 1, 14, 14, 256), (40, 2, 16, 16, 256), (2, 1, 7, 7, 384), (130, 1, 8, 8, 384),
    (2, 1, 14, 14, 388), (1, 2, 9, 7, 448), (2, 1, 14, 14, 512), (1, 1, 14, 14, 772), (33, 1, 14, 14, 1024), (1, 1, 14, 14, 2048),
    (1, 1, 5, 7, 6148)])
def test_projections_against_float64(B, T, H, W, Cc):
    mod = GatedCSSM(channels=Cc, kernel_size=1, gate_type="factored")
    g = torch.Generator(device="cuda").manual_seed(B * 1000 + Cc)
    x = torch.randn((B, T, H, W, Cc), device="cuda", generator=g)
    v = mod.init(5, tuple(x.shape), bias_scale=0.3)
    b = mod.bind(v)
    p = v["params"]
    st = b.stages(x, upto="in_proj")
    f64 = lambda a: torch.from_numpy(np.asarray(a, np.float64)).cuda()
    want = x.double().reshape(-1, Cc) @ f64(p["in_proj"]["kernel"]) + f64(p["in_proj"]["bias"])
    want = want.reshape(B * T, H, W, 2 * Cc).permute(0, 3, 1, 2)
    got = st["xz"].double()
    rel = lambda a, r: float((a - r).norm() / r.norm())
    tol = 8e-7 if Cc <= 384 else (max(24, 4 * int(2 * (Cc / 64 + 1) ** 0.5)) * 0.5 + 1) * 2.0 ** -24
    assert rel(got[:, :Cc], want[:, :Cc]) < tol
    assert rel(got[:, Cc:], torch.nn.functional.silu(want[:, Cc:])) < 1.5 * tol
    # out_proj of these planes (planar in, channels-last out)
    d = b.desc(tuple(x.shape))
    lay = b.workspace_layout(d)
    y = torch.full_like(x, float("nan"))
    check(b.L.cssm_gated_out_proj(C.byref(d), C.byref(b.w), b.buf.get("ws", lay.total).data_ptr() + lay.xz_planar,
                                  y.data_ptr(), torch.cuda.current_stream().cuda_stream), "out_proj")
    ref = got[:, :Cc].permute(0, 2, 3, 1) @ f64(p["out_proj"]["kernel"]) + f64(p["out_proj"]["bias"])
    assert rel(y.double().reshape(ref.shape), ref) < tol
    torch.cuda.synchronize()
    assert device_error() == 0


@pytest.mark.parametrize("Cc", [64, 256, 384])
def test_bias_at_a_four_byte_offset(Cc):
    """Biases that are views into a flat parameter buffer, one float off any wider alignment: resident
    weights (64, and in_proj at 256) and streamed ones (out_proj at 256, both at 384) give the bits of the
    same call with aligned biases."""
    mod = GatedCSSM(channels=Cc, kernel_size=1, gate_type="factored")
    x = torch.randn((1, 2, 14, 13, Cc), device="cuda", generator=torch.Generator(device="cuda").manual_seed(Cc))
    v = mod.init(5, tuple(x.shape), bias_scale=0.3)
    want = mod.bind(v)(x).clone()
    p = dict(v["params"])
    for name in ("in_proj", "out_proj"):
        b = torch.from_numpy(p[name]["bias"]).cuda()
        flat = torch.zeros(b.numel() + 1, device="cuda")
        flat[1:] = b
        p[name] = {"kernel": p[name]["kernel"], "bias": flat[1:]}
        assert flat[1:].data_ptr() % 16 == 4
    got = mod.bind({"params": p})(x)
    torch.cuda.synchronize()
    assert torch.equal(got, want)
    assert device_error() == 0


@pytest.mark.parametrize("Cc", [32, 48, 256, 512])
def test_values_without_finite_parts(Cc):
    """Infinities, NaN and finite values above the largest bfloat16 in a few pixels of either projection's
    input: their rows are what float64 makes of them (rounded to float32), all other rows stay as they are."""
    big = float(np.finfo(np.float32).max)
    odd = {3: float("inf"), 40: -float("inf"), 41: big, 90: -big, 129: 3.395e38, 300: float("nan")}
    mod = GatedCSSM(channels=Cc, kernel_size=1, gate_type="factored")
    x = torch.randn((1, 2, 13, 15, Cc), device="cuda", generator=torch.Generator(device="cuda").manual_seed(Cc))
    v = mod.init(5, tuple(x.shape), bias_scale=0.3)
    b, p = mod.bind(v), v["params"]
    f64 = lambda a: torch.from_numpy(np.asarray(a, np.float64)).cuda()
    d = b.desc(tuple(x.shape))
    lay = b.workspace_layout(d)

    def same(got, want):
        want32 = want.float()
        assert torch.equal(got.isnan(), want32.isnan()) and torch.equal(got.isinf(), want32.isinf())
        inf = want32.isinf()
        assert torch.equal(got[inf], want32[inf])
        rows = [r for r in range(got.shape[0]) if r not in odd]
        assert float((got[rows].double() - want[rows]).norm() / want[rows].norm()) < 1.2e-6
        for r in (41, 90, 129):
            ok = want32[r].isfinite()
            assert ok.any() and float((got[r][ok].double() / want[r][ok] - 1).abs().max()) < 1e-4

    x.view(-1, Cc)[list(odd), Cc // 3] = torch.tensor(list(odd.values()), device="cuda")
    xz = b.stages(x, upto="in_proj")["xz"]
    same(xz[:, :Cc].permute(0, 2, 3, 1).reshape(-1, Cc),
         x.double().view(-1, Cc) @ f64(p["in_proj"]["kernel"])[:, :Cc] + f64(p["in_proj"]["bias"])[:Cc])
    planes = torch.randn((2, 2 * Cc, 13, 15), device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
    rows = planes[:, :Cc].permute(0, 2, 3, 1).reshape(-1, Cc)
    rows[list(odd), Cc // 3] = torch.tensor(list(odd.values()), device="cuda")
    planes[:, :Cc] = rows.view(2, 13, 15, Cc).permute(0, 3, 1, 2)
    y = torch.empty_like(x)
    check(b.L.cssm_gated_out_proj(C.byref(d), C.byref(b.w), planes.data_ptr(), y.data_ptr(),
                                  torch.cuda.current_stream().cuda_stream), "out_proj")
    same(y.view(-1, Cc), rows.double() @ f64(p["out_proj"]["kernel"]) + f64(p["out_proj"]["bias"]))
    torch.cuda.synchronize()
    assert device_error() == 0
