"""The short convs of the gated block (3x3 over the plane, four causal taps over time, SiLU, plane sums) at
the plane sizes where the per-warp and per-CTA kernels change: one pixel, one row or column, strips that
end inside a plane, the last plane of a warp and the first of each CTA size, more pixels than either takes
(general kernel), planes that leave the last CTA short, against float64.

Tolerance: nine fused multiply-adds, four more and a SiLU (expf and a division, 4 ulp): each term rounds at
2^-24 of partial sums no larger than twice the 2-norm of the result, sqrt(17) * 2 * 2^-24 = 5e-7; the
sums add log2(HW) roundings and a sum of hundreds of values of both signs, so they are compared with
the 2-norm of the plane: 2e-6."""
import numpy as np
import pytest
import torch
import torch.nn.functional as F

from cssm_b200 import GatedCSSM

pytestmark = pytest.mark.gpu
SIZES = [(1, 1), (1, 9), (9, 1), (4, 8), (5, 7), (7, 7), (8, 8), (5, 13), (11, 12), (14, 14), (14, 16), (15, 15), (16, 16),
         (16, 17), (9, 32), (8, 33), (20, 20), (23, 22), (28, 28), (28, 32), (29, 31), (25, 41), (32, 33), (45, 45), (46, 45),
         (56, 56), (60, 60), (63, 65), (64, 65), (4, 128), (1, 2000), (2000, 1)]


@pytest.mark.parametrize("ksp", [0, 3])
@pytest.mark.parametrize("H,W", SIZES)
def test_short_convs_against_float64(H, W, ksp):
    B, T, C = 3, (1, 2, 6)[(H + W) % 3], 20
    m = GatedCSSM(channels=C, kernel_size=1, gate_type="factored", rope_mode="none", short_conv_spatial_size=ksp)
    g = torch.Generator(device="cuda").manual_seed(H * 100 + W)
    x = torch.randn((B, T, H, W, C), device="cuda", generator=g)
    v = m.init(3, tuple(x.shape), bias_scale=0.3)
    b, p = m.bind(v), v["params"]
    raw = b.stages(x, upto="in_proj")["xz"].double().clone()
    st = b.stages(x, upto="short_conv")
    f64 = lambda a: torch.from_numpy(np.asarray(a, np.float64)).cuda()
    y = raw[:, :C]
    if ksp:
        y = F.conv2d(y, f64(p["short_conv_spatial"]["kernel"]).permute(3, 2, 0, 1), f64(p["short_conv_spatial"]["bias"]),
                     padding=1, groups=C)
    y = F.pad(y.reshape(B, T, C, H * W), (0, 0, 0, 0, 3, 0))
    w = f64(p["short_conv_temporal"]["kernel"]).reshape(4, C, 1)
    y = sum(w[j] * y[:, j:j + T] for j in range(4)) + f64(p["short_conv_temporal"]["bias"]).reshape(C, 1)
    y = F.silu(y).reshape(B * T, C, H, W)
    got = st["xz"].double()
    assert float((got[:, :C] - y).norm() / y.norm()) < 5e-7
    assert torch.equal(got[:, C:], raw[:, C:])                       # the z planes are left alone
    s = y.sum((2, 3))
    assert float((st["ctx_sum"].double() - s).norm() / max(float(y.norm()), float(s.norm()))) < 2e-6
