"""Projections of the gated block's last frame with weights split beforehand (csrc/gemm_split.cu, above 192 channels, where the caller leaves
room behind the workspace): row counts that end inside a tile, column counts around the 32-column groups of the split weights.

Both calls add the same products of the same three bfloat16 parts; column tiles of another width change no sum, so what differs is at most
the order of the epilogue's float32 sums: two projections behind each other stay below 4 * 8e-7 = 3.2e-6, held to 4e-6 (the GEMM's bound at these K)."""
import ctypes as C

import numpy as np
import pytest
import torch

from cssm_b200 import GatedCSSM, device_error
from cssm_b200._lib import check
from oracle import cssm_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Cc", [192, 196, 208, 256, 260, 384, 388, 512])
@pytest.mark.parametrize("B,T,H,W", [(1, 1, 3, 3), (2, 3, 9, 14), (5, 2, 14, 14), (37, 1, 16, 16)])
def test_room_behind_the_workspace(Cc, B, T, H, W):
    kw = dict(kernel_size=3, gate_type="factored", short_conv_spatial_size=3)
    mod = GatedCSSM(channels=Cc, rope_mode="none", **kw)
    x = torch.randn((B, T, H, W, Cc), device="cuda", generator=torch.Generator(device="cuda").manual_seed(Cc + B))
    v = mod.init(3, tuple(x.shape), bias_scale=0.1)
    b = mod.bind(v)
    d = b.desc(tuple(x.shape))
    plan, n = b.plan(d), b.L.cssm_gated_workspace_bytes(C.byref(d))
    room = 3 * 2 * 3 * (Cc + 64) * (Cc + 64)                  # three parts of two bytes of 3 C^2 weights, in whole blocks
    ys = []
    for extra in (0, room, room):
        ws = torch.full((n + extra + 256,), 0xFF, dtype=torch.uint8, device="cuda")
        y = torch.full((B, H, W, Cc), float("nan"), device="cuda")
        check(b.L.cssm_gated_forward_last(C.byref(d), C.byref(b.w), plan.data_ptr(), x.data_ptr(), y.data_ptr(), ws.data_ptr(), n + extra,
                                          torch.cuda.current_stream().cuda_stream), "forward_last")
        torch.cuda.synchronize()
        assert bool((ws[n + extra:] == 0xFF).all())           # nothing past the room that was given
        ys.append(y.cpu().numpy())
    assert orc.rel_l2(ys[1], ys[0]) <= 4e-6
    assert np.array_equal(ys[1], ys[2])
    if B * Cc <= 800:
        ref = orc.gated_forward(v["params"], x.cpu().numpy(), rope_mode="none", **kw)
        assert orc.rel_l2(ys[1], ref[:, -1]) <= 1e-4
    assert device_error() == 0
