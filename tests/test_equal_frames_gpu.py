"""Clips of equal frames, last frame only, without RoPE (the float32 mixers of the image classifier): one projection per image and
as many frames as the temporal conv tells apart, against the block on clips that hold the frame T times."""
import numpy as np
import pytest
import torch

from cssm_b200 import SimpleCSSM
from oracle import simple_oracle as so
from oracle import cssm_oracle as orc

pytestmark = pytest.mark.gpu


# steps below, at and above the number of temporal taps; no temporal conv; spatial conv of 0, 3 and 5 taps; a plane a warp and a CTA
@pytest.mark.parametrize("T", [2, 3, 4, 5, 9])
@pytest.mark.parametrize("kt,ksp,side", [(4, 3, (22, 34)), (0, 3, (22, 34)), (1, 0, (20, 20)), (2, 3, (20, 20)), (3, 3, (90, 88)), (5, 5, (20, 24))])
@pytest.mark.parametrize("gate", ["factored", "dense"])
def test_last_frame_of_a_repeated_image(T, kt, ksp, side, gate):
    E = 16
    m = SimpleCSSM(cssm_type="gated", embed_dim=E, kernel_size=5, gate_type=gate, seq_len=T, pos_embed="none", stem_layers=1,
                   pool_type="max", short_conv_size=kt, short_conv_spatial_size=ksp)
    x = np.random.default_rng(T).random((3, *side, 1)).astype(np.float32)
    H, W = m.feature_hw(*side)
    bkw = dict(kernel_size=5, rope_mode="none", gate_type=gate, short_conv_size=kt, short_conv_spatial_size=ksp)
    p = so.init_simple_params(5, cin=1, embed_dim=E, H=H, W=W, num_classes=2, cssm_type="gated", stem_mode="default", stem_layers=1,
                              bias_scale=0.1, block_kwargs=bkw)
    ref = so.simple_forward(p, x, cssm_type="gated", seq_len=T, stem_mode="default", stem_layers=1, pool_type="max", block_kwargs=bkw)
    bound = m.bind({"params": p})
    xd = torch.from_numpy(x).cuda()
    got = bound(xd, last_frame_only=True).cpu().numpy()
    assert orc.rel_l2(got, ref) <= 1e-4
    full = bound(xd).cpu().numpy()                       # every frame through the block
    assert orc.rel_l2(got, full) <= 2e-6
