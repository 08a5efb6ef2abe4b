"""Per-channel spatial gates multiplied into k and v by the projection's store (64 channels, planes of whole tiles) or by a launch of
their own, against the oracle."""
import numpy as np
import pytest
import torch

from cssm_b200 import DeltaNetCSSM, GatedDeltaNetCSSM
from oracle import cssm_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,T,H,W,C", [(2, 3, 8, 8, 8), (1, 2, 9, 11, 24), (2, 2, 16, 16, 48), (1, 2, 12, 10, 96), (1, 2, 32, 32, 64), (1, 2, 64, 64, 64),
                                       (1, 2, 10, 10, 160)])
def test_gdn_channel_gates(B, T, H, W, C):
    kw = dict(delta_key_dim=4, kernel_size=3, gate_type="channel", qkv_conv_size=1)
    x = np.random.default_rng(C).standard_normal((B, T, H, W, C)).astype(np.float32)
    p = orc.init_gdn_params(3, C, H, W, bias_scale=0.1, **kw)
    ref = orc.gdn_forward(p, x, rope_mode="mrope", **kw)
    got = GatedDeltaNetCSSM(channels=C, rope_mode="mrope", **kw).apply({"params": p}, torch.from_numpy(x).cuda()).cpu().numpy()
    assert orc.rel_l2(got, ref) <= 1e-4


@pytest.mark.parametrize("B,T,H,W,C", [(2, 3, 8, 8, 8), (1, 2, 9, 11, 24), (2, 2, 16, 16, 48), (1, 2, 12, 10, 96), (1, 2, 64, 64, 64)])
def test_deltanet_channel_gates(B, T, H, W, C):
    x = np.random.default_rng(C).standard_normal((B, T, H, W, C)).astype(np.float32)
    p = orc.init_deltanet_params(3, C, H, W, kernel_size=3, gate_type="channel", bias_scale=0.1)
    p["output_proj"]["bias"][:] = 0
    ref = orc.deltanet_forward(p, x, kernel_size=3, gate_type="channel", rope_mode="spatiotemporal")
    got = DeltaNetCSSM(channels=C, kernel_size=3, gate_type="channel", rope_mode="spatiotemporal").apply({"params": p}, torch.from_numpy(x).cuda())
    assert orc.rel_l2(got.cpu().numpy(), ref) <= 1e-4
