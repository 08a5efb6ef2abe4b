"""Context sums of blocks without a qkv conv, through the gates of whole blocks against the oracle: channel counts below, at and
above a warp's 128 channels and counts that leave lanes idle, rows shorter and longer than one trip, one source frame for
several steps."""
import numpy as np
import pytest
import torch

from cssm_b200 import GatedDeltaNetCSSM, SimpleCSSM
from oracle import cssm_oracle as orc
from oracle import simple_oracle as so

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,T,H,W,C", [(1, 1, 7, 2, 4), (2, 3, 8, 9, 12), (1, 2, 8, 33, 48), (2, 2, 9, 16, 80), (1, 3, 8, 8, 128), (1, 2, 7, 20, 160)])
@pytest.mark.parametrize("mode", ["none", "mrope"])
def test_rowsum_shapes(B, T, H, W, C, mode):
    kw = dict(delta_key_dim=4, kernel_size=1, gate_type="factored", qkv_conv_size=1)
    x = np.random.default_rng(C + W).standard_normal((B, T, H, W, C)).astype(np.float32)
    p = orc.init_gdn_params(3, C, H, W, bias_scale=0.1, **kw)
    ref = orc.gdn_forward(p, x, rope_mode=mode, **kw)
    m = GatedDeltaNetCSSM(channels=C, rope_mode=mode, **kw)
    got = m.apply({"params": p}, torch.from_numpy(x).cuda()).cpu().numpy()
    assert orc.rel_l2(got, ref) <= 1e-4


@pytest.mark.parametrize("mode", ["none", "mrope", "temporal"])
def test_one_source_frame_for_all_steps(mode):
    kw = dict(delta_key_dim=4, qkv_conv_size=1)
    m = SimpleCSSM(cssm_type="gdn", embed_dim=32, kernel_size=1, gate_type="factored", seq_len=5, pos_embed=mode, stem_layers=1,
                   pool_type="max", **kw)
    x = np.random.default_rng(0).random((2, 24, 36, 1)).astype(np.float32)
    H, W = m.feature_hw(24, 36)
    bkw = dict(kernel_size=1, rope_mode=mode, gate_type="factored", short_conv_size=4, **kw)
    p = so.init_simple_params(5, cin=1, embed_dim=32, H=H, W=W, num_classes=2, cssm_type="gdn", stem_mode="default", stem_layers=1,
                              bias_scale=0.1, block_kwargs=bkw)
    ref = so.simple_forward(p, x, cssm_type="gdn", seq_len=5, stem_mode="default", stem_layers=1, pool_type="max", block_kwargs=bkw)
    got = m.bind({"params": p})(torch.from_numpy(x).cuda()).cpu().numpy()
    assert orc.rel_l2(got, ref) <= 1e-4
