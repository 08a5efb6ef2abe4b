"""The 64-channel float32 projections on planes of whole 128-pixel tiles (csrc/gemm_tc.cu: raw tiles by TMA, A in TMEM): each form of the
input (rows with and without rotation, its angles from shared memory or per lane; planes, gated, RMS-normalised) and of the output
against the oracle."""
import numpy as np
import pytest
import torch

from cssm_b200 import AdditiveCSSM, DeltaNetCSSM, GatedCSSM, GatedDeltaNetCSSM, device_error
from oracle import cssm_oracle as orc

pytestmark = pytest.mark.gpu

# image rows of 16, 32 and 64 pixels (angles in shared memory), of 8, 24, 48 and 128 (per lane), one and several tiles a frame
PLANES = [(8, 16), (4, 32), (2, 64), (16, 8), (16, 24), (8, 48), (2, 128), (64, 64)]


def _rel(mod, p, x, ref, **kw):
    got = mod.bind({"params": p})(torch.from_numpy(x).cuda(), **kw).cpu().numpy()
    assert device_error() == 0
    return orc.rel_l2(got, ref)


@pytest.mark.parametrize("H,W", PLANES)
@pytest.mark.parametrize("rope", ["none", "spatiotemporal", "mrope"])
def test_blocks(H, W, rope):
    """3 x TF32 products are 2^-21 off a product; the blocks' bound against the oracle is 1e-4 throughout."""
    B, T = (1, 2) if H * W > 1024 else (2, 3)
    x = np.random.default_rng(H + W).standard_normal((B, T, H, W, 64)).astype(np.float32)
    p = orc.init_gated_params(1, 64, H, W, kernel_size=1, gate_type="factored", bias_scale=0.1)
    kw = dict(kernel_size=1, gate_type="factored", rope_mode=rope)
    ref, m = orc.gated_forward(p, x, **kw), GatedCSSM(channels=64, **kw)
    assert _rel(m, p, x, ref) <= 1e-4
    assert _rel(m, p, x, ref[:, -1], last_frame_only=True) <= 1e-4
    p = orc.init_gdn_params(2, 64, H, W, delta_key_dim=4, kernel_size=1, qkv_conv_size=1, bias_scale=0.1, perturb_rms=True)
    kw = dict(delta_key_dim=4, kernel_size=1, qkv_conv_size=1, rope_mode=rope)
    ref, m = orc.gdn_forward(p, x, **kw), GatedDeltaNetCSSM(channels=64, gate_type="factored", **kw)
    assert _rel(m, p, x, ref) <= 1e-4
    assert _rel(m, p, x, ref[:, -1], last_frame_only=True) <= 1e-4
    kw = dict(kernel_size=1, gate_type="channel", rope_mode=rope)
    p = orc.init_deltanet_params(3, 64, H, W, kernel_size=1, gate_type="channel", bias_scale=0.1)
    assert _rel(DeltaNetCSSM(channels=64, **kw), p, x, orc.deltanet_forward(p, x, **kw)) <= 1e-4
    p = orc.init_additive1_params(4, 64, H, W, kernel_size=1, gate_type="channel", bias_scale=0.1)
    assert _rel(AdditiveCSSM(single_state=True, channels=64, **kw), p, x, orc.additive1_forward(p, x, **kw)) <= 1e-4


@pytest.mark.parametrize("tiles", [1, 147, 149, 700])
def test_tiles_per_cta(tiles):
    """Fewer tiles than SMs, one round and a few more, several rounds: equal clips give equal outputs wherever their tiles run."""
    p = orc.init_gdn_params(5, 64, 8, 16, delta_key_dim=4, kernel_size=1, qkv_conv_size=1, bias_scale=0.1)
    m = GatedDeltaNetCSSM(channels=64, delta_key_dim=4, kernel_size=1, qkv_conv_size=1, rope_mode="mrope", gate_type="factored").bind({"params": p})
    x = torch.from_numpy(np.random.default_rng(7).standard_normal((1, 5, 8, 16, 64)).astype(np.float32)).cuda()
    n = -(-tiles // 5)
    one = m(x).clone()
    many = m(x.expand(n, -1, -1, -1, -1).contiguous())
    assert torch.equal(many, many[:1].expand_as(many))
    # (few clips take the projection and the temporal conv in two launches)
    assert (many[0] - one[0]).norm() <= 5e-6 * one.norm()
    assert device_error() == 0


@pytest.mark.parametrize("scale", [1e-10, 1e4, 1e8])
def test_scaled_rows(scale):
    """The RMS row factor meets the products, not the values: rows far from 1 give what the oracle gives."""
    kw = dict(delta_key_dim=4, kernel_size=1, qkv_conv_size=1, rope_mode="none")
    p = orc.init_gdn_params(6, 64, 8, 16, delta_key_dim=4, kernel_size=1, qkv_conv_size=1, bias_scale=0.1)
    x = np.random.default_rng(8).standard_normal((1, 2, 8, 16, 64)).astype(np.float32) * np.float32(scale)
    assert _rel(GatedDeltaNetCSSM(channels=64, gate_type="factored", **kw), p, x, orc.gdn_forward(p, x, **kw)) <= 1e-4
