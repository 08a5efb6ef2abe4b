"""q, k, v projection and temporal conv in one launch (csrc/gemm_qkv_tconv.cu: 64 channels, planes of whole 128-pixel tiles, two
sequences for three SMs and more or up to four steps) against the block on fewer clips, which from five steps on goes through the two
launches, and against the oracle."""
import numpy as np
import pytest
import torch

from cssm_b200 import GatedDeltaNetCSSM, device_error
from oracle import cssm_oracle as orc

pytestmark = pytest.mark.gpu


# one step to more than the accumulator ring holds, each tap count, sequences that do not divide among the CTAs
@pytest.mark.parametrize("kt,T", [(4, 1), (4, 2), (4, 3), (4, 4), (4, 5), (4, 6), (4, 11), (1, 3), (2, 5), (3, 6)])
@pytest.mark.parametrize("gate,inputs,B,H,W", [("factored", True, 19, 32, 32), ("factored", False, 27, 24, 32), ("channel", True, 21, 32, 32),
                                               ("dense", True, 150, 8, 16)])
def test_joined_launch(kt, T, gate, inputs, B, H, W):
    """Both sides are 3 x TF32 products (2^-21 a product) and the same float32 chain behind them; the oracle's bound is that of the block's
    other tests."""
    kw = dict(delta_key_dim=4, kernel_size=3, gate_type=gate, short_conv_size=kt, use_input_gates=inputs)
    x = np.random.default_rng(10 * T + kt).standard_normal((B, T, H, W, 64)).astype(np.float32)
    p = orc.init_gdn_params(kt, 64, H, W, bias_scale=0.1, **kw)
    m = GatedDeltaNetCSSM(channels=64, rope_mode="mrope", qkv_conv_size=1, **kw).bind({"params": p})
    xd = torch.from_numpy(x).cuda()
    got = m(xd).clone()
    last = m(xd, last_frame_only=True).clone()
    few = torch.cat([m(xd[i:i + 1].contiguous()).clone() for i in range(B)])
    assert orc.rel_l2(got.cpu().numpy(), few.cpu().numpy()) <= 5e-6
    assert orc.rel_l2(last.cpu().numpy(), few[:, -1].cpu().numpy()) <= 5e-6
    pick = [0, B - 1]
    ref = orc.gdn_forward(p, x[pick], rope_mode="mrope", qkv_conv_size=1, **kw)
    assert orc.rel_l2(got[pick].cpu().numpy(), ref) <= 1e-4
    assert device_error() == 0


@pytest.mark.parametrize("kt", [1, 2, 3])
@pytest.mark.parametrize("T", [5, 7])
def test_fewer_taps_above_four_steps(kt, T):
    """Each tap count against the two launches (up to four steps the joined one takes any number of clips)."""
    kw = dict(delta_key_dim=4, kernel_size=3, gate_type="factored", short_conv_size=kt)
    x = torch.from_numpy(np.random.default_rng(T + kt).standard_normal((20, T, 32, 32, 64)).astype(np.float32)).cuda()
    m = GatedDeltaNetCSSM(channels=64, rope_mode="mrope", qkv_conv_size=1, **kw).bind({"params": orc.init_gdn_params(kt, 64, 32, 32, bias_scale=0.1, **kw)})
    got = m(x).clone()
    few = torch.cat([m(x[i:i + 1].contiguous()).clone() for i in range(20)])
    assert orc.rel_l2(got.cpu().numpy(), few.cpu().numpy()) <= 5e-6
    assert device_error() == 0


@pytest.mark.parametrize("kt,T", [(4, 1), (4, 2), (4, 3), (4, 4), (3, 4), (2, 4), (1, 3), (3, 2), (2, 1)])
@pytest.mark.parametrize("B,H,W", [(1, 8, 16), (30, 16, 16)])
def test_few_steps_against_float64(kt, T, B, H, W):
    """Up to four steps: the q and k planes that the launch leaves.  Products off by 2^-22 at most and the accumulator's eight truncations
    (3.3e-7 together, tests/test_tc_projections_gpu.py), SiLU and four taps of float32 FMAs."""
    m = GatedDeltaNetCSSM(channels=64, delta_key_dim=4, kernel_size=3, rope_mode="none", qkv_conv_size=1, gate_type="factored",
                          short_conv_size=kt, use_input_gates=False)
    x = torch.randn((B, T, H, W, 64), device="cuda", generator=torch.Generator(device="cuda").manual_seed(T + kt))
    v = m.init(3, tuple(x.shape), bias_scale=0.3)
    b, p = m.bind(v), v["params"]
    b(x)
    f64 = lambda a: torch.from_numpy(np.asarray(a, np.float64)).cuda()
    qkv = b.buf.get("ws", 0).view(torch.float32)[:3 * x.numel()].view(B, T, 192, H, W)
    s = x.double() @ f64(p["qkv_proj"]["kernel"]) + f64(p["qkv_proj"]["bias"])
    for i, name in enumerate("qk"):
        c = p[f"short_conv_{name}"]
        k = f64(c["kernel"]).reshape(kt, 64)
        past = torch.nn.functional.pad(s[..., i * 64:(i + 1) * 64], (0, 0) * 3 + (kt - 1, 0))
        want = torch.nn.functional.silu(sum(past[:, j:j + T] * k[j] for j in range(kt)) + f64(c["bias"])).permute(0, 1, 4, 2, 3)
        assert float((qkv[:, :, i * 64:(i + 1) * 64].double() - want).norm() / want.norm()) < 5e-7
    assert device_error() == 0


@pytest.mark.parametrize("rope", ["none", "spatiotemporal"])
@pytest.mark.parametrize("conv", [1, 3])
def test_input_forms(rope, conv):
    """Rotated rows or not; rows of the input or of the depthwise conv; a second call over the same buffers."""
    kw = dict(delta_key_dim=2, kernel_size=3, gate_type="factored", qkv_conv_size=conv)
    x = np.random.default_rng(conv).standard_normal((20, 3, 32, 32, 64)).astype(np.float32)
    p = orc.init_gdn_params(9, 64, 32, 32, bias_scale=0.1, **kw)
    m = GatedDeltaNetCSSM(channels=64, rope_mode=rope, **kw).bind({"params": p})
    xd = torch.from_numpy(x).cuda()
    got = m(xd).clone()
    assert torch.equal(got, m(xd))
    ref = orc.gdn_forward(p, x[[0, 19]], rope_mode=rope, **kw)
    assert orc.rel_l2(got[[0, 19]].cpu().numpy(), ref) <= 1e-4


def test_image_held_for_several_frames():
    """A model that holds one image for all frames reads every frame's rows from it."""
    from cssm_b200 import SimpleCSSM
    from oracle import simple_oracle as so
    kw = dict(delta_key_dim=4, kernel_size=3, gate_type="factored")
    m = SimpleCSSM(cssm_type="gdn", embed_dim=64, seq_len=5, pos_embed="spatiotemporal", stem_layers=1, pool_type="max", **kw)
    x = np.random.default_rng(2).random((20, 64, 64, 1)).astype(np.float32)
    H, W = m.feature_hw(64, 64)
    assert H * W % 128 == 0 and 2 * 20 * H * W // 128 >= 296
    bkw = dict(kw, rope_mode="spatiotemporal")
    p = so.init_simple_params(5, cin=1, embed_dim=64, H=H, W=W, num_classes=2, cssm_type="gdn", stem_mode="default", stem_layers=1,
                              bias_scale=0.1, block_kwargs=bkw)
    b = m.bind({"params": p})
    xd = torch.from_numpy(x).cuda()
    got = b(xd).cpu().numpy()
    few = np.concatenate([b(xd[i:i + 1]).cpu().numpy() for i in range(20)])
    ref = so.simple_forward(p, x[:2], cssm_type="gdn", seq_len=5, stem_mode="default", stem_layers=1, pool_type="max", block_kwargs=bkw)
    assert orc.rel_l2(got, few) <= 1e-5
    assert orc.rel_l2(got[:2], ref) <= 1e-4


@pytest.mark.parametrize("kt", [1, 2, 3])
def test_frames_behind_the_taps(kt):
    """A channel that q alone reads overflows in frame 0: q of frames 0 .. kt - 1 is not finite, and from frame kt on nothing may remember it."""
    kw = dict(delta_key_dim=4, kernel_size=3, gate_type="factored", short_conv_size=kt)
    B, T, c = 37, 6, 5
    x = np.random.default_rng(kt).standard_normal((B, T, 32, 32, 64)).astype(np.float32)
    p = orc.init_gdn_params(kt, 64, 32, 32, bias_scale=0.1, **kw)
    for name, leaf in p.items():
        if isinstance(leaf, dict) and "kernel" in leaf and leaf["kernel"].ndim == 2 and leaf["kernel"].shape[0] == 64 and name != "output_proj":
            w = np.array(leaf["kernel"])
            w[c] = 0
            if name == "qkv_proj":
                w[c, :64] = 100
            leaf["kernel"] = w
    x[:, 0, :, :, c] = 0
    m = GatedDeltaNetCSSM(channels=64, rope_mode="none", qkv_conv_size=1, **kw).bind({"params": p})
    want = m(torch.from_numpy(x).cuda()).clone()
    x[:, 0, 3, 7, c] = 1e38
    got = m(torch.from_numpy(x).cuda())
    assert bool(want.isfinite().all())
    assert not bool(got[:, 0].isfinite().all())
    assert torch.equal(got[:, kt:], want[:, kt:])
    assert device_error() == 0
