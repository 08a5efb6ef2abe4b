"""The 64-channel float32 projections on planes of whole 128-pixel tiles (csrc/gemm_tc.cu: raw tiles by TMA, A in TMEM): each form of the
input (rows with and without rotation, its angles from shared memory or per lane; planes, gated, RMS-normalised) and of the output
against the oracle."""
import ctypes as C

import numpy as np
import pytest
import torch

from cssm_b200 import AdditiveCSSM, DeltaNetCSSM, GatedCSSM, GatedDeltaNetCSSM, device_error
from cssm_b200._lib import check
from oracle import cssm_oracle as orc

pytestmark = pytest.mark.gpu

# image rows of 16, 32 and 64 pixels (angles in shared memory), of 8, 24, 48 and 128 (per lane), one and several tiles a frame
PLANES = [(8, 16), (4, 32), (2, 64), (16, 8), (16, 24), (8, 48), (2, 128), (64, 64)]


f64 = lambda a: torch.from_numpy(np.asarray(a, np.float64)).cuda()


def _rel(mod, p, x, ref, **kw):
    got = mod.bind({"params": p})(torch.from_numpy(x).cuda(), **kw).cpu().numpy()
    assert device_error() == 0
    return orc.rel_l2(got, ref)


def _unbiased(p, name):
    """The output projection's bias outweighs what the block computes: without it a projection that lost its remainder products is off by
    2e-4 of the block's output (the weights rounded to TF32 in the oracle), each of them."""
    p[name] = {"kernel": p[name]["kernel"], "bias": np.zeros_like(p[name]["bias"])}
    return p


@pytest.mark.parametrize("H,W", PLANES)
@pytest.mark.parametrize("rope", ["none", "spatiotemporal", "mrope"])
def test_blocks(H, W, rope):
    """Blocks measure 0.4e-6 to 2e-6 against the oracle: float32 transforms and recurrences, 3 x TF32 projections at 0.2e-6."""
    B, T = (1, 2) if H * W > 1024 else (2, 3)
    x = np.random.default_rng(H + W).standard_normal((B, T, H, W, 64)).astype(np.float32)
    p = _unbiased(orc.init_gated_params(1, 64, H, W, kernel_size=1, gate_type="factored", bias_scale=0.1), "out_proj")
    kw = dict(kernel_size=1, gate_type="factored", rope_mode=rope)
    ref, m = orc.gated_forward(p, x, **kw), GatedCSSM(channels=64, **kw)
    assert _rel(m, p, x, ref) <= 5e-6
    assert _rel(m, p, x, ref[:, -1], last_frame_only=True) <= 5e-6
    p = _unbiased(orc.init_gdn_params(2, 64, H, W, delta_key_dim=4, kernel_size=1, qkv_conv_size=1, bias_scale=0.1, perturb_rms=True),
                  "output_proj")
    kw = dict(delta_key_dim=4, kernel_size=1, qkv_conv_size=1, rope_mode=rope)
    ref, m = orc.gdn_forward(p, x, **kw), GatedDeltaNetCSSM(channels=64, gate_type="factored", **kw)
    assert _rel(m, p, x, ref) <= 5e-6
    assert _rel(m, p, x, ref[:, -1], last_frame_only=True) <= 5e-6
    kw = dict(kernel_size=1, gate_type="channel", rope_mode=rope)
    p = _unbiased(orc.init_deltanet_params(3, 64, H, W, kernel_size=1, gate_type="channel", bias_scale=0.1), "output_proj")
    assert _rel(DeltaNetCSSM(channels=64, **kw), p, x, orc.deltanet_forward(p, x, **kw)) <= 5e-6
    p = _unbiased(orc.init_additive1_params(4, 64, H, W, kernel_size=1, gate_type="channel", bias_scale=0.1), "output_proj")
    assert _rel(AdditiveCSSM(single_state=True, channels=64, **kw), p, x, orc.additive1_forward(p, x, **kw)) <= 5e-6


# The dropped products are below 2^-22 of |a||b|; the accumulator truncates at each of the eight leading MMAs, half of 2^-23 of the sum so far,
# which averages 0.56 of the last: at most 8 (0.56) 2^-24 + 2^-22 / 4 = 3.3e-7 if all went one way.  SiLU and the angles' table values
# (float32, two products of them) come on top.
STAGE = 5e-7


def _off(got, want):
    return float((got.double() - want).norm() / want.norm())


@pytest.mark.parametrize("H,W", PLANES)
@pytest.mark.parametrize("rope", ["none", "spatiotemporal", "mrope"])
def test_stages(H, W, rope):
    """The launches by themselves against float64: 64 -> 128 with SiLU on half of the columns, planes -> 64 without a gate, 64 -> 64 with SiLU,
    64 -> 192, alone and with the temporal conv behind it."""
    B, T, Cc = 2, 2, 64
    xd = torch.randn((B, T, H, W, Cc), device="cuda", generator=torch.Generator(device="cuda").manual_seed(H * W))
    xr = f64(orc.apply_rope(xd.double().cpu().numpy(), rope))
    planes = lambda a: a.reshape(B * T, H * W, -1).permute(0, 2, 1)
    lin = lambda a, q: a @ f64(q["kernel"]) + f64(q["bias"])
    silu = torch.nn.functional.silu
    m = GatedCSSM(channels=Cc, kernel_size=1, gate_type="factored", rope_mode=rope)
    v = m.init(5, tuple(xd.shape), bias_scale=0.3)
    b, p = m.bind(v), v["params"]
    xz = b.stages(xd, upto="in_proj")["xz"].reshape(B * T, 2 * Cc, H * W)
    want = planes(lin(xr, p["in_proj"]))
    assert _off(xz[:, :Cc], want[:, :Cc]) < STAGE
    assert _off(xz[:, Cc:], silu(want[:, Cc:])) < STAGE
    d = b.desc(tuple(xd.shape))
    y = torch.full_like(xd, float("nan"))
    check(b.L.cssm_gated_out_proj(C.byref(d), C.byref(b.w), b.buf.get("ws", 0).data_ptr() + b.workspace_layout(d).xz_planar, y.data_ptr(),
                                  torch.cuda.current_stream().cuda_stream), "out_proj")
    assert _off(y.reshape(B * T, H * W, Cc), lin(xz[:, :Cc].double().permute(0, 2, 1), p["out_proj"])) < STAGE

    for taps in (0, 4):
        m = GatedDeltaNetCSSM(channels=Cc, delta_key_dim=4, kernel_size=1, qkv_conv_size=1, rope_mode=rope, gate_type="factored",
                              output_gate_act="silu", use_input_gates=False, short_conv_size=taps)
        v = m.init(6, tuple(xd.shape), bias_scale=0.3)
        b, p = m.bind(v), v["params"]
        b(xd)
        n = B * T * Cc * H * W                 # workspace: q, k, v planes of every frame (v overwritten by the readout), gate planes
        ws = b.buf.get("ws", 0).view(torch.float32)
        qkv, gate = ws[:3 * n].view(B * T, 3 * Cc, H * W), ws[3 * n:4 * n].view(B * T, Cc, H * W)
        assert _off(gate, silu(planes(lin(xr, p["gate_proj"])))) < STAGE
        want = lin(xr, p["qkv_proj"])
        for i, name in enumerate("qk"):
            w = want[..., i * Cc:(i + 1) * Cc]
            if taps:
                q = p[f"short_conv_{name}"]
                k, past = f64(q["kernel"]).reshape(taps, Cc), torch.nn.functional.pad(w, (0, 0) * 3 + (taps - 1, 0))
                w = silu(sum(past[:, j:j + T] * k[j] for j in range(taps)) + f64(q["bias"]))
            assert _off(qkv[:, i * Cc:(i + 1) * Cc], planes(w)) < STAGE, (taps, name)
    assert device_error() == 0


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


@pytest.mark.parametrize("scale", [1e-3, 1e-2, 1e4, 1e8])
def test_scaled_rows(scale):
    """The RMS row factor meets the products, not the values: rows whose mean square is below, near and far above its 1e-6, without
    biases beside which they would not show."""
    kw = dict(delta_key_dim=4, kernel_size=1, qkv_conv_size=1, rope_mode="none")
    p = orc.init_gdn_params(6, 64, 8, 16, delta_key_dim=4, kernel_size=1, qkv_conv_size=1, bias_scale=0.0)
    x = np.random.default_rng(8).standard_normal((1, 2, 8, 16, 64)).astype(np.float32) * np.float32(scale)
    assert _rel(GatedDeltaNetCSSM(channels=64, gate_type="factored", **kw), p, x, orc.gdn_forward(p, x, **kw)) <= 5e-6
