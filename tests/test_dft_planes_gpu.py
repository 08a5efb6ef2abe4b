"""The folded-DFT spectral kernels (planes without a radix kernel) at the sizes where they can go wrong:
one-pixel, odd, even, prime and unequal sides, channel counts that leave a ragged plane group, T = 1 (no
state), and a plane too long for the tables (direct-DFT kernel), against the float64 oracle.

Tolerance: a plane value is four nested sums of at most 50 terms with exactly rounded twiddles, each
within sqrt(50) * 2^-24 of its norm (4e-7); the recurrence over at most three steps adds its own few
roundings, the norms of the delta rules one division: below 5e-6 of the 2-norm, checked at 1e-5."""
import numpy as np
import pytest
import torch

from oracle import cssm_oracle as orc
from cssm_b200 import AdditiveCSSM, DeltaNetCSSM, GatedCSSM, GatedDeltaNetCSSM, NoGateCSSM

pytestmark = pytest.mark.gpu
TOL = 1e-5
SIZES = [(1, 1, 1, 7, 4), (2, 3, 2, 3, 4), (1, 2, 5, 4, 8), (3, 1, 7, 7, 20), (2, 3, 8, 13, 12), (1, 3, 14, 14, 68),
         (2, 2, 16, 15, 8), (1, 2, 29, 31, 12), (1, 2, 50, 56, 8), (1, 2, 33, 90, 4), (1, 2, 2, 700, 4)]


def _check(got, ref):
    got = got.cpu().numpy()
    assert np.isfinite(got).all()
    assert orc.rel_l2(got, ref) <= TOL


@pytest.mark.parametrize("B,T,H,W,C", SIZES)
def test_gated_family(B, T, H, W, C):
    rng = np.random.default_rng(H * 100 + W)
    x = rng.standard_normal((B, T, H, W, C)).astype(np.float32)
    xd = torch.from_numpy(x).cuda()
    kw = dict(kernel_size=1, rope_mode="none", gate_type="factored")
    p = orc.init_gated_params(1, C, H, W, bias_scale=0.1, kernel_size=1, gate_type="factored")
    b = GatedCSSM(channels=C, **kw).bind({"params": p})
    ref = orc.gated_forward(p, x, **kw)
    _check(b(xd), ref)
    _check(b(xd, last_frame_only=True), ref[:, -1])
    m = NoGateCSSM(channels=C, kernel_size=1)
    p = m.init(2, x.shape, bias_scale=0.1)["params"]
    _check(m.apply({"params": p}, xd), orc.nogate_forward(p, x, kernel_size=1))
    kw["gate_type"] = "channel"
    p = orc.init_additive1_params(3, C, H, W, kernel_size=1, gate_type="channel", bias_scale=0.1)
    _check(AdditiveCSSM(channels=C, single_state=True, **kw).apply({"params": p}, xd), orc.additive1_forward(p, x, **kw))


@pytest.mark.parametrize("dk", [1, 2, 4])
@pytest.mark.parametrize("B,T,H,W,C", SIZES)
def test_delta_rules(B, T, H, W, C, dk):
    rng = np.random.default_rng(H * 100 + W + dk)
    x = rng.standard_normal((B, T, H, W, C)).astype(np.float32)
    xd = torch.from_numpy(x).cuda()
    kw = dict(delta_key_dim=dk, kernel_size=1, rope_mode="none", gate_type="factored")
    p = orc.init_gdn_params(1, C, H, W, bias_scale=0.1, perturb_rms=True, **{k: kw[k] for k in kw if k != "rope_mode"})
    b = GatedDeltaNetCSSM(channels=C, **kw).bind({"params": p})
    ref = orc.gdn_forward(p, x, **kw)
    _check(b(xd), ref)
    _check(b(xd, last_frame_only=True), ref[:, -1])
    if dk == 1:
        kw = dict(kernel_size=1, rope_mode="none", gate_type="dense" if H % 2 else "channel")
        p = orc.init_deltanet_params(3, C, H, W, kernel_size=1, gate_type=kw["gate_type"], bias_scale=0.1)
        _check(DeltaNetCSSM(channels=C, **kw).apply({"params": p}, xd), orc.deltanet_forward(p, x, **kw))


# Batches that fill the GPU, where the passes take the larger register tiles (1 x 4, 2 x 4 and 1 x 8 cells): two clips over and
# over, so that the oracle has two to do and every plane group of the batch has to repeat them.
@pytest.mark.parametrize("kind,B,T,H,W,C", [("gated", 16, 2, 56, 56, 32), ("gated", 33, 1, 16, 16, 256), ("gated", 40, 2, 24, 24, 64),
                                            ("gated", 12, 2, 28, 28, 64), ("gated", 9, 1, 51, 43, 64), ("delta", 16, 2, 28, 28, 64),
                                            ("delta", 9, 2, 47, 45, 32), ("delta", 33, 1, 14, 14, 64)])
def test_full_batches(kind, B, T, H, W, C):
    x = np.random.default_rng(H + W + C).standard_normal((2, T, H, W, C)).astype(np.float32)
    idx = np.arange(B) % 2
    xd = torch.from_numpy(x[idx]).cuda()
    kw = dict(kernel_size=1, rope_mode="none", gate_type="factored")
    if kind == "gated":
        p = orc.init_gated_params(1, C, H, W, bias_scale=0.1, kernel_size=1, gate_type="factored")
        _check(GatedCSSM(channels=C, **kw).apply({"params": p}, xd), orc.gated_forward(p, x, **kw)[idx])
    else:
        p = orc.init_gdn_params(1, C, H, W, bias_scale=0.1, perturb_rms=True, delta_key_dim=2, kernel_size=1, gate_type="factored")
        _check(GatedDeltaNetCSSM(channels=C, delta_key_dim=2, **kw).apply({"params": p}, xd),
               orc.gdn_forward(p, x, delta_key_dim=2, **kw)[idx])


@pytest.mark.parametrize("B,T,H,W,C,dk", [(31, 2, 39, 39, 32, 4), (9, 1, 28, 28, 48, 3), (40, 2, 16, 8, 64, 4), (7, 3, 47, 22, 24, 3), (2, 2, 58, 34, 64, 4)])
def test_full_batches_of_long_keys(B, T, H, W, C, dk):
    """Key dimension 3 and 4, whose tiles have an estimate of their own: one CTA of eight warps an SM, and several."""
    x = np.random.default_rng(H + W + C).standard_normal((min(B, 2), T, H, W, C)).astype(np.float32)
    idx = np.arange(B) % len(x)
    kw = dict(kernel_size=1, rope_mode="none", gate_type="factored", delta_key_dim=dk)
    p = orc.init_gdn_params(1, C, H, W, bias_scale=0.1, perturb_rms=True, kernel_size=1, gate_type="factored", delta_key_dim=dk)
    _check(GatedDeltaNetCSSM(channels=C, **kw).apply({"params": p}, torch.from_numpy(x[idx]).cuda()), orc.gdn_forward(p, x, **kw)[idx])
