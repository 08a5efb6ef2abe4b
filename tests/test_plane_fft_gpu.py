"""Square planes whose FFTs are whole in a lane's registers (csrc/gated_spectral_fft.cu, csrc/delta_spectral_fft.cuh): every side that is built,
ragged groups of planes and heads, batches of frames with some missing, one frame, one, two and four frames a CTA, and states in shared and in
global memory, against the float64 oracle.

Tolerance: a transform is at most six levels of butterflies or one direct sum of at most 23 terms with exactly rounded twiddles, so each of the
four nested ones is within 23 * 2^-24 (1.4e-6) of its norm at worst and some 2e-7 as a random walk; with a recurrence over a few
steps, the norms of the delta rules one division more, below 5e-6 of the 2-norm, checked at 1e-5."""
import numpy as np
import pytest
import torch

from oracle import cssm_oracle as orc
from cssm_b200 import AdditiveCSSM, DeltaNetCSSM, GatedCSSM, GatedDeltaNetCSSM, NoGateCSSM

pytestmark = pytest.mark.gpu
TOL = 1e-5
SIDES = [*range(5, 29), 30, 33, 34, 35, 36, 38, 39, 40, 42, 44, 45, 48, 49, 50, 52, 54, 55, 56, 60]


def _check(got, ref):
    got = got.cpu().numpy()
    assert np.isfinite(got).all()
    assert orc.rel_l2(got, ref) <= TOL


def _gated(B, T, n, C, gate, seed=0):
    rng = np.random.default_rng(100 * n + T + seed)
    x = rng.standard_normal((B, T, n, n, C)).astype(np.float32)
    kw = dict(kernel_size=min(5, n), rope_mode="none", gate_type=gate)
    p = orc.init_gated_params(1, C, n, n, bias_scale=0.1, kernel_size=kw["kernel_size"], gate_type=gate)
    p["kernel"] = (0.3 * rng.standard_normal(p["kernel"].shape)).astype(np.float32)      # so that the recurrence matters
    b = GatedCSSM(channels=C, **kw).bind({"params": p})
    ref = orc.gated_forward(p, x, **kw)
    xd = torch.from_numpy(x).cuda()
    _check(b(xd), ref)
    _check(b(xd, last_frame_only=True), ref[:, -1])
    return x, xd


@pytest.mark.parametrize("n", SIDES)
def test_sides(n):
    _gated(1, 5, n, 12, "dense")
    x, xd = _gated(2, 2, n, 20, "factored")
    p = NoGateCSSM(channels=20, kernel_size=3).init(2, x.shape, bias_scale=0.1)["params"]
    p["kernel"] = (0.3 * np.random.default_rng(n).standard_normal(p["kernel"].shape)).astype(np.float32)
    _check(NoGateCSSM(channels=20, kernel_size=3).apply({"params": p}, xd), orc.nogate_forward(p, x, kernel_size=3))
    for gate in ("factored", "channel"):
        kw = dict(kernel_size=1, rope_mode="none", gate_type=gate)
        p = orc.init_additive1_params(3, 20, n, n, kernel_size=1, gate_type=gate, bias_scale=0.1)
        _check(AdditiveCSSM(channels=20, single_state=True, **kw).apply({"params": p}, xd), orc.additive1_forward(p, x, **kw))


# one frame: planes for every SM; many planes: CTAs of one and two frames, several rounds, a last group of fewer planes
@pytest.mark.parametrize("B,T,n,C", [(40, 1, 8, 24), (60, 1, 7, 24), (60, 1, 14, 12), (30, 1, 28, 12), (40, 1, 56, 4), (200, 3, 8, 52),
                                     (300, 2, 7, 36), (37, 3, 20, 20), (75, 3, 14, 36), (20, 3, 40, 36), (19, 2, 56, 32), (54, 3, 16, 48)])
def test_batches(B, T, n, C):
    _gated(B, T, n, C, "factored")


def _gdn(B, T, n, C, dk, gate, **kw):
    rng = np.random.default_rng(100 * n + T + dk)
    x = rng.standard_normal((B, T, n, n, C)).astype(np.float32)
    kw = dict(delta_key_dim=dk, kernel_size=min(5, n), rope_mode="none", gate_type=gate, **kw)
    p = orc.init_gdn_params(1, C, n, n, bias_scale=0.1, perturb_rms=True, **{k: kw[k] for k in kw if k not in ("rope_mode", "use_spectral_l2_norm")})
    b = GatedDeltaNetCSSM(channels=C, **kw).bind({"params": p})
    ref = orc.gdn_forward(p, x, **kw)
    xd = torch.from_numpy(x).cuda()
    _check(b(xd), ref)
    _check(b(xd, last_frame_only=True), ref[:, -1])


def _deltanet(B, T, n, C, gate):
    rng = np.random.default_rng(100 * n + T)
    x = rng.standard_normal((B, T, n, n, C)).astype(np.float32)
    kw = dict(kernel_size=min(5, n), rope_mode="none", gate_type=gate)
    p = orc.init_deltanet_params(3, C, n, n, kernel_size=kw["kernel_size"], gate_type=gate, bias_scale=0.1)
    _check(DeltaNetCSSM(channels=C, **kw).apply({"params": p}, torch.from_numpy(x).cuda()), orc.deltanet_forward(p, x, **kw))


@pytest.mark.parametrize("n", SIDES)
def test_delta_rule_sides(n):
    _gdn(1, 3, n, 20, 2, "dense")
    _gdn(1, 2, n, 24, 4, "channel")
    _deltanet(1, 3, n, 12, "channel")
    _deltanet(2, 2, n, 8, "factored")


# one frame; several heads a CTA with a last group of fewer; warps with one and with all of q, k, v; states in global memory
@pytest.mark.parametrize("B,T,n,C", [(150, 1, 7, 20), (90, 2, 8, 36), (60, 3, 14, 36), (300, 2, 5, 12), (40, 1, 28, 12), (9, 3, 48, 16), (2, 3, 56, 8)])
def test_delta_rule_batches(B, T, n, C):
    for dk in (2, 4):
        _gdn(B, T, n, C, dk, "factored")
    _deltanet(B, T, n, C, "dense")
