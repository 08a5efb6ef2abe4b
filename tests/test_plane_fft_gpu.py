"""The gated family on square planes whose FFTs are whole in a lane's registers (csrc/gated_spectral_fft.cu): every side that is built, ragged
groups of planes, batches of frames with some missing, one frame, and one, two and four frames a CTA, against the float64 oracle.

Tolerance: a transform is at most six levels of butterflies or one direct sum of at most 23 terms with exactly rounded twiddles, so each of the
four nested ones is within 23 * 2^-24 (1.4e-6) of its norm at worst and some 2e-7 as a random walk; with a recurrence over a few
steps below 5e-6 of the 2-norm, checked at 1e-5."""
import numpy as np
import pytest
import torch

from oracle import cssm_oracle as orc
from cssm_b200 import AdditiveCSSM, GatedCSSM, NoGateCSSM

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
                                     (300, 2, 7, 36), (37, 3, 20, 20), (75, 3, 14, 36), (20, 3, 40, 36), (19, 2, 56, 32)])
def test_batches(B, T, n, C):
    _gated(B, T, n, C, "factored")
