"""GPU parity of the DeltaNetCSSM block through the C ABI against the NumPy oracle.
Tolerance: rel-L2 <= 1e-4 in fp32.  The output bias is zero in these cases: the block's signal
(normalised q and k) is two orders below a 0.1-scale bias, which would hide errors."""
import os

import numpy as np
import pytest
import torch

from oracle import cssm_oracle as orc
from cssm_b200 import DeltaNetCSSM

pytestmark = pytest.mark.gpu
TOL = 1e-4


def _run(case, gate_type, rope, scan_mode="associative", seed=0):
    B, T, H, W, C, ks = case
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((B, T, H, W, C)).astype(np.float32)
    p = orc.init_deltanet_params(seed + 1, C, H, W, kernel_size=ks, gate_type=gate_type,
                                 bias_scale=0.1)
    p["output_proj"]["bias"][:] = 0
    ref = orc.deltanet_forward(p, x, kernel_size=ks, gate_type=gate_type, rope_mode=rope,
                               scan_mode=scan_mode)
    mod = DeltaNetCSSM(channels=C, kernel_size=ks, gate_type=gate_type, rope_mode=rope,
                       scan_mode=scan_mode)
    y = mod.apply({"params": p}, torch.from_numpy(x).cuda()).cpu().numpy()
    assert np.isfinite(y).all()
    assert np.abs(ref).max() > 1e-5
    return orc.rel_l2(y, ref)


@pytest.mark.parametrize("case,gate_type,rope", [
    ((2, 4, 64, 64, 64, 11), "factored", "spatiotemporal"),   # 64x64 radix kernel, tensor-core GEMMs
    ((1, 3, 64, 64, 8, 11), "dense", "none"),                 # 64x64 radix kernel, dense gates
    ((3, 9, 64, 64, 4, 5), "factored", "mrope"),              # 64x64, nine steps of state
    ((3, 6, 32, 32, 8, 11), "dense", "mrope"),
    ((2, 3, 14, 10, 12, 3), "factored", "spatial_only"),      # ragged plane
    ((2, 5, 16, 16, 8, 7), "dense", "temporal"),
    ((1, 1, 7, 7, 4, 11), "factored", "none"),                # T = 1, kernel larger than the plane
    ((2, 4, 64, 64, 64, 11), "channel", "spatiotemporal"),    # the reference's default gate type
    ((2, 5, 64, 64, 8, 5), "channel", "none"),
    ((2, 6, 32, 32, 8, 11), "channel", "mrope"),
    ((2, 3, 14, 10, 12, 3), "channel", "spatial_only"),
    ((1, 1, 6, 6, 4, 3), "channel", "temporal"),
    ((2, 3, 7, 7, 4, 3), "channel", "spatiotemporal"),          # H*W not a multiple of 4
    ((2, 2, 7, 5, 12, 3), "channel", "none"),
], ids=lambda c: "x".join(map(str, c)) if isinstance(c, tuple) else str(c))
def test_block_parity(case, gate_type, rope):
    assert _run(case, gate_type, rope) <= TOL


@pytest.mark.parametrize("H,W,C", [(1, 1, 4), (2, 3, 4), (5, 8, 20), (26, 48, 8), (27, 48, 8), (51, 100, 4), (52, 100, 4)])
def test_factored_gate_vectors(H, W, C):
    """5 (H + W/2 + 1) vector entries around 256 and 512 (slices of the channels, fewer channels than slices, one
    round of a CTA's threads, two).  float32 through two projections, transforms and two steps: 1e-5."""
    assert _run((2, 2, H, W, C, 1), "factored", "none") <= 1e-5


@pytest.mark.parametrize("scan_mode", ["ssd", "quadratic", "pallas"])
def test_linear_scan_modes(scan_mode):
    assert _run((2, 6, 32, 32, 8, 5), "factored", "spatiotemporal", scan_mode=scan_mode) <= TOL
    assert _run((1, 4, 64, 64, 8, 5), "dense", "none", scan_mode=scan_mode, seed=2) <= TOL


def test_long_sequence_state():
    """T = 20: the state is carried through twenty updates of the delta rule."""
    assert _run((1, 20, 16, 16, 8, 5), "dense", "spatiotemporal", seed=4) <= TOL


def test_golden_fixture_on_gpu():
    """The committed fixture (tests/golden/deltanet_small.npz, written by make_golden.py)."""
    from tests.golden import make_golden as mg
    g = np.load(os.path.join(os.path.dirname(mg.__file__), "deltanet_small.npz"))
    _, p, kw = mg.deltanet_case()
    mod = DeltaNetCSSM(channels=g["x"].shape[-1], kernel_size=kw["kernel_size"],
                       gate_type=kw["gate_type"], rope_mode=kw["rope_mode"])
    y = mod.apply({"params": p}, torch.from_numpy(g["x"]).cuda()).cpu().numpy()
    assert orc.rel_l2(y, g["y"]) <= TOL
