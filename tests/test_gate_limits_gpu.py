"""Gate maps of wide blocks and of long planes, whose contexts and vectors take more than the 48 KB of shared
memory that a launch has by default: dense gates of 1536 and 3072 channels with enough frames for eight and
four frames a CTA, factored gates of planes of thousands of pixels a row, against the oracle."""
import numpy as np
import pytest
import torch

from oracle import cssm_oracle as orc
from cssm_b200 import AdditiveCSSM, DeltaNetCSSM, GatedCSSM, GatedDeltaNetCSSM

pytestmark = pytest.mark.gpu
# float32 sums of up to 3072 terms with random signs behind norms and transforms of up to 8000 pixels:
# sqrt(3072) * 2^-24 = 3e-6 of the 2-norm for each of the two projections in a row
TOL = 1e-5


def _block(kind, C, gate):
    kw = dict(kernel_size=1, rope_mode="none", gate_type=gate)
    if kind == "gated":
        return GatedCSSM(channels=C, **kw), orc.init_gated_params, orc.gated_forward, kw, ("kernel_size", "gate_type")
    if kind == "gdn":
        kw["delta_key_dim"] = 2
        return GatedDeltaNetCSSM(channels=C, **kw), orc.init_gdn_params, orc.gdn_forward, kw, ("kernel_size", "gate_type", "delta_key_dim")
    if kind == "deltanet":
        return DeltaNetCSSM(channels=C, **kw), orc.init_deltanet_params, orc.deltanet_forward, kw, ("kernel_size", "gate_type")
    return AdditiveCSSM(channels=C, single_state=True, **kw), orc.init_additive1_params, orc.additive1_forward, kw, ("kernel_size", "gate_type")


@pytest.mark.parametrize("kind,C,B", [("gated", 1536, 592), ("gated", 3072, 296), ("gdn", 1536, 296), ("gdn", 3072, 148),
                                      ("deltanet", 1536, 592), ("additive", 1536, 592)])
def test_dense_gates_of_wide_blocks(kind, C, B):
    H = W = 16
    m, init, fwd, kw, names = _block(kind, C, "dense")
    p = init(1, C, H, W, bias_scale=0.1, **{k: kw[k] for k in names})
    x = torch.randn((B, 1, H, W, C), device="cuda", generator=torch.Generator(device="cuda").manual_seed(C))
    y = m.apply({"params": p}, x)
    for i in (0, B - 1):
        ref = fwd(p, x[i:i + 1].cpu().numpy(), **kw)
        assert orc.rel_l2(y[i:i + 1].cpu().numpy(), ref) <= TOL
    del x, y
    torch.cuda.empty_cache()


@pytest.mark.parametrize("kind,W", [("gated", 8000), ("additive", 8000), ("deltanet", 4880), ("gdn", 4000)])
def test_factored_gates_of_long_planes(kind, W):
    C = 4
    m, init, fwd, kw, names = _block(kind, C, "factored")
    p = init(1, C, 1, W, bias_scale=0.1, **{k: kw[k] for k in names})
    x = np.random.default_rng(W).standard_normal((2, 2, 1, W, C)).astype(np.float32)
    y = m.apply({"params": p}, torch.from_numpy(x).cuda()).cpu().numpy()
    assert orc.rel_l2(y, fwd(p, x, **kw)) <= TOL
