"""The 64x64 recurrence kernel (csrc/gdn_spectral_p64.cu) against the oracle: one head to more than one a CTA, one step to several (the
first and last phases of its barriers, the inverse after the last step), gates of a frame and of a head, all frames and the last one alone,
planes that only the real columns of the spectrum see."""
import numpy as np
import pytest
import torch

from cssm_b200 import GatedDeltaNetCSSM, device_error
from oracle import cssm_oracle as orc

pytestmark = pytest.mark.gpu


def _case(B, T, C, seed, edit=None, l2=True, gates="factored"):
    kw = dict(delta_key_dim=4, kernel_size=3, gate_type=gates, qkv_conv_size=1, use_input_gates=True)
    x = np.random.default_rng(seed).standard_normal((min(B, 2), T, 64, 64, C)).astype(np.float32)
    if edit is not None:
        edit(x)
    p = orc.init_gdn_params(seed, C, 64, 64, bias_scale=0.1, **kw)
    idx = np.arange(B) % len(x)                                  # the oracle has two clips to do, the kernel all of them
    ref = orc.gdn_forward(p, x, rope_mode="none", use_spectral_l2_norm=l2, **kw)[idx]
    m = GatedDeltaNetCSSM(channels=C, rope_mode="none", use_spectral_l2_norm=l2, **kw).bind({"params": p})
    xd = torch.from_numpy(x[idx]).cuda()
    return m(xd).cpu().numpy(), m(xd, last_frame_only=True).cpu().numpy(), ref


@pytest.mark.parametrize("B,C,T", [(1, 4, 1), (1, 12, 2), (2, 4, 5), (148, 4, 1), (149, 4, 2), (40, 16, 3), (10, 64, 2)])
@pytest.mark.parametrize("gates", ["factored", "channel"])
def test_heads_and_steps(B, C, T, gates):
    """float32 transforms, projections and T steps: below 5e-6 of the 2-norm, as at 32x32."""
    y, last, ref = _case(B, T, C, 100 * T + C, gates=gates)
    assert orc.rel_l2(y, ref) <= 5e-6
    assert orc.rel_l2(last, ref[:, -1]) <= 5e-6
    assert device_error() == 0


@pytest.mark.parametrize("l2", [False, True])
@pytest.mark.parametrize("kind", ["constant rows", "alternating columns", "constant"])
def test_real_columns_alone(kind, l2):
    """Energy in columns 0 and 32 of the spectrum alone: those share one FFT, and the warp separates them."""
    def edit(x):
        if kind == "constant rows":
            x[...] = x[:, :, :, :1]
        elif kind == "alternating columns":
            x[...] = x[:, :, :, :1] * np.where(np.arange(64) % 2, -1.0, 1.0)[:, None].astype(np.float32)
        else:
            x[...] = x[:, :, :1, :1]
    y, last, ref = _case(2, 3, 16, 3, edit, l2)
    assert orc.rel_l2(y, ref) <= 2e-5
    assert orc.rel_l2(last, ref[:, -1]) <= 2e-5
