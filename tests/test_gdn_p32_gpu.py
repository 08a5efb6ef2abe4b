"""The 32x32 recurrence kernel (csrc/gdn_spectral_p32.cu) against the oracle: one head to more than two a CTA, one step to several (the
first and last phases of its barriers, the tail of its task list), all frames and the last one alone, planes that only the real
columns of the spectrum see."""
import numpy as np
import pytest
import torch

from cssm_b200 import DeltaNetCSSM, GatedDeltaNetCSSM, device_error
from oracle import cssm_oracle as orc

pytestmark = pytest.mark.gpu


def _case(B, T, C, seed, edit=None, l2=True):
    kw = dict(delta_key_dim=4, kernel_size=3, gate_type="factored", qkv_conv_size=1, use_input_gates=True)
    x = np.random.default_rng(seed).standard_normal((B, T, 32, 32, C)).astype(np.float32)
    if edit is not None:
        edit(x)
    p = orc.init_gdn_params(seed, C, 32, 32, bias_scale=0.1, **kw)
    ref = orc.gdn_forward(p, x, rope_mode="none", use_spectral_l2_norm=l2, **kw)
    m = GatedDeltaNetCSSM(channels=C, rope_mode="none", use_spectral_l2_norm=l2, **kw).bind({"params": p})
    xd = torch.from_numpy(x).cuda()
    return m(xd).cpu().numpy(), m(xd, last_frame_only=True).cpu().numpy(), ref


@pytest.mark.parametrize("B,C", [(1, 4), (1, 12), (148, 4), (149, 4), (299, 4), (20, 64)])
@pytest.mark.parametrize("T", [1, 2, 3, 5])
def test_heads_and_steps(B, C, T):
    """float32 transforms, projections and T steps: below 5e-6 of the 2-norm (csrc/gdn_spectral_dft.cu's sizes are the same)."""
    y, last, ref = _case(B, T, C, 100 * T + C)
    assert orc.rel_l2(y, ref) <= 1e-5
    assert orc.rel_l2(last, ref[:, -1]) <= 1e-5
    assert device_error() == 0


@pytest.mark.parametrize("l2", [False, True])
@pytest.mark.parametrize("kind", ["constant rows", "alternating columns", "constant"])
def test_real_columns_alone(kind, l2):
    """Energy in columns 0 and 16 of the spectrum alone: those share one FFT, and their bins' lanes separate them."""
    def edit(x):
        if kind == "constant rows":
            x[...] = x[:, :, :, :1]
        elif kind == "alternating columns":
            x[...] = x[:, :, :, :1] * np.where(np.arange(32) % 2, -1.0, 1.0)[:, None].astype(np.float32)
        else:
            x[...] = x[:, :, :1, :1]
    y, last, ref = _case(2, 3, 16, 3, edit, l2)
    assert orc.rel_l2(y, ref) <= 2e-5
    assert orc.rel_l2(last, ref[:, -1]) <= 2e-5


@pytest.mark.parametrize("B,C", [(1, 4), (2, 12), (149, 4), (20, 64)])
@pytest.mark.parametrize("T", [1, 2, 5])
def test_deltanet_channel_gates(B, C, T):
    kw = dict(kernel_size=3, rope_mode="none", gate_type="channel")
    x = np.random.default_rng(T).standard_normal((B, T, 32, 32, C)).astype(np.float32)
    m = DeltaNetCSSM(channels=C, **kw)
    p = orc.init_deltanet_params(5, C, 32, 32, kernel_size=3, gate_type="channel", bias_scale=0.1)
    p["output_proj"]["bias"][:] = 0                      # the block's signal is two orders below a 0.1-scale bias
    ref = orc.deltanet_forward(p, x, **kw)
    got = m.apply({"params": p}, torch.from_numpy(x).cuda()).cpu().numpy()
    assert orc.rel_l2(got, ref) <= 1e-4
    assert device_error() == 0
