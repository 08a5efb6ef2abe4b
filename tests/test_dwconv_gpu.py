"""The depthwise convs of the classifier's blocks (csrc/shvit_kernels.cu, dwconv_tiled_kernel) with tiles enough for every SM, where
the large tiles run: 7 x 7 on planes of whole and of ragged tiles and blocks, 3 x 3 with float32 outputs on 14 x 14 planes."""
import numpy as np
import pytest
import torch
import torch.nn.functional as F

from cssm_b200 import CSSMSHViTBlock, ConvBlock, device_error
from oracle import shvit_oracle as sv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,W", [(11, 56, 56), (38, 28, 28), (7, 72, 72), (16, 36, 36), (15, 40, 40), (40, 14, 14), (150, 7, 7), (20, 29, 28),
                                   (18, 35, 56), (16, 33, 31), (12, 41, 27), (9, 57, 56)])
@pytest.mark.parametrize("C", [64, 128])
def test_conv7(B, H, W, C):
    """A ConvBlock whose pointwise conv is the identity and whose Mlp is zero is x + gelu(conv(norm(x))); x is small beside it.  Two bf16 roundings
    (the staged norm's, shared with the reference up to ties, and the output's): 2^-9 each at most."""
    g = torch.Generator(device="cuda").manual_seed(H * W)
    n = lambda *s: torch.randn(s, device="cuda", generator=g)
    x = (n(B, H, W, C) * 2.0 ** -6).bfloat16()
    k, kb, ns, nb = n(7, 7, 1, C) / 7, 0.3 * n(C), 1 + 0.2 * n(C), 0.2 * n(C)
    zero = lambda *s: torch.zeros(s, device="cuda")
    p = {"norm1": {"scale": ns, "bias": nb}, "dwconv": {"dwconv": {"kernel": k, "bias": kb}},
         "pwconv": {"kernel": torch.eye(C, device="cuda"), "bias": zero(C)}, "norm2": {"scale": ns, "bias": nb},
         "mlp": {"fc1": {"kernel": zero(C, 4 * C), "bias": zero(4 * C)}, "fc2": {"kernel": zero(4 * C, C), "bias": zero(C)}}}
    y = ConvBlock(dim=C).bind({"params": p})(x)
    h = F.layer_norm(x.double(), (C,), ns.double(), nb.double(), 1e-6).bfloat16().double()
    conv = F.conv2d(h.permute(0, 3, 1, 2), k.double().permute(3, 2, 0, 1), kb.double(), padding=3, groups=C).permute(0, 2, 3, 1)
    want = F.gelu(conv, approximate="tanh")
    d = y.double() - x.double() - want
    assert device_error() == 0
    assert float(d.norm() / want.norm()) < 4e-3
    # no pixel of its own: the largest outputs are some ten times the root mean square, a rounding 2^-8 of that
    assert float(d.abs().max() / want.pow(2).mean().sqrt()) < 0.1


@pytest.mark.parametrize("B,H,C", [(48, 14, 256), (40, 14, 128), (20, 16, 256), (170, 7, 64)])
def test_position_conv_of_float32_mixers(B, H, C):
    """Against the oracle on the first and the last image; without a position conv's tap the block is off by more than 0.05."""
    kw = dict(num_timesteps=2, kernel_size=3)
    p, _ = sv.init_shvit_params(H + C, (H * 4, H * 4), embed_dims=(C, C, C, C), depths=(1, 1, 1, 1), use_cssm_stages=(True,) * 4,
                                kernel_sizes=(3, 3, 3, 3))
    p = p["stage0_block0"]
    x = torch.randn((B, H, H, C), generator=torch.Generator().manual_seed(B)).to(torch.bfloat16)
    y = CSSMSHViTBlock(dim=C, **kw).bind({"params": p})(x.cuda())[[0, B - 1]].double().cpu().numpy()
    want = sv.cssm_block(x[[0, B - 1]].double().numpy(), p, **kw)
    assert device_error() == 0
    assert np.linalg.norm(y - want) / np.linalg.norm(want) < 6e-3
