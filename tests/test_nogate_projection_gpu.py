"""Output projection of the ungated block at 64 channels (y - x stored by the kernel itself, csrc/gemm_tc.cu): one tile, fewer tiles
than SMs, and several rounds with an uneven last one, against the oracle."""
import numpy as np
import pytest
import torch

from cssm_b200 import NoGateCSSM
from oracle import cssm_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,T,H,W", [(1, 1, 8, 16), (1, 3, 16, 16), (3, 1, 32, 32), (1, 2, 64, 64), (101, 3, 16, 8), (37, 2, 32, 32)])
def test_projection_of_the_ungated_block(B, T, H, W):
    """3 x TF32 products and float32 transforms: below 1e-6 of the 2-norm, held to 5e-6."""
    x = np.random.default_rng(B).standard_normal((B, T, H, W, 64)).astype(np.float32)
    mod = NoGateCSSM(channels=64, kernel_size=5)
    p = mod.init(1, x.shape, bias_scale=0.1)["params"]
    y = mod.apply({"params": p}, torch.from_numpy(x).cuda()).cpu().numpy()
    pick = sorted({0, B // 2, B - 1})
    assert np.isfinite(y).all()
    assert orc.rel_l2(y[pick], orc.nogate_forward(p, x[pick], kernel_size=5)) <= 5e-6
