"""Column tiles of the planar three-way split GEMM above 256 channels (csrc/gemm_split.cu): row counts at which tiles of 96 and of 128
columns are chosen, one and several rounds, N a multiple of neither, through the ungated block against the oracle."""
import numpy as np
import pytest
import torch

from cssm_b200 import NoGateCSSM
from oracle import cssm_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,C", [(2, 384), (25, 384), (71, 384), (153, 384), (25, 320), (71, 416), (107, 448), (30, 512), (71, 512), (25, 260)])
def test_column_tiles(B, C):
    """Six products of three bfloat16 parts (2^-24 a product, sums of C terms) and float32 transforms: held to 5e-6 of the 2-norm."""
    x = np.random.default_rng(B).standard_normal((B, 1, 14, 14, C)).astype(np.float32)
    mod = NoGateCSSM(channels=C, kernel_size=3)
    p = mod.init(1, x.shape, bias_scale=0.1)["params"]
    y = mod.apply({"params": p}, torch.from_numpy(x).cuda()).cpu().numpy()
    assert np.isfinite(y).all()
    pick = sorted({0, B // 2, B - 1})
    ref = orc.nogate_forward(p, x[pick], kernel_size=3)
    assert orc.rel_l2(y[pick] + x[pick], ref + x[pick]) <= 5e-6        # the projection itself: the block subtracts its input
