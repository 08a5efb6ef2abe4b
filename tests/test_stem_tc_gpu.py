"""GPU parity of the stem kernels (first layers of one or three input channels, four pixels a quad of lanes; later layers of
32 and 64 channels on the tensor cores) against the oracle."""
import numpy as np
import pytest
import torch

from cssm_b200 import SimpleCSSM
from oracle import cssm_oracle as orc
from oracle import simple_oracle as so

pytestmark = pytest.mark.gpu


def _stem(E, layers, x, stem_mode="default", edit=None):
    clip = stem_mode == "pathtracker"
    m = SimpleCSSM(cssm_type="gated", embed_dim=E, kernel_size=1, pos_embed="none", seq_len=x.shape[1] if clip else 1,
                   stem_mode=stem_mode, stem_layers=layers, gate_type="factored", pool_type="max")
    H, W = m.feature_hw(*x.shape[-3:-1])
    bkw = dict(kernel_size=1, rope_mode="none", gate_type="factored", short_conv_size=4, short_conv_spatial_size=3)
    p = so.init_simple_params(7, cin=x.shape[-1], embed_dim=E, H=H, W=W, num_classes=2, cssm_type="gated", stem_mode=stem_mode,
                              stem_layers=layers, bias_scale=0.1, block_kwargs=bkw)
    if edit is not None:
        edit(p)
    ref = so.stem_forward(p, x.reshape(-1, *x.shape[-3:]).astype(np.float64), stem_mode=stem_mode, stem_layers=layers)
    got = m.bind({"params": p}).stem(torch.from_numpy(x).cuda()).cpu().numpy()
    return got, np.asarray(ref).reshape(got.shape)


# sides: one window, tiles of 16 x 8 cut on either side, odd (padded pool windows), whole tiles; three layers
@pytest.mark.parametrize("E", [32, 64])
@pytest.mark.parametrize("layers,shape", [(2, (1, 2, 2, 1)), (2, (2, 30, 18, 1)), (2, (1, 34, 66, 3)), (2, (3, 64, 32, 1)), (3, (2, 37, 75, 1)),
                                          (4, (1, 96, 160, 3))])
def test_later_layers(E, layers, shape):
    """float32 sums of 9 E terms behind LayerNorms, a few layers deep: sqrt(576) * 2^-24 = 1.5e-6 of the 2-norm a layer."""
    got, ref = _stem(E, layers, np.random.default_rng(shape[1]).random(shape).astype(np.float32))
    assert orc.rel_l2(got, ref) <= 5e-6


@pytest.mark.parametrize("E", [16, 32, 48, 64])
@pytest.mark.parametrize("shape", [(1, 1, 1, 1), (1, 7, 9, 1), (2, 15, 16, 3), (5, 33, 20, 1)])
def test_first_layer(E, shape):
    got, ref = _stem(E, 1, np.random.default_rng(shape[2]).random(shape).astype(np.float32))
    assert orc.rel_l2(got, ref) <= 5e-6


@pytest.mark.parametrize("E", [32, 64])
@pytest.mark.parametrize("shape", [(1, 1, 1, 1, 3), (1, 3, 5, 7, 3), (2, 4, 9, 11, 1), (2, 3, 32, 32, 3)])
def test_pointwise_layer(E, shape):
    got, ref = _stem(E, 1, np.random.default_rng(shape[2]).random(shape).astype(np.float32), stem_mode="pathtracker")
    assert orc.rel_l2(got, ref) <= 5e-6


def test_weight_beyond_bfloat16():
    """A weight above the largest bfloat16 (3.39e38) has no finite parts; times inputs of 1e-37 the sums are ordinary numbers."""
    def edit(p):
        w = np.asarray(p["conv2"]["kernel"]).copy()
        w[1, 1, 3, 5] = 3.4e38
        p["conv2"]["kernel"] = w
        n = p["norm1"]
        n["scale"] = np.full_like(np.asarray(n["scale"]), 0.0)
        n["bias"] = np.full_like(np.asarray(n["bias"]), 1e-37)
    got, ref = _stem(64, 2, np.random.default_rng(1).random((1, 24, 24, 1)).astype(np.float32), edit=edit)
    assert np.isfinite(got).all()
    assert orc.rel_l2(got, ref) <= 5e-6
