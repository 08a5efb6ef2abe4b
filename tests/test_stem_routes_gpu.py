"""Stem layers that the tensor-core kernel does not take, against the oracle: later layers of a caller whose workspace holds the two
layer buffers and no more (csrc/simple_model.cu: stem_layer_pair at 64 channels, the window kernel and, below a wave of
windows, the quad kernel at 32), and first layers of many input channels."""
import ctypes as C

import numpy as np
import pytest
import torch

from cssm_b200 import SimpleCSSM
from cssm_b200._lib import check
from oracle import cssm_oracle as orc
from oracle import simple_oracle as so

pytestmark = pytest.mark.gpu


def _model(E, layers, shape, seed=7):
    m = SimpleCSSM(cssm_type="gated", embed_dim=E, kernel_size=1, pos_embed="none", seq_len=1, stem_layers=layers, gate_type="factored",
                   pool_type="max")
    H, W = m.feature_hw(*shape[1:3])
    bkw = dict(kernel_size=1, rope_mode="none", gate_type="factored", short_conv_size=4, short_conv_spatial_size=3)
    p = so.init_simple_params(seed, cin=shape[-1], embed_dim=E, H=H, W=W, num_classes=2, cssm_type="gated", stem_mode="default",
                              stem_layers=layers, bias_scale=0.1, block_kwargs=bkw)
    return m.bind({"params": p}), p, (shape[0], H, W, E)


# float32 sums of up to 9 * 64 terms behind LayerNorms: sqrt(576) * 2^-24 = 1.5e-6 of the 2-norm a layer
@pytest.mark.parametrize("E", [32, 64])
@pytest.mark.parametrize("layers,shape", [(2, (1, 3, 5, 1)), (2, (2, 30, 18, 3)), (2, (1, 128, 128, 1)), (2, (5, 256, 250, 1)), (3, (2, 37, 75, 1))])
def test_two_buffers_are_enough(E, layers, shape):
    b, p, out = _model(E, layers, shape)
    x = np.random.default_rng(shape[1]).random(shape).astype(np.float32)
    xd = torch.from_numpy(x).cuda()
    half = (shape[0] * ((shape[1] + 1) // 2) * ((shape[2] + 1) // 2) * E * 4 + 255) // 256 * 256
    ws = torch.full((2 * half + 256,), 0xFF, dtype=torch.uint8, device="cuda")
    feat = torch.full(out, float("nan"), device="cuda")
    d = b.desc(tuple(shape))
    check(b.L.cssm_simple_stem(C.byref(d), C.byref(b.w), xd.data_ptr(), feat.data_ptr(), ws.data_ptr(), 2 * half,
                               torch.cuda.current_stream().cuda_stream), "stem")
    ref = np.asarray(so.stem_forward(p, x.astype(np.float64), stem_mode="default", stem_layers=layers))
    assert orc.rel_l2(feat.cpu().numpy(), ref) <= 5e-6
    assert bool((ws[2 * half:] == 0xFF).all())


@pytest.mark.parametrize("E", [32, 64])
@pytest.mark.parametrize("shape", [(1, 1, 1, 32), (1, 5, 3, 36), (2, 17, 24, 48), (3, 33, 31, 64), (1, 9, 10, 96), (2, 40, 44, 16)])
def test_first_layer_of_many_channels(E, shape):
    b, p, _ = _model(E, 1, shape)
    x = np.random.default_rng(shape[3]).standard_normal(shape).astype(np.float32)
    ref = np.asarray(so.stem_forward(p, x.astype(np.float64), stem_mode="default", stem_layers=1))
    assert orc.rel_l2(b.stem(torch.from_numpy(x).cuda()).cpu().numpy().reshape(ref.shape), ref) <= 5e-6


# three quarters of 148 SMs with a CTA of 256 pixels: 111 CTAs (the first of each pair has 108)
@pytest.mark.parametrize("stem,shape", [("default", (3, 96, 96, 1)), ("default", (3, 96, 98, 1)), ("default", (3, 96, 98, 3)), ("default", (1, 9, 7, 3)),
                                        ("pathtracker", (1, 27, 32, 32, 3)), ("pathtracker", (1, 28, 32, 32, 3)), ("pathtracker", (2, 1, 5, 3, 1))])
def test_first_layer_of_few_and_many_pixels(stem, shape):
    clip = stem == "pathtracker"
    m = SimpleCSSM(cssm_type="gated", embed_dim=64, kernel_size=1, pos_embed="none", seq_len=shape[1] if clip else 1, stem_mode=stem,
                   stem_layers=1, gate_type="factored", pool_type="max")
    H, W = m.feature_hw(*shape[-3:-1])
    bkw = dict(kernel_size=1, rope_mode="none", gate_type="factored", short_conv_size=4, short_conv_spatial_size=3)
    p = so.init_simple_params(3, cin=shape[-1], embed_dim=64, H=H, W=W, num_classes=2, cssm_type="gated", stem_mode=stem, stem_layers=1,
                              bias_scale=0.1, block_kwargs=bkw)
    x = np.random.default_rng(shape[-2]).random(shape).astype(np.float32)
    got = m.bind({"params": p}).stem(torch.from_numpy(x).cuda()).cpu().numpy()
    ref = np.asarray(so.stem_forward(p, x.reshape(-1, *shape[-3:]).astype(np.float64), stem_mode=stem, stem_layers=1)).reshape(got.shape)
    assert orc.rel_l2(got, ref) <= 5e-6


# a window's largest value is at the smallest normalised one where a channel's scale is negative, and its bias where it is zero
@pytest.mark.parametrize("E", [32, 64])
@pytest.mark.parametrize("shape", [(2, 17, 24, 1), (1, 16, 15, 3), (4, 96, 98, 1)])
def test_scales_of_any_sign(E, shape):
    _, p, _ = _model(E, 1, shape)
    rng = np.random.default_rng(shape[1])
    p["norm1"]["scale"] = (rng.standard_normal(E) * (np.arange(E) % 7 != 3)).astype(np.float32)
    b = SimpleCSSM(cssm_type="gated", embed_dim=E, kernel_size=1, pos_embed="none", seq_len=1, stem_layers=1, gate_type="factored",
                   pool_type="max").bind({"params": p})
    x = rng.standard_normal(shape).astype(np.float32)
    ref = np.asarray(so.stem_forward(p, x.astype(np.float64), stem_mode="default", stem_layers=1))
    assert orc.rel_l2(b.stem(torch.from_numpy(x).cuda()).cpu().numpy().reshape(ref.shape), ref) <= 5e-6
