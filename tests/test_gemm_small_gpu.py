"""The few-row bf16 GEMM (csrc/gemm_small.cu) through the C entry points: one row, ragged row tiles, two, four and eight warps a tile,
step counts that leave warps without work, long K loops, and the classifier block whose fc1 takes its LayerNorm on the way."""
import numpy as np
import pytest
import torch
import torch.nn.functional as F

from cssm_b200._lib import check, lib

pytestmark = pytest.mark.gpu


def _st():
    return torch.cuda.current_stream().cuda_stream


# 2-norm of the difference: one bf16 rounding of the output, 2^-9 at most, 0.29 of that in the mean
@pytest.mark.parametrize("M,K,N,act,res", [(1, 64, 64, 0, False), (31, 32, 32, 1, True), (33, 96, 96, 2, True), (49, 128, 160, 0, True),
                                           (65, 160, 64, 1, False), (7, 224, 32, 0, False), (100, 256, 96, 2, True), (49, 288, 64, 0, True),
                                           (196, 1024, 256, 0, True), (49, 1536, 384, 1, True), (20, 2080, 64, 0, False)])
def test_small_gemm(M, K, N, act, res):
    L = lib()
    g = torch.Generator(device="cuda").manual_seed(M + K + N)
    A = torch.randn((M, K), device="cuda", generator=g).to(torch.bfloat16)
    W = torch.randn((K, N), device="cuda", generator=g) / K ** 0.5
    b = torch.randn((N + 1,), device="cuda", generator=g)[1:]            # 4-byte aligned only
    R = torch.randn((M, N), device="cuda", generator=g).to(torch.bfloat16) if res else None
    wt = torch.empty((N, L.cssm_bf16_packed_ld(K)), dtype=torch.bfloat16, device="cuda")
    check(L.cssm_bf16_pack_weight(W.data_ptr(), K, N, None, wt.data_ptr(), _st()), "pack")
    out = torch.full((M + 1, N), 7.0, dtype=torch.bfloat16, device="cuda")
    check(L.cssm_bf16_gemm(A.data_ptr(), M, K, wt.data_ptr(), N, b.data_ptr(), act, R.data_ptr() if res else None,
                           out.data_ptr(), _st()), "gemm")
    ref = A.double() @ W.to(torch.bfloat16).double() + b.double()
    ref = F.gelu(ref, approximate="tanh") if act == 1 else F.silu(ref) if act == 2 else ref
    if res:
        ref = ref + R.double()
    assert float((out[:M].double() - ref).norm() / ref.norm()) <= 3e-3
    assert bool((out[M] == 7.0).all())                                    # no store past the last row


@pytest.mark.parametrize("B,Hi,Wi,Cin,Cout", [(1, 3, 3, 32, 64), (1, 8, 8, 32, 64), (1, 7, 5, 64, 64), (2, 13, 10, 96, 96), (1, 14, 14, 256, 384)])
def test_small_conv(B, Hi, Wi, Cin, Cout):
    L = lib()
    g = torch.Generator(device="cuda").manual_seed(Hi * Cin)
    x = torch.randn((B, Hi, Wi, Cin), device="cuda", generator=g).to(torch.bfloat16)
    W = torch.randn((3, 3, Cin, Cout), device="cuda", generator=g) / (9 * Cin) ** 0.5
    b = torch.randn((Cout,), device="cuda", generator=g)
    wt = torch.empty((Cout, L.cssm_bf16_conv3x3s2_packed_ld(Cin, Wi, Cout)), dtype=torch.bfloat16, device="cuda")
    check(L.cssm_bf16_pack_conv3x3s2_weight(W.data_ptr(), Cin, Cout, Wi, None, wt.data_ptr(), _st()), "pack")
    Ho, Wo = (Hi + 1) // 2, (Wi + 1) // 2
    out = torch.empty((B, Ho, Wo, Cout), dtype=torch.bfloat16, device="cuda")
    check(L.cssm_bf16_conv3x3s2(x.data_ptr(), B, Hi, Wi, Cin, wt.data_ptr(), Cout, b.data_ptr(), 0, out.data_ptr(), _st()), "conv")
    th, tw = max((Ho - 1) * 2 + 3 - Hi, 0), max((Wo - 1) * 2 + 3 - Wi, 0)
    xp = F.pad(x.double().permute(0, 3, 1, 2), (tw // 2, tw - tw // 2, th // 2, th - th // 2))
    ref = F.conv2d(xp, W.to(torch.bfloat16).double().permute(3, 2, 0, 1), b.double(), stride=2).permute(0, 2, 3, 1)
    assert float((out.double() - ref).norm() / ref.norm()) <= 3e-3


@pytest.mark.parametrize("C,side", [(64, 9), (96, 5), (128, 28), (256, 6), (384, 7), (512, 3)])
def test_fc1_with_its_layernorm(C, side):
    """A ConvBlock of one image against the oracle: LayerNorm inside the GEMM (128 and 256 channels: one step of K for each of four and
    eight warps), in a launch of its own (96, 384 and 512), and the fused Mlp (64)."""
    from cssm_b200.shvit import CSSMSHViT
    from oracle import shvit_oracle as sv
    rng = np.random.default_rng(C)
    dims = (C,) * 4
    kw = dict(embed_dims=dims, depths=(1, 1, 1, 1), kernel_sizes=(1, 1, 1, 1), use_cssm_stages=(False,) * 4)
    hw = (4 * side, 4 * side)
    p, s = sv.init_shvit_params(3, hw, num_classes=10, **kw)
    x = torch.from_numpy(rng.standard_normal((1, *hw, 3)).astype(np.float32)).to(torch.bfloat16)
    net = CSSMSHViT(num_classes=10, num_timesteps=1, short_conv_spatial_size=0, **kw)
    got = net.apply({"params": p, "batch_stats": s}, x.cuda()).float().cpu().numpy()
    want = sv.shvit_forward(p, s, x.float().numpy().astype(np.float64), num_timesteps=1, **kw)
    assert float(np.abs(got - want).max() / max(np.abs(want - want.mean()).max(), 1e-30)) <= 2e-2


@pytest.mark.parametrize("side", [3, 9])
def test_fc1_with_its_layernorm_two_warps_a_tile(side):
    """64 channels in a mixer block, whose Mlp has a depthwise conv in it and so does not run in the fused kernel."""
    from cssm_b200.shvit import CSSMSHViT
    from oracle import shvit_oracle as sv
    kw = dict(embed_dims=(64,) * 4, depths=(1, 1, 1, 1), kernel_sizes=(1, 1, 1, 1), use_cssm_stages=(True,) * 4)
    hw = (4 * side, 4 * side)
    p, s = sv.init_shvit_params(5, hw, num_classes=10, short_conv_spatial_size=0, **kw)
    x = torch.from_numpy(np.random.default_rng(side).standard_normal((1, *hw, 3)).astype(np.float32)).to(torch.bfloat16)
    net = CSSMSHViT(num_classes=10, num_timesteps=1, short_conv_spatial_size=0, **kw)
    got = net.apply({"params": p, "batch_stats": s}, x.cuda()).float().cpu().numpy()
    want = sv.shvit_forward(p, s, x.float().numpy().astype(np.float64), num_timesteps=1, short_conv_spatial_size=0, **kw)
    assert float(np.abs(got - want).max() / max(np.abs(want - want.mean()).max(), 1e-30)) <= 2e-2
