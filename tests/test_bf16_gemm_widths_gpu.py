"""The bf16 GEMM (csrc/gemm_bf16.cu) at widths where a bias, a residual by TMA and the staging slots compete for shared memory, and a
whole classifier of such widths."""
import numpy as np
import pytest
import torch
import torch.nn.functional as F

from cssm_b200 import CSSMSHViT, CssmError, device_error, lib
from cssm_b200._lib import check
from oracle import cssm_oracle as orc
from oracle import shvit_oracle as sv

pytestmark = pytest.mark.gpu


def _gemm(M, K, N, act, res, bias_offset=0, bias=True):
    L = lib()
    st = torch.cuda.current_stream().cuda_stream
    g = torch.Generator(device="cuda").manual_seed(M + K + N)
    A = torch.randn((M, K), device="cuda", generator=g).to(torch.bfloat16)
    W = torch.randn((K, N), device="cuda", generator=g) / K ** 0.5
    b = torch.randn((N + bias_offset,), device="cuda", generator=g)[bias_offset:]
    R = torch.randn((M, N), device="cuda", generator=g).to(torch.bfloat16) if res else None
    wt = torch.empty((N, L.cssm_bf16_packed_ld(K)), dtype=torch.bfloat16, device="cuda")
    check(L.cssm_bf16_pack_weight(W.data_ptr(), K, N, None, wt.data_ptr(), st), "pack")
    out = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device="cuda")
    check(L.cssm_bf16_gemm(A.data_ptr(), M, K, wt.data_ptr(), N, b.data_ptr() if bias else None, act,
                           R.data_ptr() if res else None, out.data_ptr(), st), "gemm")
    torch.cuda.synchronize()
    assert device_error() == 0
    tf32 = torch.backends.cuda.matmul.allow_tf32
    torch.backends.cuda.matmul.allow_tf32 = False
    worst = 0.0
    for r in range(0, M, 20000):
        ref = A[r:r + 20000].float() @ W.to(torch.bfloat16).float() + (b if bias else 0.0)
        ref = F.gelu(ref, approximate="tanh") if act == 1 else F.silu(ref) if act == 2 else ref
        if res:
            ref = ref + R[r:r + 20000].float()
        worst = max(worst, float((out[r:r + 20000].float() - ref).norm() / ref.norm()))
    torch.backends.cuda.matmul.allow_tf32 = tf32
    # one bf16 rounding of the output: 2^-9 at most, 2^-9 / sqrt(3) in the mean square; the approximated GELU and SiLU half of that
    assert worst < 3e-3, worst


@pytest.mark.parametrize("M,K,N", [(2400, 2048, 512), (4700, 2048, 512), (5000, 256, 512), (5000, 640, 640), (30000, 448, 896),
                                   (1300, 3072, 768), (3000, 1024, 448), (5000, 128, 1024), (700, 64, 2560)])
def test_residual_with_a_long_bias(M, K, N):
    _gemm(M, K, N, 0, True)
    _gemm(M, K, N, 2, True, bias=False)


def test_long_bias_off_sixteen_bytes():
    """Copied to shared memory whatever its alignment, at the cost of a stage."""
    _gemm(5000, 640, 640, 0, True, bias_offset=1)
    _gemm(2400, 2048, 512, 0, True, bias_offset=3)


def test_long_bias_read_in_place_has_to_be_aligned():
    """Beyond 2048 columns the bias is read from global memory, sixteen bytes at a time: refused on the host otherwise."""
    with pytest.raises(CssmError):
        _gemm(5000, 64, 2304, 0, False, bias_offset=1)


def test_default_widths():
    """The constructor's own widths (128 to 512): 64 images of 224 x 224, whose last stage has 25 row tiles, against the oracle, and the
    host entry, which takes 128 in two chunks."""
    kw = dict(embed_dims=(128, 256, 384, 512), depths=(1, 2, 4, 1))
    p, s = sv.init_shvit_params(3, (224, 224), num_classes=10, **kw)
    bound = CSSMSHViT(num_classes=10).bind({"params": p, "batch_stats": s})
    x = torch.randn((128, 224, 224, 3), generator=torch.Generator().manual_seed(0)).to(torch.bfloat16)
    y = bound(x[:64].cuda()).cpu().numpy()
    ref = sv.shvit_forward(p, s, x[[0, 63]].float().numpy().astype(np.float64), **kw)
    assert orc.rel_l2(y[[0, 63]], ref) <= 2e-2
    xh, lh = x.pin_memory(), torch.empty((128, 10), dtype=torch.float32).pin_memory()
    bound.forward_host(xh, lh)
    assert np.array_equal(lh[:64].numpy(), y)
    assert device_error() == 0


@pytest.mark.parametrize("M,K,N,act", [(60001, 64, 64, 0), (40001, 64, 192, 2), (100003, 256, 512, 1), (30011, 384, 576, 0), (25001, 576, 1344, 1),
                                       (9001, 128, 2304, 2), (20001, 96, 160, 0), (50001, 448, 320, 1)])
def test_several_tiles_a_cta(M, K, N, act):
    """No residual, more tiles than SMs: accumulators, ring and slots come round; an odd number of 64-column boxes, which the two warps of a
    quadrant take in turn; a bias from global memory; direct stores (160 columns)."""
    _gemm(M, K, N, act, False)


@pytest.mark.parametrize("B,H,Cin,Cout,act", [(256, 28, 64, 576, 0), (260, 27, 64, 576, 1), (20, 28, 128, 960, 0)])
def test_conv_of_192_column_tiles(B, H, Cin, Cout, act):
    """The strided conv at widths of 192-column tiles whose bias would take the fourth stage: seven tiles a CTA, and fewer."""
    L = lib()
    st = torch.cuda.current_stream().cuda_stream
    g = torch.Generator(device="cuda").manual_seed(B + Cout)
    x = torch.randn((B, H, H, Cin), device="cuda", generator=g).to(torch.bfloat16)
    W = torch.randn((3, 3, Cin, Cout), device="cuda", generator=g) / (9 * Cin) ** 0.5
    b = torch.randn((Cout,), device="cuda", generator=g)
    wt = torch.empty((Cout, L.cssm_bf16_conv3x3s2_packed_ld(Cin, H, Cout)), dtype=torch.bfloat16, device="cuda")
    check(L.cssm_bf16_pack_conv3x3s2_weight(W.data_ptr(), Cin, Cout, H, None, wt.data_ptr(), st), "pack")
    Ho = (H + 1) // 2
    out = torch.full((B, Ho, Ho, Cout), float("nan"), dtype=torch.bfloat16, device="cuda")
    check(L.cssm_bf16_conv3x3s2(x.data_ptr(), B, H, H, Cin, wt.data_ptr(), Cout, b.data_ptr(), act, out.data_ptr(), st), "conv")
    # 'SAME' of stride 2: one row and column of zeros behind an even plane, one on each side of an odd one
    xp = F.pad(x.double().permute(0, 3, 1, 2), (0, 1, 0, 1) if H % 2 == 0 else (1, 1, 1, 1))
    ref = F.conv2d(xp, W.to(torch.bfloat16).double().permute(3, 2, 0, 1), b.double(), stride=2).permute(0, 2, 3, 1)
    ref = F.gelu(ref, approximate="tanh") if act else ref
    assert device_error() == 0
    assert float((out.double() - ref).norm() / ref.norm()) < 3e-3
