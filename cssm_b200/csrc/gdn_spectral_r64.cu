// GDN fused spectral kernel for 64x64 planes, d_k = d_v = 4, static images (one frame of q, k, v per batch element, the T gate steps
// run per bin; frames of their own: csrc/gdn_spectral_p64.cu).  A CTA runs one (batch, head) after another
// with two groups of 288 threads, each with its own transform buffers: a group transforms
// every other q / k plane into the shared spectra (shared memory, in the column lanes' own bin order),
// the norms are applied there in place, and then each group takes every other v plane: transform,
// all steps of its state row, readout, inverse transform over the v plane.
//
// Bound: the T steps of a bin, four rows of sixteen complex products rounded to bfloat16.  The two groups fit next to the spectra because a
// group's inverse columns go over its forward rows (one more barrier a v row) and the lanes without a column need no spectrum slot
// and one exchange region.
#include "r64.cuh"
#include "kernels.cuh"
#include "gdn_common.cuh"

namespace cssm {

constexpr int G64_NT = 2 * R64_NT;
constexpr int G64_COLS = 33 * 8;                       // lanes with a column
constexpr int G64_EXG = 34;                            // exchange regions of a group
constexpr int G64_SPEC_CF = 8 * 8 * G64_COLS;          // [plane 0..7][q 0..7][column lane]
constexpr int G64_ZR_CF = R64_ZR_CF > R64_GB_CF ? R64_ZR_CF : R64_GB_CF;
constexpr int G64_GRP_CF = G64_EXG * EX_GROUP_STRIDE + G64_ZR_CF;
constexpr int G64_SMEM_CF = G64_SPEC_CF + 2 * G64_GRP_CF;
static_assert(G64_SMEM_CF * sizeof(cf) <= 226 * 1024, "one CTA per SM");

// r64_init for one group; the lanes without a column share the last exchange region
__device__ __forceinline__ void g64_init(R64Ctx& c, cf* EX, cf* ZR, int tid) {
  c.EX = EX; c.ZR = ZR; c.GB = ZR;
  c.warp = tid >> 5; c.lane = tid & 31; c.sub = c.lane & 3; c.a = c.lane >> 2;
  c.grp = c.warp * 4 + c.sub;
  c.row_on = c.warp < 8; c.col_warp = true; c.col_on = c.grp <= 32;
  c.exg = EX + min(c.grp, G64_EXG - 1) * EX_GROUP_STRIDE;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    float s, co;
    sincospif(-(float)(c.a * k) / 32.0f, &s, &co);
    c.tw[k] = mk(co, s);
  }
}

__global__ void __launch_bounds__(G64_NT, 1) gdn_spectral_r64(const GdnSpectralArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ float red[2][9][4];
  cf* SPEC = reinterpret_cast<cf*>(smem_raw);
  const int half = threadIdx.x >= R64_NT ? 1 : 0, tid = threadIdx.x - half * R64_NT;
  cf* own = SPEC + G64_SPEC_CF + half * G64_GRP_CF;

  R64Ctx c;
  cf* ZR = own + G64_EXG * EX_GROUP_STRIDE;
  g64_init(c, own, ZR, tid);
  auto group_sync = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(half + 1), "n"(R64_NT) : "memory"); };
  constexpr int HW = 4096, NB = 64 * 33, DK = 4;
  const int nh = a.C / DK, heads = a.B * nh;
  const float invHW = 1.0f / (float)HW;
  // slot of this lane in the spectra (warp 8 has one column: lanes 0, 4, 8, ...)
  const int slot = c.warp < 8 ? tid : 256 + c.a;
  pdl_sync();

  // plane 2 i + half: i = 0, 1 q, 2, 3 k, 4, 5 v; i = 6: the first of the next head
  auto plane_of = [&](int bh, int i) -> float* {
    if (i >= 6) { bh += gridDim.x; i = 0; }
    if (bh >= heads) bh = blockIdx.x;                       // harmless re-read past the end
    const int b = bh / nh, hd = bh - b * nh, idx = 2 * i + half;
    return a.qkv + ((size_t)b * 3 * a.C + (size_t)(idx >> 2) * a.C + hd * DK + (idx & 3)) * HW;
  };
  cf nx[8];                                   // rows of the NEXT plane, fetched one pass ahead
  r64_load_rows(c, plane_of(blockIdx.x, 0), nx);

  for (int bh = blockIdx.x; bh < heads; bh += gridDim.x) {
    const int b = bh / nh, hd = bh - b * nh;
    const cf* wh = a.what + (size_t)hd * NB + (c.grp << 3) + c.a;
    // ---- q planes (i = 0, 1) and k planes (i = 2, 3) ----
#pragma unroll 1
    for (int i = 0; i < 4; ++i) {
      // own ZR free; at the first plane also: nobody reads the spectra of the head before any more
      if (i == 0) __syncthreads(); else group_sync();
      {
        cf cur[8];
#pragma unroll
        for (int m = 0; m < 8; ++m) cur[m] = nx[m];
        r64_load_rows(c, plane_of(bh, i + 1), nx);
        r64_row_fwd_regs(c, cur);
      }
      group_sync();
      float acc = 0.f;
      cf v[8];
      r64_col_fwd(c, v);
      if (c.col_on) {
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          SPEC[((2 * i + half) * 8 + q) * G64_COLS + slot] = v[q];
          acc += v[q].x * v[q].x + v[q].y * v[q].y;
        }
      }
      for (int off = 16; off > 0; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off);
      if (c.lane == 0) red[half][c.warp][i] = acc;
    }
    __syncthreads();
    // ---- normalise in place, the bins split between the groups:
    //      q_hat = q*nq; k_hat = (k*nk) / sqrt(sum_i |.|^2 + 1e-6)
    {
      float mine = 0.f;                      // lanes 0..7: plane norms
      if (c.lane < 8) {
#pragma unroll
        for (int w = 0; w < 9; ++w) mine += red[c.lane & 1][w][c.lane >> 1];
        mine = a.use_l2 ? rsqrtf(mine + 1e-6f) : 1.f;
      }
      float nrm[8];
#pragma unroll
      for (int p = 0; p < 8; ++p) nrm[p] = __shfl_sync(0xffffffffu, mine, p);
      if (c.col_on) {
        cf* sp = SPEC + half * 4 * G64_COLS + slot;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          cf kv[4];
          float ks = 0.f;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const cf z = sp[((4 + i) * 8 + q) * G64_COLS];
            kv[i] = mk(z.x * nrm[4 + i], z.y * nrm[4 + i]);
            ks += kv[i].x * kv[i].x + kv[i].y * kv[i].y;
            const cf qq = sp[(i * 8 + q) * G64_COLS];
            sp[(i * 8 + q) * G64_COLS] = mk(qq.x * nrm[i], qq.y * nrm[i]);
          }
          const float kn = rsqrtf(ks + 1e-6f);
#pragma unroll
          for (int i = 0; i < 4; ++i) sp[((4 + i) * 8 + q) * G64_COLS] = mk(kv[i].x * kn, kv[i].y * kn);
        }
      }
    }
    __syncthreads();
    // gates of step 0 of this batch element's T steps
    const float2* abp = a.ab + ((size_t)b * a.T * a.ab_heads + (a.ab_heads > 1 ? hd : 0)) * NB + (c.grp << 3) + c.a;
    // ---- v rows: transform, state update, readout, inverse transform over the v plane ----
#pragma unroll 1
    for (int i = 4; i < 6; ++i) {
      const int vr = 2 * (i - 4) + half;
      if (i > 4) group_sync();               // ZR free: the row before has left it
      r64_row_fwd_regs(c, nx);
      group_sync();
      cf v[8];
      r64_col_fwd(c, v);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        cf kk[4], qq[4], o = mk(0.f, 0.f);
        if (c.col_on) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            qq[j] = SPEC[(j * 8 + q) * G64_COLS + slot];
            kk[j] = SPEC[((4 + j) * 8 + q) * G64_COLS + slot];
          }
          o = gdn_bin_static<4>(kk, qq, v[q], wh[q * 264], abp + q * 264, (size_t)a.ab_heads * NB, a.T);
        }
        v[q] = mk(o.x * invHW, o.y * invHW);
      }
      r64_load_rows(c, plane_of(bh, i + 1), nx);
      fft64_lane8<true>(v, c.tw, c.exg, c.a);
      group_sync();                          // every column of ZR has been read: GB may go over it
#pragma unroll
      for (int n1 = 0; n1 < 8; ++n1)
        if (c.col_on) c.GB[(c.a + 8 * n1) * R64_GBS + c.grp] = v[n1];
      group_sync();
      if (c.row_on) {
        r64_row_inv(c, v);
        float* y0 = a.qkv + ((size_t)b * 3 * a.C + 2 * a.C + hd * DK + vr) * HW + (2 * c.grp) * 64 + c.a;
#pragma unroll
        for (int n1 = 0; n1 < 8; ++n1) {
          y0[8 * n1] = v[n1].x;
          y0[64 + 8 * n1] = v[n1].y;
        }
      }
    }
  }
}

int launch_gdn_spectral_r64(const GdnSpectralArgs& a, cudaStream_t st) {
  if (!a.static_image) return CSSM_ERR_UNSUPPORTED;
  const size_t smem = (size_t)G64_SMEM_CF * sizeof(cf);
  cudaError_t e = func_smem(gdn_spectral_r64, smem);
  if (e != cudaSuccess) { set_cuda_error(e); return CSSM_ERR_CUDA; }
  const int heads = a.B * (a.C / 4), sms = sm_count();
  launch_k(gdn_spectral_r64, heads < sms ? heads : sms, G64_NT, smem, st, a);
  return check_launch();
}

}  // namespace cssm
