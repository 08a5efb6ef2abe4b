// GDN fused spectral kernel for 32x32 planes, d_k = d_v = 4.  A CTA (288 threads, two per SM) runs one
// (batch, head) after another.  The four planes of q, of k and of v are each transformed side by side
// (r32.cuh geometry: plane = group / 17 in column passes).  Per step:
//   1. q planes: rows, columns -> spectra parked in shared memory (SPEC), sum |.|^2 per plane
//   2. k planes: the same
//   3. v planes: rows, columns -> each column lane (v row = its plane) reads the 4 k and 4 q
//      values of its bins from SPEC, normalises them, updates its state row S[v][0..3], reads out
//      o[v], inverse columns, inverse rows -> o planes over the v planes.
// Bound: the shared-memory pipe and the latency of the barriered passes.  With the state in shared memory
// (70 KB per head) one CTA of nine warps fits an SM; the state of the running heads (20 MB) stays in L2
// just as well: scratch goes by CTA, not by head, a bin's row is requested two bins ahead, the first step
// reads none and the last one writes none.  128 x 32 x 32 x 32 x 64: 4.59 -> 3.85 ms.  Where every head has an SM of
// its own (SMST) the state stays in shared memory, which is nearer: block 4 x 32 x 32 x 32 x 64 (64 heads) 743 us
// from L2 (two CTAs on one SM at that), 536 so; 9 x 32 (144 heads) 905 and 695; 10 x 32 (160 heads) 933 from L2,
// 1031 with one CTA per SM and its state in shared memory.
#include "r32.cuh"
#include "kernels.cuh"
#include "gdn_common.cuh"

namespace cssm {

constexpr int G32_THREADS = 288;
constexpr int G32_ZRS = 36, G32_GBS = 18;
constexpr int G32_EX_CF = 72 * EX32_STRIDE;
constexpr int G32_ZR_CF = 4 * 16 * G32_ZRS;
constexpr int G32_GB_CF = 4 * 32 * G32_GBS;
constexpr int G32_SPEC_CF = 8 * 8 * 17 * 4;            // [q planes 0-3, k planes 4-7][r][kw][q]
constexpr int G32_COLS = 68 * 4;                        // lanes with a column
constexpr int G32_SMEM_BYTES = (G32_EX_CF + G32_ZR_CF + G32_GB_CF + G32_SPEC_CF) * 8;
static_assert(G32_SMEM_BYTES <= 112 * 1024, "two CTAs per SM");
constexpr int G32_STATE_BYTES = 4 * 8 * G32_COLS * 8;   // [i][r][column lane]
static_assert(G32_SMEM_BYTES + G32_STATE_BYTES <= 226 * 1024, "one CTA per SM");

// LAST: only the last step's output planes are produced (compile-time switch).
// STATIC: static-image fast path (one data frame per batch element, the T gate steps run per bin).
// SMST: state in shared memory, one CTA per SM.
template <bool LAST, bool STATIC, bool SMST>
__global__ void __launch_bounds__(G32_THREADS, STATIC || SMST ? 1 : 2) gdn_spectral_r32(const GdnSpectralArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cf* EX = reinterpret_cast<cf*>(smem_raw);
  cf* ZR = EX + G32_EX_CF;
  cf* GB = ZR + G32_ZR_CF;
  cf* SPEC = GB + G32_GB_CF;
  __shared__ float red[9][8];

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int q = lane & 3, g8 = lane >> 2;
  const int grp = warp * 8 + g8;
  cf* exg = EX + grp * EX32_STRIDE;
  const bool row_on = warp < 8;
  const bool col_on = grp < 68;
  constexpr int HW = 1024, NB = 32 * 17, DK = 4;
  const int nh = a.C / DK, heads = a.B * nh;

  cf tw[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    float s, co;
    sincospif(-(float)(q * k) / 16.0f, &s, &co);
    tw[k] = mk(co, s);
  }
  const int rpl = grp >> 4, rpair = grp & 15;
  const int roff = (2 * rpair) * 32 + q;
  const int cpl = col_on ? grp / 17 : 0, kw = col_on ? grp % 17 : 0;
  const int kneg = (32 - kw) & 31;
  const int par = q & 1, ph = q >> 1;

  // state S[i][r][column lane]; a thread only ever touches its own slots
  cf* S = (SMST ? SPEC + G32_SPEC_CF : a.state + (size_t)blockIdx.x * DK * DK * NB) + tid;
  const float invHW = 1.0f / (float)HW;

  const int Tdata = STATIC ? 1 : a.T;          // frames of q, k, v per batch element
  // rows of the NEXT pass's planes, fetched one pass ahead; pass 3: the first of step t + 1 (of the
  // next head).  last_only: steps before the last one skip the q planes.
  auto first_pass = [&](int t) -> int { return (LAST && t < Tdata - 1) ? 1 : 0; };
  cf nx[8];
  auto fetch_rows = [&](int bh, int t, int pass) {
    if (!row_on) return;
    if (pass == 3) { ++t; if (t >= Tdata) { t = 0; bh += gridDim.x; } pass = first_pass(t); }
    if (bh >= heads) return;
    const int b = bh / nh, hd = bh - b * nh;
    const float* r0 = a.qkv + ((size_t)(b * Tdata + t) * 3 * a.C + (size_t)pass * a.C + hd * DK + rpl) * HW + roff;
#pragma unroll
    for (int m = 0; m < 8; ++m) nx[m] = mk(r0[4 * m], r0[32 + 4 * m]);
  };
  pdl_sync();
  fetch_rows(blockIdx.x, 0, first_pass(0));
  for (int bh = blockIdx.x; bh < heads; bh += gridDim.x) {
  const int b = bh / nh, hd = bh - b * nh;
  const cf* wh = a.what + (size_t)hd * NB + (kw << 2) + q;
  for (int t = 0; t < Tdata; ++t) {
    const size_t frame = (size_t)(b * Tdata + t);
    float* base = a.qkv + frame * 3 * a.C * HW;
    float ssq[2] = {0.f, 0.f};
    const bool emit = !LAST || t == Tdata - 1;       // same for the whole CTA
    cf v[8];
    // ---- passes 0 (q), 1 (k), 2 (v): forward transform of four planes at once ----
#pragma unroll 1
    for (int pass = emit ? 0 : 1; pass < 3; ++pass) {     // q is only needed for the readout
      __syncthreads();                       // ZR free (previous column pass finished)
      if (row_on) {
        cf u[8];
#pragma unroll
        for (int m = 0; m < 8; ++m) u[m] = nx[m];
        if (pass < 2) fetch_rows(bh, t, pass + 1);
        fft32_fwd(u, tw, exg, q);
        cf* zr = ZR + (rpl * 16 + rpair) * G32_ZRS;
#pragma unroll
        for (int r = 0; r < 8; ++r) zr[q + 4 * (r >> 2) + 8 * (r & 3)] = u[r];
      }
      __syncthreads();
      {
        const cf* zr = ZR + (cpl * 16) * G32_ZRS;
#pragma unroll
        for (int m = 0; m < 8; ++m) {
          const cf z1 = zr[(ph + 2 * m) * G32_ZRS + kw];
          const cf z2 = zr[(ph + 2 * m) * G32_ZRS + kneg];
          v[m] = par ? mk(0.5f * (z1.y + z2.y), 0.5f * (z2.x - z1.x))
                     : mk(0.5f * (z1.x + z2.x), 0.5f * (z1.y - z2.y));
        }
        fft32_fwd(v, tw, exg, q);
        if (pass < 2) {
          float acc = 0.f;
#pragma unroll
          for (int r = 0; r < 8; ++r) {
            if (col_on) {
              SPEC[(((pass * 4 + cpl) * 8 + r) * 17 + kw) * 4 + q] = v[r];
              acc += v[r].x * v[r].x + v[r].y * v[r].y;
            }
          }
          if (pass == 0) ssq[0] = acc; else ssq[1] = acc;
        }
      }
    }
    // ---- per-plane sums over all bins: lanes of plane p live in groups 17p .. 17p+16 ----
    {
      // each lane contributes to red[warp][pass*4 + plane] through a warp-level segmented sum
#pragma unroll
      for (int pass = 0; pass < 2; ++pass)
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          float c = (col_on && cpl == p) ? ssq[pass] : 0.f;
          for (int off = 16; off > 0; off >>= 1) c += __shfl_down_sync(0xffffffffu, c, off);
          if (lane == 0) red[warp][pass * 4 + p] = c;
        }
    }
    __syncthreads();                          // SPEC and red complete
    {
      float mine = 0.f;                        // lanes 0..7: plane norms
      if (lane < 8) {
#pragma unroll
        for (int w = 0; w < 9; ++w) mine += red[w][lane];
        mine = a.use_l2 ? rsqrtf(mine + 1e-6f) : 1.f;
      }
      float nrm[8];
#pragma unroll
      for (int p = 0; p < 8; ++p) nrm[p] = __shfl_sync(0xffffffffu, mine, p);
      const float2* abp = a.ab + ((STATIC ? (size_t)b * a.T : frame) * a.ab_heads + (a.ab_heads > 1 ? hd : 0)) * NB + (kw << 2) + q;
      cf sreg[2][4];
      float2 gab[2], w2[2];
      auto fetch = [&](int r) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          sreg[r & 1][i] = (t > 0 && col_on) ? S[(i * 8 + r) * G32_COLS] : mk(0.f, 0.f);
        gab[r & 1] = col_on ? __ldg(abp + r * (17 * 4)) : make_float2(0.f, 0.f);
        w2[r & 1] = col_on ? __ldg(reinterpret_cast<const float2*>(wh) + r * (17 * 4)) : make_float2(0.f, 0.f);
      };
      if (!STATIC) { fetch(0); fetch(1); }
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        cf kk[4], qq[4];
        float ks = 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const cf zk = SPEC[(((4 + i) * 8 + r) * 17 + kw) * 4 + q];
          kk[i] = mk(zk.x * nrm[4 + i], zk.y * nrm[4 + i]);
          ks += kk[i].x * kk[i].x + kk[i].y * kk[i].y;
          qq[i] = mk(0.f, 0.f);
          if (emit) {
            const cf zq = SPEC[(((0 + i) * 8 + r) * 17 + kw) * 4 + q];
            qq[i] = mk(zq.x * nrm[i], zq.y * nrm[i]);
          }
        }
        const float kn = rsqrtf(ks + 1e-6f);
#pragma unroll
        for (int i = 0; i < 4; ++i) kk[i] = mk(kk[i].x * kn, kk[i].y * kn);
        cf o = mk(0.f, 0.f);
        if (STATIC) {
          if (col_on) o = gdn_bin_static<4>(kk, qq, v[r], wh[r * (17 * 4)], abp + r * (17 * 4), (size_t)a.ab_heads * NB, a.T);
        } else {
          const float2 g = gab[r & 1];
          const cf aw = mk(g.x * w2[r & 1].x, g.x * w2[r & 1].y);
          if (emit) o = gdn_bin_update_regs<4, true>(sreg[r & 1], kk, qq, v[r], aw, g.y);
          else gdn_bin_update_regs<4, false>(sreg[r & 1], kk, qq, v[r], aw, g.y);
          if (col_on && t + 1 < Tdata) {
#pragma unroll
            for (int i = 0; i < 4; ++i) S[(i * 8 + r) * G32_COLS] = sreg[r & 1][i];
          }
          if (r + 2 < 8) fetch(r + 2);
        }
        v[r] = mk(o.x * invHW, o.y * invHW);
      }
      // the next step's first planes (q or k; this step's output goes over v planes)
      fetch_rows(bh, t, 3);
      if (emit) {
        fft32_inv(v, tw, exg, q);
        cf* gb = GB + (cpl * 32) * G32_GBS;
#pragma unroll
        for (int m = 0; m < 8; ++m)
          if (col_on) gb[(q + 4 * m) * G32_GBS + kw] = v[m];
      }
    }
    __syncthreads();
    // ---- inverse rows of the four output planes, written over the v planes ----
    if (row_on && emit) {
      const cf* ge = GB + (rpl * 32 + 2 * rpair) * G32_GBS;
      const cf* go = ge + G32_GBS;
      cf u[8];
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const int k = q + 4 * (r >> 2) + 8 * (r & 3);
        const int kk = k <= 16 ? k : 32 - k;
        cf e = ge[kk], o = go[kk];
        if ((r == 0 || r == 2) && q == 0) { e.y = 0.f; o.y = 0.f; }
        u[r] = (k <= 16) ? mk(e.x - o.y, e.y + o.x) : mk(e.x + o.y, o.x - e.y);
      }
      fft32_inv(u, tw, exg, q);
      float* y0 = base + (size_t)(2 * a.C + hd * DK + rpl) * HW + roff;
#pragma unroll
      for (int m = 0; m < 8; ++m) {
        y0[4 * m] = u[m].x;
        y0[32 + 4 * m] = u[m].y;
      }
    }
  }
  }
}

int launch_gdn_spectral_r32(const GdnSpectralArgs& a, cudaStream_t st) {
  const int heads = a.B * (a.C / 4), sms = sm_count(), slots = (a.static_image ? 1 : 2) * sms;
  const bool smst = heads <= sms && !a.static_image;
  auto kern = a.static_image ? gdn_spectral_r32<false, true, false>
              : smst ? (a.last_only ? gdn_spectral_r32<true, false, true> : gdn_spectral_r32<false, false, true>)
                     : (a.last_only ? gdn_spectral_r32<true, false, false> : gdn_spectral_r32<false, false, false>);
  const size_t smem = G32_SMEM_BYTES + (smst ? G32_STATE_BYTES : 0);
  cudaError_t e = func_smem(kern, smem);
  if (e != cudaSuccess) { set_cuda_error(e); return CSSM_ERR_CUDA; }
  const PdlOff alone(uneven_rounds(heads, a.static_image ? 1 : 2));
  launch_k(kern, heads < slots ? heads : slots, G32_THREADS, smem, st, a);
  return check_launch();
}

}  // namespace cssm
