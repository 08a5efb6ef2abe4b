// Fused spectral kernels of the two delta-rule blocks (GatedDeltaNetCSSM of key dimension 2 and 4, DeltaNetCSSM) for square planes of the sides
// in PF_SIDES, with whole FFTs in a lane's registers (csrc/plane_fft.cuh); other planes and key dimensions: csrc/delta_spectral_dft.cu.
//
// A CTA takes some heads of one batch element (DeltaNet: channels) and walks the steps.  A step: the warps transform the q, k and v planes,
// at most G of them each (and the step before's output back, which lies where v was), with the planes' energies on the way; then all
// threads share the bins.  The states lie in shared memory, or in the caller's scratch where that leaves more room for CTAs.
//
// Bound: instruction issue and the latency of the step's chain at 8 to 16 warps an SM.  The folded DFT (O(N) work a value) it took over from,
// passes in us, before -> now: GDN 12 x 8 x 28 x 28 x 64, key dimension 2 214 -> 171, 4 307 -> 181; 12 x 8 x 48 x 48 x 64 791 -> 310, 3170 -> 413 (key dimension 4
// did not fit in shared memory from 48 on); DeltaNet 12 x 8 x 28 x 28 x 64 228 -> 170, 12 x 8 x 8 x 8 x 64 76 -> 66; geometric mean over 24 sides and
// five batches 1.26 (key dimension 2), 1.69 (4) and 1.24 (DeltaNet) times as fast.
#pragma once
#include <string.h>
#include "kernels.cuh"
#include "plane_fft.cuh"
#include "gdn_common.cuh"

namespace cssm {

extern __shared__ __align__(16) float pf_smem[];

struct DeltaFftArgs {
  int B, T, C, heads, hgroups, tasks;      // heads a CTA; tasks: groups of at most G planes of one of q, k, v
  int smem_state, last_only, use_l2;
};

// Registers: the FFTs take some 2.2 N + 25, the bins of key dimension 4 a hundred.
constexpr int delta_fft_warps(int n, int dk) { return n <= 16 ? (dk == 4 ? 16 : 20) : n <= 32 ? 16 : 12; }

// GDN's and DeltaNet's bins differ in Rule: bins(), and scale_keys(), which may scale the key spectra of a lane's column.
template <int N, int DK, class Rule>
__global__ void __launch_bounds__(512) __maxnreg__(65536 / 32 / delta_fft_warps(N, DK) / 8 * 8)
delta_spectral_fft(const typename Rule::Args a, const DeltaFftArgs d) {
  typedef Pf<N> P;
  pdl_sync();
  const int b = blockIdx.x / d.hgroups, h0 = (blockIdx.x - b * d.hgroups) * d.heads, nh = min(d.heads, d.C / DK - h0), n = nh * DK;
  float* nrm = pf_smem + 3 * d.heads * DK * P::PLANE;                   // [q | k][n] half the scales of the planes
  float4* state = reinterpret_cast<float4*>(nrm + (3 * d.heads * DK + 3) / 4 * 4);
#pragma unroll 1
  for (int t = 0; t <= d.T; ++t) {
    const bool emit = !d.last_only || t == d.T - 1, emitted = t > 0 && (!d.last_only || t == d.T);
    // transforms: half of the warps take v (the step before's output back first), the others q and k; or every warp all three
    const int warps = blockDim.x >> 5, split = warps >= 2 * d.tasks ? 1 : 0;
#pragma unroll 1
    for (int u = 0; u < 4; ++u) {
      const int warp = pf_warp(), task = split && warp >= d.tasks ? warp - d.tasks : warp;
      const bool vw = warp < d.tasks;                                   // u 0: output back, 1: v, 2: q, 3: k
      if (u < 2 ? !vw : split && vw) continue;
      if (u == 0 ? !emitted : t == d.T || (u == 2 && !emit)) continue;
      const int role = u == 2 ? 0 : u == 3 ? 1 : 2, p0 = task * P::GMAX, m = min(P::GMAX, n - p0);
      if (m <= 0) continue;
      float* region = pf_smem + (role * n + p0) * P::PLANE;
      float* gp = Rule::planes(a) + (((size_t)b * d.T + (u == 0 ? t - 1 : t)) * 3 * d.C + (size_t)role * d.C + h0 * DK + p0) * (N * N);
      if (u > 0) {
        P::load(gp, region, m);
        P::wait();
      }
#pragma unroll 1
      for (int pass = 0; pass < 2; ++pass) {
        const int lane = pf_lane(), pc = lane / P::WF, kw = lane - pc * P::WF, pr = lane / P::HH, j = lane - pr * P::HH;
        const bool rows = (pass == 0) == (u > 0), two = j + P::HH < N;
        float e = 0.f;
        if (rows ? pr < m : pc < m) {
          float* at = region + (rows ? pr * P::PLANE + j * P::PITCH : pc * P::PLANE + 2 * kw);
          cf z[N];
          if (!rows) P::load_col(at, z);
          else if (u > 0) P::load_rows(at, two, z);
          else P::get_rows(at, two, z);
          lane_dft<N>(z);
          if (!rows) {
            if (u == 3 && Rule::SCALE_KEYS) Rule::scale_keys(a, (size_t)b * d.T + t, kw, z);
            if (u >= 2) {
#pragma unroll
              for (int h = 0; h < N; ++h) e = fmaf(z[h].x, z[h].x, fmaf(z[h].y, z[h].y, e));
            }
            P::store_col(at, z);
          } else if (u > 0) P::put_rows(at, two, z);
          else P::store_rows(at, two, z);
        }
        if (!rows && u >= 2) {
          // half-spectrum energies of the planes, in a fixed order
#pragma unroll 1
          for (int p = 0; p < m; ++p) {
            float s = pc == p ? e : 0.f;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (lane == 0) nrm[role * n + p0 + p] = d.use_l2 ? 0.5f * rsqrtf(0.25f * s + 1e-6f) : 0.5f;
          }
        }
        __syncwarp();
      }
      if (u == 0) P::template store<false>(region, gp, nullptr, m);
    }
    if (t == d.T) break;
    __syncthreads();
    Rule::template bins<N>(a, d, b, t, h0, nh, nrm, state, emit);
    __syncthreads();
  }
}

struct DeltaFftPlan { int heads, warps, ctas, tasks, smem_state; size_t smem; double cost; };

template <int N, int DK>
inline size_t delta_fft_bytes(int heads, bool st) {
  return (size_t)3 * heads * DK * Pf<N>::PLANE * 4 + (size_t)(3 * heads * DK + 3) / 4 * 16 + (st ? (size_t)heads * DK * DK * Pf<N>::NB * 8 : 0);
}
// Heads and warps of a CTA, and where the states lie, by an estimate of a step's time: the transforms of the longest warp (split: half of the
// warps have v and the output, the others q and k), the bins shared out, fixed parts, times what the waves of CTAs cost (as in
// csrc/gated_spectral_fft.cu; a CTA of one warp 1.1 times that: 382 x 1 x 7 x 7 x 32 63 us with four heads and one warp, 59 with eight and two).
// Of 78 shapes it is within 3 % of the best of all choices on 74, and 4 to 7 % off on the others, which are of one or two frames.
template <int N, int DK>
inline DeltaFftPlan delta_fft_plan(int B, int C, int T, bool need_smem_state) {
  const int most = delta_fft_warps(N, DK), sms = sm_count(), nh = C / DK;
  DeltaFftPlan best;
  best.cost = 1e30; best.heads = 0;
  for (int heads = 1; heads <= nh && heads <= 16; ++heads) {
    const int n = heads * DK, tasks = (n + Pf<N>::GMAX - 1) / Pf<N>::GMAX;
    if (tasks > 8 || (heads > 1 && (long long)B * ((nh + heads - 1) / heads) * 2 < sms)) break;
    for (int v = 0; v < 4; ++v) {
      const bool st = (v & 1) == 0, split = v & 2;
      if (!st && (need_smem_state || T == 1)) continue;
      const int warps = split ? 2 * tasks : tasks;
      const size_t smem = delta_fft_bytes<N, DK>(heads, st && T > 1);
      int c = (int)(227 * 1024 / (smem + 1024));
      if (c * warps > most) c = most / warps;
      if (c < 1) continue;
      const long long groups = (long long)B * ((nh + heads - 1) / heads), slots = (long long)sms * c;
      const long long full = groups / slots, rest = (groups % slots + sms - 1) / sms;
      const double fft = (split ? 2 : 4) * 2.0 * N * 20 * (0.7 + 0.3 * (double)n / (tasks * Pf<N>::GMAX));
      const double bin = (double)heads * Pf<N>::NB / (32 * warps) * (DK * DK * 28 + 60) * (st ? 1.0 : 1.4);
      const double cost = (warps == 1 ? 1.1 : 1.0) * (fft + bin + 400 + 1500.0 / T) * (full * (3.7 + 0.17 * c * warps) + (rest > 0 ? 3.7 + 0.17 * rest * warps : 0));
      if (cost < best.cost * 0.98) best = {heads, warps, c, tasks, st && T > 1 ? 1 : 0, smem, cost};
    }
  }
  return best;
}

template <int N, int DK, class Rule>
inline int delta_fft_launch(const typename Rule::Args& a, int B, int T, int C, int last_only, int use_l2, bool need_smem_state, cudaStream_t st) {
  const DeltaFftPlan p = delta_fft_plan<N, DK>(B, C, T, need_smem_state);
  if (p.heads == 0) return CSSM_ERR_UNSUPPORTED;
  DeltaFftArgs d;
  d.B = B; d.T = T; d.C = C; d.heads = p.heads; d.hgroups = (C / DK + p.heads - 1) / p.heads; d.tasks = p.tasks;
  d.smem_state = p.smem_state; d.last_only = last_only; d.use_l2 = use_l2;
  const size_t smem = spread_smem(p.smem, (long long)B * d.hgroups);
  const cudaError_t e = func_smem(delta_spectral_fft<N, DK, Rule>, smem);
  if (e != cudaSuccess) { set_cuda_error(e); return CSSM_ERR_CUDA; }
  launch_k(delta_spectral_fft<N, DK, Rule>, B * d.hgroups, 32 * p.warps, smem, st, a, d);
  return check_launch();
}

}  // namespace cssm
