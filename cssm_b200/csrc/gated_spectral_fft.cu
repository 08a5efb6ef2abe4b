// Fused spectral kernel of the gated block for square planes of the sides in PF_SIDES (64x64 and 32x32 have their own, others
// csrc/gated_spectral_dft.cu): rfft2 -> gated recurrence over T -> irfft2 -> * silu(z), with whole FFTs in a lane's registers
// (csrc/plane_fft.cuh).
//
// A CTA of F warps takes G consecutive channels of one batch element, F frames at a time, a warp a frame: each transforms its frame, then
// all warps share the bins of the F frames (a thread has a column's bins in HB rows, frame after frame, so a bin's state
// is read and written once in F frames and no warp waits for another's recurrence), then each transforms its frame back.
//
// Bound: instruction issue (46 to 50 % of the slots, shared-memory pipe 34 to 59 %) at the 12 to 20 warps an SM that registers and planes leave.
// The folded DFT (O(N) work a value, shared-memory operands) it took over from, passes in us, before -> now:
// gated 16 x 8 x 56 x 56 x 32 343 -> 236, 3 x 8 x 48 x 48 x 64 152 -> 87, 24 x 8 x 28 x 28 x 64 207 -> 142, 64 x 8 x 14 x 14 x 64 140 -> 116, 159 x 8 x 7 x 7 x 64
// 108 -> 89; geometric mean over 44 sides and three batches 1.185 times as fast.  On the way (28 x 28, a pass): frames handed from
// warp to warp along the recurrence 155 to 223 (a step's bins are then one long chain), passes as calls 189 to 290 (callee-saved registers
// through local memory, which misses L1 beside this much shared memory).
#define CSSM_F32X2 0          // (a lane's FFT is register renaming then: csrc/lane_fft.cuh)
#include <string.h>
#include "kernels.cuh"
#include "plane_fft.cuh"

namespace cssm {

struct GatedFftArgs {
  float* xz; const cf* khat; const float4* gates; const float* dchan;
  int B, T, C, G, cgroups, groups, last_only, mode;           // mode: see launch_spectral
  int equal;          // > 0: clips of equal frames, of which the T first are there: steps of frame T - 1 (z planes: the first frame's)
};

// Warps an SM, and so registers a thread (96, 128, 168: the FFTs alone take some 2.2 N + 25).
constexpr int gated_fft_warps(int n) { return n <= 16 ? 20 : n <= 32 ? 16 : 12; }

extern __shared__ __align__(16) float pf_smem[];

// A batch of F frames: warp `warp` has HB rows of bins of every column, all frames of them.  f: the lane's column in the first
// frame's region (frames `stride` floats apart), st: its state, gx, kx: gates and kernel spectrum of its column.
template <int N, int F, bool EQUAL>
__device__ __forceinline__ void gated_bins(const GatedFftArgs& a, float* f, int stride, float2* st, const float4* gx, const float2* kx, const float* dcp,
                                           int warp, int nf, bool on, bool first, bool keep, bool all, bool end) {
  typedef Pf<N> P;
  constexpr int HB = (N + F - 1) / F, U = 4 / F;              // rows whose gates and kernel spectra are on their way
  const int hb = min(warp * HB, N - 1), cnt = min(HB, N - warp * HB);      // (small planes: the last warps have none)
  f += hb * P::PITCH; st += 32 * hb; gx += hb * P::WF; kx += hb * P::WF;
  const bool gates = a.mode != 1, need_k = !first || nf > 1 || EQUAL;
  float dc[F];
#pragma unroll
  for (int i = 0; i < F; ++i) dc[i] = dcp != nullptr ? __ldg(dcp + (size_t)min(i, nf - 1) * a.C) : 1.f;
  float4 gt[U][F];
  float2 k[U];
  // (never skipped: a skipped load would keep its registers live through the whole step)
  auto fetch = [&](int u, int h) {
    const int hc = max(0, min(h, cnt - 1));
#pragma unroll
    for (int i = 0; i < F; ++i)
      gt[u][i] = gates ? __ldg(gx + hc * P::WF + min(i, nf - 1) * P::NB) : make_float4(1.f, 1.f, 1.0f / (N * N), 0.f);
    k[u] = need_k ? __ldg(kx + hc * P::WF) : make_float2(0.f, 0.f);
  };
#pragma unroll
  for (int u = 0; u < U; ++u) fetch(u, u);
  if (F > 1) __syncthreads();
  if (!on) return;
#pragma unroll 1
  for (int h0 = 0; h0 < cnt; h0 += U) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const bool in = h0 + u < cnt;
      float2 x[F], s = make_float2(0.f, 0.f);
#pragma unroll
      for (int i = 0; i < F; ++i) x[i] = in && i < nf ? *reinterpret_cast<const float2*>(f + i * stride + u * P::PITCH) : make_float2(0.f, 0.f);
      if (!first && in) s = st[32 * u];
      cf h = mk(s.x, s.y);
#pragma unroll
      for (int i = 0; i < F; ++i) {
        const float4 g = gt[u][i];
        const float ga = g.x * dc[i], gu = 0.5f * g.y;                   // (spectra are doubled)
        const cf A = mk(k[u].x * ga, k[u].y * ga);
        cf V = mk(gu * x[i].x, gu * x[i].y);
        if (V.x * V.x + V.y * V.y < g.w * g.w) V = mk(g.w, 0.f);
        if (i < nf) {
          h = mk(fmaf(A.x, h.x, fmaf(-A.y, h.y, V.x)), fmaf(A.x, h.y, fmaf(A.y, h.x, V.y)));
          if (EQUAL && end && i == nf - 1)
            for (int r = 1; r < a.equal; ++r) h = mk(fmaf(A.x, h.x, fmaf(-A.y, h.y, V.x)), fmaf(A.x, h.y, fmaf(A.y, h.x, V.y)));
          if (in && (all || (end && i == nf - 1))) *reinterpret_cast<float2*>(f + i * stride + u * P::PITCH) = make_float2(g.z * h.y, g.z * h.x);
        }
      }
      if (keep && in) st[32 * u] = make_float2(h.x, h.y);
      fetch(u, h0 + u + U);
    }
    f += U * P::PITCH; st += 32 * U;
  }
}

template <int N, int F>
__global__ void __launch_bounds__(32 * F) __maxnreg__(65536 / 32 / gated_fft_warps(N) / 8 * 8) gated_spectral_fft(const GatedFftArgs a) {
  typedef Pf<N> P;
  pdl_sync();
  const int batches = (a.T + F - 1) / F;
#pragma unroll 1
  for (int s = 0; s < (a.groups - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x * batches; ++s) {
    const int gi = s / batches, grp = blockIdx.x + gi * gridDim.x, t0 = (s - gi * batches) * F;
    const int b = grp / a.cgroups, c0 = (grp - b * a.cgroups) * a.G, n = min(a.G, a.C - c0), nf = min(F, a.T - t0);
    const bool end = t0 + F >= a.T;
    {
      const int warp = pf_warp();
      if (warp < nf) {
        P::load(a.xz + (((size_t)b * a.T + t0 + warp) * 2 * a.C + c0) * (N * N), pf_smem + warp * a.G * P::PLANE, n);
        P::wait();
      }
    }
#pragma unroll 1
    for (int pass = 0; pass < 4; ++pass) {
      if (pass == 2) {
        const int lane = pf_lane(), warp = pf_warp(), pc = lane / P::WF, kw = lane - pc * P::WF;
        const size_t frame = (size_t)b * a.T + t0;
        float* f = pf_smem + pc * P::PLANE + 2 * kw;
        float2* st = reinterpret_cast<float2*>(pf_smem + F * a.G * P::PLANE) + lane;
        const float4* gx = a.gates + frame * P::NB + kw;
        const int pk = min(pc, n - 1);
        const float2* kx = reinterpret_cast<const float2*>(a.khat) + (size_t)(c0 + pk) * P::NB + kw;
        const float* dc = a.mode == 3 ? a.dchan + frame * a.C + c0 + pk : nullptr;
        if (a.equal > 0) gated_bins<N, F, true>(a, f, a.G * P::PLANE, st, gx, kx, dc, warp, nf, pc < n, t0 == 0, !end, !a.last_only, end);
        else gated_bins<N, F, false>(a, f, a.G * P::PLANE, st, gx, kx, dc, warp, nf, pc < n, t0 == 0, !end, !a.last_only, end);
        if (F > 1) __syncthreads(); else __syncwarp();
      }
      const int lane = pf_lane(), warp = pf_warp(), reg = warp * a.G * P::PLANE;
      if (warp >= nf || (pass >= 2 && a.last_only && !(end && warp == nf - 1))) continue;
      const int pc = lane / P::WF, kw = lane - pc * P::WF, pr = lane / P::HH, j = lane - pr * P::HH;
      const bool rows = pass == 0 || pass == 3, two = j + P::HH < N;
      if (rows ? pr < n : pc < n) {
        float* at = pf_smem + (rows ? reg + pr * P::PLANE + j * P::PITCH : reg + pc * P::PLANE + 2 * kw);
        cf z[N];
        if (pass == 0) P::load_rows(at, two, z);
        else if (pass == 3) P::get_rows(at, two, z);
        else P::load_col(at, z);
        lane_dft<N>(z);
        if (pass == 0) P::put_rows(at, two, z);
        else if (pass == 3) P::store_rows(at, two, z);
        else P::store_col(at, z);
      }
      __syncwarp();
      if (pass == 3) {
        const size_t frame = (size_t)b * a.T + t0 + warp;
        float* xp = a.xz + (frame * 2 * a.C + c0) * (N * N);
        if (a.mode == 0) {
          const size_t zf = a.equal > 0 ? (size_t)b * a.T : frame;
          P::template store<true>(pf_smem + reg, xp, a.xz + (zf * 2 * a.C + a.C + c0) * (N * N), n);
        } else {
          P::template store<false>(pf_smem + reg, xp, nullptr, n);
        }
      }
    }
  }
}

// Registers and shared memory of a kernel decide F and G together with what the waves look like: a batch of frames costs a warp
// 3.7 clocks an instruction by itself and 0.17 more for every warp on its SM (two points of 16 x 8 x 56 x 56 x 32: 3.5 warps an SM
// 150 us, ten 90), half of it whatever the number of planes.  On 63 shapes of nine sides F as chosen is within 2 % of the best of 1, 2
// and 4 but for two (6 %), always 1, 2 or 4 are 1.27, 1.07 (T > 1) and 1.01 times as slow in the mean.  Three where it saves a tenth
// by this count, as where four leave an SM short of a CTA: 16 x 8 x 56 x 56 x 32 243 -> 238 us, 54 x 3 x 16 x 16 x 48 52 -> 48; with a
// smaller margin one shape in seven of 139 loses 2 to 6 %.
template <int N>
static int gated_fft_n(GatedFftArgs& a, cudaStream_t st) {
  typedef Pf<N> P;
  const int warps = gated_fft_warps(N), sms = sm_count();
  const size_t state = a.T > 1 ? (size_t)N * 32 * 8 : 0;
  double best = 1e30;
  int F = 1, ctas = 1, G = 1;
  for (int g = a.C < P::GMAX ? a.C : P::GMAX; g >= 1; g = g > 1 ? (g + 1) / 2 : 0) {
    const long long groups = (long long)a.B * ((a.C + g - 1) / g);
    for (int f : {1, 2, 4, 3}) {
      if (f > 1 && f / 2 >= a.T) continue;
      const size_t smem = (size_t)f * g * P::PLANE * 4 + state;
      int c = (int)(227 * 1024 / (smem + 1024));
      if (c * f > warps) c = warps / f;
      if (c < 1) continue;
      const long long slots = (long long)sms * c, full = groups / slots, rest = (groups % slots + sms - 1) / sms;
      const double one = (a.T + f - 1) / f * (0.5 + 0.5 * g / P::GMAX);
      const double cost = one * (full * (3.7 + 0.17 * c * f) + (rest > 0 ? 3.7 + 0.17 * rest * f : 0));
      if (cost < best * (f == 3 ? 0.9 : 0.98)) { best = cost; F = f; ctas = c; G = g; }
    }
  }
  const int n = (a.C + G - 1) / G;
  a.G = (a.C + n - 1) / n;
  a.cgroups = (a.C + a.G - 1) / a.G;
  a.groups = a.B * a.cgroups;
  const int slots = sms * ctas, grid = a.groups < slots ? a.groups : slots;
  const PdlOff alone(uneven_rounds(a.groups, ctas));
  const size_t smem = spread_smem((size_t)F * a.G * P::PLANE * 4 + state, grid);
  auto kern = F == 1 ? gated_spectral_fft<N, 1> : F == 2 ? gated_spectral_fft<N, 2> : F == 3 ? gated_spectral_fft<N, 3> : gated_spectral_fft<N, 4>;
  const cudaError_t e = func_smem(kern, smem);
  if (e != cudaSuccess) { set_cuda_error(e); return CSSM_ERR_CUDA; }
  launch_k(kern, grid, 32 * F, smem, st, a);
  return check_launch();
}

// Which calls the kernel takes: square planes of its sides.  A single frame leaves a warp's chain of four FFTs alone on its scheduler
// unless there are more planes than SMs, and the loads of odd rows are 4 bytes each: 1 x 1 x 56 x 56 x 32 37.6 us (folded DFT 33.4),
// 59 x 1 x 23 x 23 x 32 46.2 (41.8), but 78 x 1 x 20 x 20 x 32 41.9 (46.2), 637 x 1 x 7 x 7 x 32 42.1 (51.5).  From two frames on it is ahead everywhere
// (16 x 2 x 16 x 16 x 16 28.7, 30.8; 2 x 5 x 39 x 39 x 48 60.1, 60.2).
bool gated_spectral_fft_takes(int B, int T, int H, int W, int C) {
  if (H != W) return false;
  if (T == 1 && ((H % 2 != 0 && H > 9) || (long long)B * C * (H / 2 + 1) < 32LL * sm_count())) return false;
#define X(n) case n:
  switch (H) { PF_SIDES(X) return true; }
#undef X
  return false;
}

int launch_gated_spectral_fft(int B, int T, int H, int C, const cf* khat, const float* gates, float* xz, int last_only, int mode,
                              cudaStream_t st, const float* dchan, int equal_steps) {
  GatedFftArgs a;
  memset(&a, 0, sizeof(a));
  a.xz = xz; a.khat = khat; a.gates = reinterpret_cast<const float4*>(gates); a.dchan = dchan;
  a.B = B; a.T = T; a.C = C; a.last_only = last_only; a.mode = mode; a.equal = equal_steps;
#define X(n) case n: return gated_fft_n<n>(a, st);
  switch (H) { PF_SIDES(X) }
#undef X
  return CSSM_ERR_UNSUPPORTED;
}

}  // namespace cssm
