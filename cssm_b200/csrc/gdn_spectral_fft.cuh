// GDN's rule for csrc/delta_spectral_fft.cuh; one source file for each key dimension.
#pragma once
#include "delta_spectral_fft.cuh"

namespace cssm {

template <int DK> struct GdnFftRule {
  typedef GdnSpectralArgs Args;
  static constexpr bool SCALE_KEYS = false;
  static __device__ __forceinline__ float* planes(const Args& a) { return a.qkv; }
  template <int N> static __device__ __forceinline__ void scale_keys(const Args&, size_t, int, cf (&)[N]) {}

  template <int N>
  static __device__ __forceinline__ void bins(const Args& a, const DeltaFftArgs& d, int b, int t, int h0, int nh, const float* nrm, float4* state, bool emit) {
    typedef Pf<N> P;
    constexpr int NB = P::NB;
    const int n = nh * DK, total = nh * NB;
    const float2* abf = a.ab + ((size_t)b * a.T + t) * a.ab_heads * NB;
    const bool first = t == 0, last = t + 1 == a.T;
    const float inv = 1.0f / (N * N);
    auto where = [&](int i, int& hl, int& r, int& pos) {
      hl = i / NB;
      r = i - hl * NB;
      const int h = r / P::WF;
      pos = h * P::PITCH + 2 * (r - h * P::WF);
    };
    float2 gab, gw;
    auto fetch = [&](int i) {                                 // (never skipped: see csrc/gated_spectral_fft.cu)
      const int ic = min(i, total - 1), hl = ic / NB, r = ic - hl * NB;
      gab = __ldg(abf + (a.ab_heads > 1 ? (size_t)(h0 + hl) * NB : 0) + r);
      gw = __ldg(reinterpret_cast<const float2*>(a.what) + (size_t)(h0 + hl) * NB + r);
    };
    fetch(threadIdx.x);
#pragma unroll 1
    for (int i = threadIdx.x; i < total; i += blockDim.x) {
      int hl, r, pos;
      where(i, hl, r, pos);
      const float* sp = pf_smem + (hl * DK) * P::PLANE + pos;
      cf kk[DK], qq[DK], vv[DK];
      float ks = 0.f;
#pragma unroll
      for (int j = 0; j < DK; ++j) {
        const float2 k = *reinterpret_cast<const float2*>(sp + (n + j) * P::PLANE), v = *reinterpret_cast<const float2*>(sp + (2 * n + j) * P::PLANE);
        const float s = nrm[n + hl * DK + j];
        kk[j] = mk(k.x * s, k.y * s);
        ks += kk[j].x * kk[j].x + kk[j].y * kk[j].y;
        vv[j] = mk(0.5f * v.x, 0.5f * v.y);                   // (spectra are doubled; nrm holds the halves of k and q)
        qq[j] = mk(0.f, 0.f);
        if (emit) {
          const float2 q = *reinterpret_cast<const float2*>(sp + j * P::PLANE);
          const float u = nrm[hl * DK + j];
          qq[j] = mk(q.x * u, q.y * u);
        }
      }
      const float kn = rsqrtf(ks + 1e-6f);
#pragma unroll
      for (int j = 0; j < DK; ++j) kk[j] = mk(kk[j].x * kn, kk[j].y * kn);
      const cf aw = mk(gab.x * gw.x, gab.x * gw.y);
      const float beta = gab.y;
      fetch(i + blockDim.x);
      float4* ss = state + (size_t)hl * DK * (DK / 2) * NB + r;
      float2* gs = reinterpret_cast<float2*>(a.state) + ((size_t)(b * (a.C / DK) + h0 + hl) * DK * DK) * NB + r;
      cf S[DK][DK];
#pragma unroll
      for (int v = 0; v < DK; ++v)
#pragma unroll
        for (int j = 0; j < DK; j += 2) {
          float4 w = make_float4(0.f, 0.f, 0.f, 0.f);
          if (!first) {
            if (d.smem_state) w = ss[(v * (DK / 2) + j / 2) * NB];
            else { const float2 x = gs[(v * DK + j) * NB], y = gs[(v * DK + j + 1) * NB]; w = make_float4(x.x, x.y, y.x, y.y); }
          }
          S[v][j] = mk(w.x, w.y); S[v][j + 1] = mk(w.z, w.w);
        }
#pragma unroll
      for (int v = 0; v < DK; ++v) {
        const cf o = gdn_bin_update_regs<DK, true>(S[v], kk, qq, vv[v], aw, beta);
        if (!last) {
#pragma unroll
          for (int j = 0; j < DK; j += 2) {
            if (d.smem_state) ss[(v * (DK / 2) + j / 2) * NB] = make_float4(S[v][j].x, S[v][j].y, S[v][j + 1].x, S[v][j + 1].y);
            else { gs[(v * DK + j) * NB] = make_float2(S[v][j].x, S[v][j].y); gs[(v * DK + j + 1) * NB] = make_float2(S[v][j + 1].x, S[v][j + 1].y); }
          }
        }
        if (emit) *reinterpret_cast<float2*>(pf_smem + (2 * n + hl * DK + v) * P::PLANE + pos) = make_float2(o.y * inv, o.x * inv);
      }
    }
  }
};

template <int DK>
inline int launch_gdn_fft_dk(const GdnSpectralArgs& a, cudaStream_t st) {
#define X(n) case n: return delta_fft_launch<n, DK, GdnFftRule<DK>>(a, a.B, a.T, a.C, a.last_only, a.use_l2, false, st);
  switch (a.H) { PF_SIDES(X) }
#undef X
  return CSSM_ERR_UNSUPPORTED;
}

}  // namespace cssm
