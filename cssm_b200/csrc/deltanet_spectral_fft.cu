// DeltaNet on square planes with whole FFTs in a lane's registers (csrc/delta_spectral_fft.cuh)
#define CSSM_F32X2 0
#include "delta_spectral_fft.cuh"

namespace cssm {

struct DnFftRule {
  typedef DnSpectralArgs Args;
  static constexpr bool SCALE_KEYS = true;
  static __device__ __forceinline__ float* planes(const Args& a) { return a.qkv; }
  // B_k scales the key spectra (gate maps)
  template <int N> static __device__ __forceinline__ void scale_keys(const Args& a, size_t frame, int kw, cf (&z)[N]) {
    if (a.chan != nullptr) return;
    const float4* gm = a.abkv + frame * Pf<N>::NB + kw;
#pragma unroll
    for (int h = 0; h < N; ++h) {
      const float s = __ldg(&gm[h * Pf<N>::WF].z);
      z[h] = mk(s * z[h].x, s * z[h].y);
    }
  }
  template <int N>
  static __device__ __forceinline__ void bins(const Args& a, const DeltaFftArgs&, int b, int t, int h0, int nh, const float* nrm, float4* state4, bool) {
    typedef Pf<N> P;
    constexpr int NB = P::NB;
    const int total = nh * NB;
    const size_t frame = (size_t)b * a.T + t;
    const float4* gm = a.abkv + frame * NB;
    const float* cg = a.cg + frame * NB;
    const bool chan = a.chan != nullptr, first = t == 0, last = t + 1 == a.T;
    const float floor_mag = a.goom_floor ? 1e-7f : 0.f;
    float2* state = reinterpret_cast<float2*>(state4);
    float4 gt;
    float2 w;
    float c;
    auto fetch = [&](int i) {                                 // (never skipped: see csrc/gated_spectral_fft.cu)
      const int ic = min(i, total - 1), cl = ic / NB, r = ic - cl * NB;
      w = __ldg(reinterpret_cast<const float2*>(a.what) + (size_t)(h0 + cl) * NB + r);
      if (chan) {
        const float2 ab = __ldg(a.chan + frame * a.C + h0 + cl);
        gt = make_float4(ab.x, ab.y, 1.f, 1.f);
        c = 1.0f / (N * N);
      } else {
        gt = __ldg(gm + r);
        c = __ldg(cg + r);
      }
    };
    fetch(threadIdx.x);
#pragma unroll 1
    for (int i = threadIdx.x; i < total; i += blockDim.x) {
      const int cl = i / NB, r = i - cl * NB, hh = r / P::WF, pos = hh * P::PITCH + 2 * (r - hh * P::WF);
      const float* sp = pf_smem + cl * P::PLANE + pos;
      const float2 q = *reinterpret_cast<const float2*>(sp), k = *reinterpret_cast<const float2*>(sp + nh * P::PLANE),
                   v = *reinterpret_cast<const float2*>(sp + 2 * nh * P::PLANE);
      const float nq = nrm[cl], nk = nrm[nh + cl];
      const float2 s = first ? make_float2(0.f, 0.f) : state[i];
      const cf kv = mk(k.x * nk, k.y * nk), qv = mk(q.x * nq, q.y * nq);
      const float gv = 0.5f * gt.w;                            // (spectra are doubled; nrm holds the halves of k and q)
      const cf vv = mk(v.x * gv, v.y * gv);
      const float kp = kv.x * kv.x + kv.y * kv.y, sc = gt.x * (1.0f - gt.y * kp), beta = gt.y, cs = c;
      cf A = mk(w.x * sc, w.y * sc);
      fetch(i + blockDim.x);
      const float am = sqrtf(A.x * A.x + A.y * A.y), sq = a.rho / (1.0f + am);
      A = mk(A.x * sq, A.y * sq);
      if (am * sq < floor_mag) A = mk(floor_mag, 0.f);
      cf U = cmulc(vv, kv);                                    // v * conj(k)
      U = mk(U.x * beta, U.y * beta);
      if (U.x * U.x + U.y * U.y < floor_mag * floor_mag) U = mk(floor_mag, 0.f);
      cf h = cmul(A, mk(s.x, s.y));
      h.x += U.x; h.y += U.y;
      const cf o = cmul(h, qv);
      if (!last) state[i] = make_float2(h.x, h.y);
      *reinterpret_cast<float2*>(pf_smem + (2 * nh + cl) * P::PLANE + pos) = make_float2(o.y * cs, o.x * cs);
    }
  }
};

int launch_deltanet_spectral_fft(const DnSpectralArgs& a, cudaStream_t st) {
#define X(n) case n: return delta_fft_launch<n, 1, DnFftRule>(a, a.B, a.T, a.C, 0, 1, true, st);
  switch (a.H) { PF_SIDES(X) }
#undef X
  return CSSM_ERR_UNSUPPORTED;
}

}  // namespace cssm
