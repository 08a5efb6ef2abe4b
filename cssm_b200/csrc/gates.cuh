// Building blocks of the gate-map kernels: the context of a few frames, the two vectors of a factored
// gate, and dense gates of several frames at once.  All of them are chains of cold loads of weights, so
// every thread keeps 8 to 24 loads in flight and the long sums are cut over the threads of the CTA.
#pragma once
#include "common.cuh"

namespace cssm {

// sum over c in [c0, c1) of ctx[c] * w[c * ld], 16 loads in flight; ctx is 16-byte aligned.  Whole blocks of
// 16 run without predicates and with 16-byte reads of ctx: with one warp or two per scheduler the kernels
// here are bound by the length of a thread's own instruction stream.
__device__ __forceinline__ float gate_dot(const float* __restrict__ ctx, const float* __restrict__ w, int ld, int c0, int c1) {
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  int c = c0;
  if ((c0 & 3) == 0) {
    const float* p = w + (size_t)c0 * ld;
    for (; c + 16 <= c1; c += 16) {
      float v[16];
#pragma unroll
      for (int u = 0; u < 16; ++u) { v[u] = __ldg(p); p += ld; }
#pragma unroll
      for (int u = 0; u < 16; u += 4) {
        const float4 x = *reinterpret_cast<const float4*>(ctx + c + u);
        acc[0] = fmaf(x.x, v[u], acc[0]); acc[1] = fmaf(x.y, v[u + 1], acc[1]);
        acc[2] = fmaf(x.z, v[u + 2], acc[2]); acc[3] = fmaf(x.w, v[u + 3], acc[3]);
      }
    }
  }
  for (; c < c1; c += 16) {
    float v[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) v[u] = c + u < c1 ? __ldg(w + (size_t)(c + u) * ld) : 0.f;
#pragma unroll
    for (int u = 0; u < 16; ++u) acc[u & 3] = fmaf(c + u < c1 ? ctx[c + u] : 0.f, v[u], acc[u & 3]);
  }
  return (acc[0] + acc[1]) + (acc[2] + acc[3]);
}

// ctx[f][c] = mean over the plane of frames f0 .. f0+nf-1 (+ temporal code): from the per-frame sums
// (`sums`, (BT, C)) or from row sums (`part`, (BT, H, C)).  scratch: blockDim.x floats.  Ends with a barrier.
struct GateCtxSrc {
  const float* sums; const float* part; const float* tcode;      // tcode (T, C) or null
  int T, C, H, per_clip;                                         // per_clip: part holds one frame per clip
  float inv;
};
__device__ __forceinline__ void gate_ctx(const GateCtxSrc& s, int f0, int nf, float* ctx, float* scratch) {
  const int n = nf * s.C, nt = blockDim.x, tid = threadIdx.x;
  const int S = (s.sums != nullptr || n >= nt) ? 1 : nt / n;     // slices of the rows
  for (int i0 = 0; i0 < n; i0 += nt) {
    const int sl = tid / n, i = i0 + (S == 1 ? tid : tid - sl * n);
    float v = 0.f;
    if (i < n && (S == 1 || sl < S)) {
      const int f = i / s.C, c = i - f * s.C, fr = f0 + f;
      if (s.sums != nullptr) v = __ldg(s.sums + (size_t)fr * s.C + c);
      else {
        const float* p = s.part + (size_t)(s.per_clip ? fr / s.T : fr) * s.H * s.C + c;
        const int h0 = S == 1 ? 0 : sl * s.H / S, h1 = S == 1 ? s.H : (sl + 1) * s.H / S;
        for (int h = h0; h < h1; h += 8) {
          float t[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) t[u] = h + u < h1 ? __ldg(p + (size_t)(h + u) * s.C) : 0.f;
#pragma unroll
          for (int u = 0; u < 8; ++u) v += t[u];
        }
      }
    }
    if (S > 1) {
      scratch[tid] = v;
      __syncthreads();
      if (tid < n)
        for (int k = 1; k < S; ++k) v += scratch[k * n + tid];
    }
    if (i < n && (S == 1 || sl == 0)) {
      const int f = i / s.C, c = i - f * s.C;
      v *= s.inv;
      if (s.tcode != nullptr) v += __ldg(s.tcode + (size_t)((f0 + f) % s.T) * s.C + c);
      ctx[i] = v;
    }
  }
  __syncthreads();
}

// vec[o] = bias + ctx . column of every factored-gate vector of one frame: segment q has ncol(q) columns of
// gk[q] (C, ncol).  off[q] .. off[q+1] are its entries; scratch: blockDim.x floats.  Ends with a barrier.
template <int NSEG>
__device__ __forceinline__ void gate_vectors(const float* const (&gk)[NSEG], const float* const (&gb)[NSEG],
                                             const int (&off)[NSEG + 1], int nseg, const float* ctx, int C, float* vec,
                                             float* scratch) {
  const int total = off[nseg], nt = blockDim.x, tid = threadIdx.x;
  int S = total >= nt ? 1 : nt / total;
  if (S > 8) S = 8;
  for (int o0 = 0; o0 < total; o0 += nt) {
    const int sl = S == 1 ? 0 : tid / total, o = S == 1 ? o0 + tid : tid - sl * total;
    float v = 0.f;
    if (o < total && sl < S) {
      int q = 0;
#pragma unroll
      for (int k = 1; k < NSEG; ++k) if (k < nseg && o >= off[k]) q = k;
      const float* w = gk[0];
      const float* bp = gb[0];
      int col = o, ncol = off[1];
#pragma unroll
      for (int k = 1; k < NSEG; ++k)
        if (k == q) { w = gk[k]; bp = gb[k]; col = o - off[k]; ncol = off[k + 1] - off[k]; }
      v = gate_dot(ctx, w + col, ncol, sl * C / S, (sl + 1) * C / S) + (sl == 0 ? __ldg(bp + col) : 0.f);
    }
    if (S > 1) {
      scratch[tid] = v;
      __syncthreads();
      if (tid < total)
        for (int k = 1; k < S; ++k) v += scratch[k * total + tid];
    }
    if (sl == 0 && o < total) vec[o] = v;
  }
  __syncthreads();
}

// r[gate][frame] = bias + ctx[frame] . column `col` of the NG dense gates (C, ncol) for G frames (C % 4 == 0)
template <int NG, int G>
__device__ __forceinline__ void gate_dense(const float* const* gk, const float* const* gb, int ncol, int col, int C,
                                           const float* ctx, float (&r)[NG][G]) {
  constexpr int UN = NG <= 3 ? 8 : 4;
#pragma unroll
  for (int q = 0; q < NG; ++q) {
    const float b = __ldg(gb[q] + col);
#pragma unroll
    for (int f = 0; f < G; ++f) r[q][f] = b;
  }
  for (int c = 0; c < C; c += UN) {
    float w[NG][UN];
#pragma unroll
    for (int q = 0; q < NG; ++q)
#pragma unroll
      for (int u = 0; u < UN; ++u) w[q][u] = (UN == 4 || c + u < C) ? __ldg(gk[q] + (size_t)(c + u) * ncol + col) : 0.f;
#pragma unroll
    for (int f = 0; f < G; ++f)
#pragma unroll
      for (int u = 0; u < UN; u += 4) {
        if (UN > 4 && c + u >= C) continue;
        const float4 x = *reinterpret_cast<const float4*>(ctx + f * C + c + u);
#pragma unroll
        for (int q = 0; q < NG; ++q) {
          r[q][f] = fmaf(x.x, w[q][u], r[q][f]);     r[q][f] = fmaf(x.y, w[q][u + 1], r[q][f]);
          r[q][f] = fmaf(x.z, w[q][u + 2], r[q][f]); r[q][f] = fmaf(x.w, w[q][u + 3], r[q][f]);
        }
      }
  }
}

// Frames per CTA of a dense-gate launch with `chunks` CTAs per frame group: a weight read serves that many
// frames, as long as the SMs stay covered and two CTAs fit an SM with their contexts.
inline int gate_dense_frames(int BT, int chunks, int C) {
  for (int G : {8, 4})
    if ((long long)(BT / G) * chunks >= sm_count() && (size_t)(G * C + 128) * sizeof(float) <= 100 * 1024) return G;
  return 1;
}
// CTAs per frame of a factored-gate launch (512 threads, and each makes all vectors of its frame): enough for every SM,
// at most one per 256 bins
inline int gate_chunks(int BT, int NB) {
  const int want = sm_count();
  int chunks = 1;
  if (BT < want) {
    chunks = (want + BT - 1) / BT;
    const int maxc = (NB + 255) / 256;
    if (chunks > maxc) chunks = maxc;
  }
  return chunks;
}

// Launch of a gate-map kernel: its contexts and vectors may need more than the 48 KB a launch has by default
// (wide blocks, long planes).
template <class... P, class... A>
inline int launch_gates(void (*kern)(P...), dim3 grid, int threads, size_t smem, cudaStream_t st, A... args) {
  if (smem > 48 * 1024) {
    const cudaError_t e = func_smem(kern, smem);
    if (e != cudaSuccess) { set_cuda_error(e); return CSSM_ERR_CUDA; }
  }
  launch_k(kern, grid, dim3(threads), smem, st, args...);
  return check_launch();
}

}  // namespace cssm
