// Plane transforms in a lane's registers (csrc/lane_fft.cuh) for one warp working on several N x N planes side by side.
//
// The planes lie one behind the other in the warp's region of shared memory, rows PITCH floats apart (an odd number of 16 bytes, so
// that the 16-byte accesses of lanes in consecutive rows meet different banks), and each pass goes over them in place:
//   rows      lane = (plane, j) packs the real rows j and j + ceil(N / 2) into one FFT, separates them in its registers and leaves the
//             N / 2 + 1 entries of each half spectrum in the row's place; back, it does the reverse;
//   columns   lane = (plane, kw).
// Forward spectra are twice the transform (the halves of the separation are left out).  There is one copy of the FFT for all passes:
// the inverse transform is the forward one with real and imaginary parts exchanged, so whoever writes a spectrum to be
// transformed back writes (Im, Re).
#pragma once
#include "lane_fft.cuh"

namespace cssm {

// The lane's and the warp's number, opaque: what follows from it is made where it is needed (hoisted out of the loop over steps it lay in registers
// beside the FFTs, and spilled).
__device__ __forceinline__ int pf_lane() {
  int l;
  asm volatile("mov.u32 %0, %%laneid;" : "=r"(l));
  return l;
}
__device__ __forceinline__ int pf_warp() {
  int t = threadIdx.x;
  asm volatile("" : "+r"(t));
  return t >> 5;
}

template <int N> struct Pf {
  static constexpr int WF = N / 2 + 1, HH = (N + 1) / 2;        // columns; row pairs
  static constexpr int GMAX = 32 / WF;                          // planes a warp
  static constexpr int PITCH = ((2 * WF + 3) / 4 | 1) * 4;      // floats
  static constexpr int PLANE = N * PITCH;
  static constexpr int V = N % 4 == 0 ? 4 : N % 2 == 0 ? 2 : 1; // floats an access of global memory
  static constexpr int NB = N * WF;

  static __device__ __forceinline__ void load_rows(const float* ra, bool two, cf (&z)[N]) {
    const float* rb = ra + HH * PITCH;
#pragma unroll
    for (int c = 0; c < N / 4; ++c) {
      const float4 u = reinterpret_cast<const float4*>(ra)[c];
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (N % 2 == 0 || two) v = reinterpret_cast<const float4*>(rb)[c];
      z[4 * c] = mk(u.x, v.x); z[4 * c + 1] = mk(u.y, v.y); z[4 * c + 2] = mk(u.z, v.z); z[4 * c + 3] = mk(u.w, v.w);
    }
#pragma unroll
    for (int c = N / 4 * 4; c < N; ++c) z[c] = mk(ra[c], N % 2 == 0 || two ? rb[c] : 0.f);
  }
  // rows from (.y, .x) of z
  static __device__ __forceinline__ void store_rows(float* ra, bool two, const cf (&z)[N]) {
    float* rb = ra + HH * PITCH;
#pragma unroll
    for (int c = 0; c < N / 4; ++c) {
      reinterpret_cast<float4*>(ra)[c] = make_float4(z[4 * c].y, z[4 * c + 1].y, z[4 * c + 2].y, z[4 * c + 3].y);
      if (N % 2 == 0 || two) reinterpret_cast<float4*>(rb)[c] = make_float4(z[4 * c].x, z[4 * c + 1].x, z[4 * c + 2].x, z[4 * c + 3].x);
    }
#pragma unroll
    for (int c = N / 4 * 4; c < N; ++c) {
      ra[c] = z[c].y;
      if (N % 2 == 0 || two) rb[c] = z[c].x;
    }
  }
  static __device__ __forceinline__ void put_rows(float* ra, bool two, const cf (&z)[N]) {
    float* rb = ra + HH * PITCH;
#pragma unroll
    for (int k = 0; k < WF; k += 2) {
      const cf u = z[k], v = z[(N - k) % N];
      float4 a = make_float4(u.x + v.x, u.y - v.y, 0.f, 0.f), b = make_float4(u.y + v.y, v.x - u.x, 0.f, 0.f);
      if (k + 1 < WF) {
        const cf s = z[k + 1], t = z[N - k - 1];
        a.z = s.x + t.x; a.w = s.y - t.y; b.z = s.y + t.y; b.w = t.x - s.x;
      }
      *reinterpret_cast<float4*>(ra + 2 * k) = a;
      if (N % 2 == 0 || two) *reinterpret_cast<float4*>(rb + 2 * k) = b;
    }
  }
  static __device__ __forceinline__ void get_rows(const float* ra, bool two, cf (&z)[N]) {
    const float* rb = ra + HH * PITCH;
#pragma unroll
    for (int k = 0; k < WF; k += 2) {
      const float4 a = *reinterpret_cast<const float4*>(ra + 2 * k);
      float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
      if (N % 2 == 0 || two) b = *reinterpret_cast<const float4*>(rb + 2 * k);
      // Z[k] = A[k] + i B[k], Z[N - k] = conj A[k] + i conj B[k], exchanged; columns 0 and N / 2: real parts only
      if (k == 0 || 2 * k == N) z[k] = mk(b.y, a.y);
      else { z[k] = mk(a.x + b.y, a.y - b.x); z[N - k] = mk(b.y - a.x, a.y + b.x); }
      if (k + 1 < WF) {
        if (2 * (k + 1) == N) z[k + 1] = mk(b.w, a.w);
        else { z[k + 1] = mk(a.z + b.w, a.w - b.z); z[N - k - 1] = mk(b.w - a.z, a.w + b.z); }
      }
    }
  }
  static __device__ __forceinline__ void load_col(const float* col, cf (&z)[N]) {
#pragma unroll
    for (int h = 0; h < N; ++h) {
      const float2 v = *reinterpret_cast<const float2*>(col + h * PITCH);
      z[h] = mk(v.x, v.y);
    }
  }
  static __device__ __forceinline__ void store_col(float* col, const cf (&z)[N]) {
#pragma unroll
    for (int h = 0; h < N; ++h) *reinterpret_cast<float2*>(col + h * PITCH) = make_float2(z[h].x, z[h].y);
  }

  // Accesses of V floats of the planes, dealt out to the lanes: access i = lane + 32 u is at floats V i of the planes and `off` of the region.
  struct Walk {
    static constexpr int R = N / V;
    int i, col, off;
    __device__ __forceinline__ Walk() {
      i = pf_lane();
      const int row = i / R;
      col = i - row * R;
      off = row * PITCH + col * V;
    }
    __device__ __forceinline__ void next() {
      i += 32;
      off += 32 / R * PITCH + 32 % R * V;
      if (32 % R != 0) {
        col += 32 % R;
        if (col >= R) { col -= R; off += PITCH - N; }
      }
    }
  };
  // n planes from global memory, asynchronously
  static __device__ __forceinline__ void load(const float* __restrict__ src, float* region, int n) {
    const int total = n * N * (N / V);
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(region);
    Walk w;
    const float* s = src + w.i * V;
#pragma unroll 4
    for (; w.i < total; w.next(), s += 32 * V) {
      const uint32_t dst = base + 4 * w.off;
      if constexpr (V == 4) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(s) : "memory");
      else asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst), "l"(s), "n"(V * 4) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  static __device__ __forceinline__ void wait() {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
  }
  struct __align__(V * 4) Vec { float f[V]; };
  // n planes to global memory, times the planes z where MUL
  template <bool MUL>
  static __device__ __forceinline__ void store(const float* region, float* __restrict__ dst, const float* __restrict__ z, int n) {
    const int total = n * N * (N / V);
    constexpr int U = 8;
    Walk w;
    Vec* d = reinterpret_cast<Vec*>(dst) + w.i;
    const Vec* zp = reinterpret_cast<const Vec*>(z) + w.i;
    float zv[U][V];
    auto fetch = [&](int u, int at) {                          // (never skipped: a skipped load would keep its registers live through the whole step)
      const Vec* p = zp + (at < total ? 32 * u : total - 1 - at + 32 * u);
      if constexpr (V == 4) { const float4 t = __ldg(reinterpret_cast<const float4*>(p)); zv[u][0] = t.x; zv[u][1] = t.y; zv[u][2] = t.z; zv[u][3] = t.w; }
      else if constexpr (V == 2) { const float2 t = __ldg(reinterpret_cast<const float2*>(p)); zv[u][0] = t.x; zv[u][1] = t.y; }
      else zv[u][0] = __ldg(reinterpret_cast<const float*>(p));
    };
    if (MUL) {
#pragma unroll
      for (int u = 0; u < U; ++u) fetch(u, w.i + 32 * u);
    }
#pragma unroll 1
    while (w.i < total) {
      zp += 32 * U;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (w.i < total) {
          Vec o = *reinterpret_cast<const Vec*>(region + w.off);
          if (MUL) {
#pragma unroll
            for (int e = 0; e < V; ++e) o.f[e] *= zv[u][e];
            fetch(u, w.i + 32 * U);
          }
          d[32 * u] = o;
        }
        w.next();
      }
      d += 32 * U;
    }
    __syncwarp();
  }
};

// The sides that are built: at most 32 columns (N / 2 + 1), and no prime factor from 29 on, whose direct transforms are long.
#define PF_SIDES(X) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12) X(13) X(14) X(15) X(16) X(17) X(18) X(19) X(20) X(21) X(22) X(23) X(24) \
  X(25) X(26) X(27) X(28) X(30) X(33) X(34) X(35) X(36) X(38) X(39) X(40) X(42) X(44) X(45) X(48) X(49) X(50) X(52) X(54) X(55) X(56) X(60)

}  // namespace cssm
