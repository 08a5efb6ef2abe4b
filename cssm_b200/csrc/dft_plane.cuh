// Plane transforms of any size as products with folded DFT matrices, for one CTA working on P planes
// side by side.
//
// A length-N DFT with real twiddle symmetry needs half of its terms: with s_n = x_n + x_{N-n} and
// d_n = x_n - x_{N-n} (n = 0 .. N/2; a self-paired n has s = x, d = 0)
//   X_k = sum_n s_n cos(2 pi n k / N) - i sum_n d_n sin(2 pi n k / N),   X_{N-k}: the sine term negated.
// Every one of the four passes of a plane (rows, columns, inverse columns, inverse rows) is then the
// same small matrix product
//   acc[x][y] += (op[n][x].xy * tw[n][y], op[n][x].zw * tw[n][y])     (elementwise, packed f32x2)
// with tw[n][y] = (cos, -sin)(2 pi n y / N), n and y = 0 .. N/2, and op two packed pairs per entry:
//   pass          x             y            n            op[n][x]
//   rows          row pair      column k     pixel pair   (s, d) of row p | (s, d) of row H-p
//   columns       column        row freq     row pair     (a.re, -b.im) | (a.im, b.re)    a, b = Y_p +- Y_{H-p}
//   inv. columns  column        row pair     row freq     (A.re, B.im) | (A.im, -B.re)    A, B = G_k +- G_{H-k}
//   inv. rows     row pair      pixel pair   column k     f (Re, Im) of row p | of row H-p, f = 1 or 2
// and what a thread finishes is already folded for the next pass, because its cell holds both members
// of a pair.  The products run from shared memory in register tiles of RT x YT cells; ldx is odd so that
// both the reads (consecutive lanes = consecutive x) and the transposed writes are free of bank conflicts.
#pragma once
#include "common.cuh"

namespace cssm {

// A CTA has NT = 256 threads (two per SM) or 128 (four).  (NT from blockDim instead: 10 % slower.)

typedef unsigned long long dp_u64;

__device__ __forceinline__ dp_u64 dp_fma2(dp_u64 a, dp_u64 b, dp_u64 c) {
  dp_u64 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ float2 dp_unpack(dp_u64 v) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
  return f;
}

// tw[n][y], n, y = 0 .. N/2, row stride ld >= N/2 + 1 (a multiple of 4; the rest is zero)
template <int NT>
__device__ inline void dp_fill_table(float2* tw, int N, int ld) {
  const int M = N / 2 + 1;
  for (int i = threadIdx.x; i < M * ld; i += NT) {
    const int n = i / ld, y = i - n * ld;
    float2 v = make_float2(0.f, 0.f);
    if (y < M) sincospif(-2.0f * (float)((n * y) % N) / (float)N, &v.y, &v.x);
    tw[i] = v;
  }
}

// One pass: op [Nred][ldx] 16-byte entries, tw [Nred][ldy] pairs.  epi(x, y0, m, lo, hi) takes the first m of
// the YT cells (x, y0 ..) of a tile row at once, so that it can have their loads in flight together.
template <int RT, int YT, int NT, class Epi>
__device__ __forceinline__ void dp_pass(const ulonglong2* __restrict__ op, int ldx, const dp_u64* __restrict__ tw,
                                        int ldy, int Nred, int X, int Y, Epi&& epi) {
  const int nx = (X + RT - 1) / RT, ny = (Y + YT - 1) / YT;
  for (int tile = threadIdx.x; tile < nx * ny; tile += NT) {
    const int ty = tile / nx, tx = tile - ty * nx;
    dp_u64 lo[RT][YT], hi[RT][YT];
    const ulonglong2* po[RT];
#pragma unroll
    for (int j = 0; j < RT; ++j) {
      po[j] = op + min(tx + j * nx, X - 1);
#pragma unroll
      for (int e = 0; e < YT; ++e) lo[j][e] = hi[j][e] = 0ull;
    }
    const dp_u64* pt = tw + ty * YT;
#pragma unroll 2
    for (int n = 0; n < Nred; ++n) {
      dp_u64 t[YT];
      if constexpr (YT >= 2) {
#pragma unroll
        for (int e = 0; e < YT; e += 2) {
          const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(pt + e);
          t[e] = v.x; t[e + 1] = v.y;
        }
      } else {
        t[0] = *pt;
      }
      pt += ldy;
#pragma unroll
      for (int j = 0; j < RT; ++j) {
        const ulonglong2 o = *po[j];
        po[j] += ldx;
#pragma unroll
        for (int e = 0; e < YT; ++e) {
          lo[j][e] = dp_fma2(o.x, t[e], lo[j][e]);
          hi[j][e] = dp_fma2(o.y, t[e], hi[j][e]);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < RT; ++j) {
      const int x = tx + j * nx;
      if (x >= X) continue;
      float2 l[YT], h[YT];
#pragma unroll
      for (int e = 0; e < YT; ++e) { l[e] = dp_unpack(lo[j][e]); h[e] = dp_unpack(hi[j][e]); }
      epi(x, ty * YT, min(YT, Y - ty * YT), l, h);
    }
  }
}

// Sizes of a plane group; the divisions are by run-time constants of the launch.
struct DpGeom {
  int H, W, Hp, Wp, ldw, ldh;         // Hp = H/2 + 1 row pairs, Wp = W/2 + 1 = Wf; table strides
  FastDiv dHp, dWp, dW;
};
inline DpGeom dp_geom(int H, int W) {
  DpGeom g;
  g.H = H; g.W = W; g.Hp = H / 2 + 1; g.Wp = W / 2 + 1;
  g.ldw = (g.Wp + 3) / 4 * 4; g.ldh = (g.Hp + 3) / 4 * 4;
  g.dHp = FastDiv(g.Hp); g.dWp = FastDiv(g.Wp); g.dW = FastDiv(W);
  return g;
}
// entries of one operand region for P planes
__host__ __device__ inline int dp_ld_rows(const DpGeom& g, int P) { return (P * g.Hp) | 1; }
__host__ __device__ inline int dp_ld_cols(const DpGeom& g, int P) { return (P * g.Wp) | 1; }
inline size_t dp_region_bytes(const DpGeom& g, int P) {
  const size_t a = (size_t)g.Wp * dp_ld_rows(g, P), b = (size_t)g.Hp * dp_ld_cols(g, P);
  const size_t plane = ((size_t)P * g.H * (g.W | 1) * 4 + 15) / 16;       // the result planes pass through one
  size_t m = a > b ? a : b;
  m = m > plane ? m : plane;
  return m * 16;
}
// Both tables and four pairs more: a tile of eight cells may read that far past the last row (cells it throws away).
__host__ __device__ inline int dp_table_pairs(const DpGeom& g) { return g.Wp * g.ldw + g.Hp * g.ldh + 4; }
constexpr size_t DP_SMEM_LIMIT = 226 * 1024 + 32;        // (the four pairs refuse no plane that fitted without them)
inline size_t dp_table_bytes(const DpGeom& g) { return (size_t)dp_table_pairs(g) * 8; }

// P planes from global memory (consecutive, HW apart) -> folded row operand [pixel pair][row pair].
// Four entries (16 loads) in flight per thread.
template <int NT>
__device__ __forceinline__ void dp_load_fold(const DpGeom& g, const float* __restrict__ src, float4* S, int ldx, int P) {
  const int total = P * g.Hp * g.Wp;
  for (int i0 = threadIdx.x; i0 < total; i0 += 4 * NT) {
    float v[4][4];
    int dst[4];
    bool sn[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = min(i0 + u * NT, total - 1);
      const int x = g.dWp.div(i), n = i - x * g.Wp;
      const int pl = g.dHp.div(x), p = x - pl * g.Hp;
      const float* r0 = src + (pl * g.H + p) * g.W;
      const bool self_p = p == 0 || 2 * p == g.H;
      sn[u] = n == 0 || 2 * n == g.W;
      const int m = sn[u] ? n : g.W - n;
      const float* r1 = r0 + (g.H - 2 * p) * g.W;
      v[u][0] = r0[n]; v[u][1] = r0[m];
      v[u][2] = self_p ? 0.f : r1[n]; v[u][3] = self_p ? 0.f : r1[m];
      dst[u] = i0 + u * NT < total ? n * ldx + x : -1;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (dst[u] >= 0)
        S[dst[u]] = sn[u] ? make_float4(v[u][0], 0.f, v[u][2], 0.f)
                          : make_float4(v[u][0] + v[u][1], v[u][0] - v[u][1], v[u][2] + v[u][3], v[u][2] - v[u][3]);
  }
}

// rows: folded pixels -> folded column operand [row pair][plane * Wp + k]
template <int RT, int YT, int NT>
__device__ __forceinline__ void dp_rows(const DpGeom& g, const float4* S, int ldx, const float2* TW, float4* U, int ldc, int P) {
  dp_pass<RT, YT, NT>(reinterpret_cast<const ulonglong2*>(S), ldx, reinterpret_cast<const dp_u64*>(TW), g.ldw, g.Wp,
                  P * g.Hp, g.Wp, [&](int x, int k0, int m, const float2* y0, const float2* y1) {
    const int pl = g.dHp.div(x), p = x - pl * g.Hp;
    const bool self = p == 0 || 2 * p == g.H;
    float4* dst = U + p * ldc + pl * g.Wp + k0;
#pragma unroll
    for (int e = 0; e < YT; ++e)
      if (e < m)
        dst[e] = self ? make_float4(y0[e].x, 0.f, y0[e].y, 0.f)
                      : make_float4(y0[e].x + y1[e].x, y1[e].y - y0[e].y, y0[e].y + y1[e].y, y0[e].x - y1[e].x);
  });
}

// columns: epi(col, k0, m, F, G) with F[e] = F_{k0+e} and G[e] = F_{H-k0-e} of that column, k = 0 .. H/2
// (G is meaningless for a self-paired k)
template <int RT, int YT, int NT, class Epi>
__device__ __forceinline__ void dp_cols(const DpGeom& g, const float4* U, int ldc, const float2* TH, int P, Epi&& epi) {
  dp_pass<RT, YT, NT>(reinterpret_cast<const ulonglong2*>(U), ldc, reinterpret_cast<const dp_u64*>(TH), g.ldh, g.Hp,
                  P * g.Wp, g.Hp, [&](int x, int k0, int m, const float2* lo, const float2* hi) {
    cf f0[YT], f1[YT];
#pragma unroll
    for (int e = 0; e < YT; ++e) {
      f0[e] = mk(lo[e].x + lo[e].y, hi[e].x + hi[e].y);
      f1[e] = mk(lo[e].x - lo[e].y, hi[e].x - hi[e].y);
    }
    epi(x, k0, m, f0, f1);
  });
}

// spectrum pair (G_k, G_{H-k}) -> entry of the inverse column operand
__device__ __forceinline__ float4 dp_fold_spec(bool self, cf g0, cf g1) {
  if (self) return make_float4(g0.x, 0.f, g0.y, 0.f);
  return make_float4(g0.x + g1.x, g0.y - g1.y, g0.y + g1.y, g1.x - g0.x);
}

// inverse columns: [k][col] -> inverse row operand [column k][row pair]
template <int RT, int YT, int NT>
__device__ __forceinline__ void dp_inv_cols(const DpGeom& g, const float4* V, int ldc, const float2* TH, float4* R, int ldx, int P) {
  dp_pass<RT, YT, NT>(reinterpret_cast<const ulonglong2*>(V), ldc, reinterpret_cast<const dp_u64*>(TH), g.ldh, g.Hp,
                  P * g.Wp, g.Hp, [&](int x, int p0, int m, const float2* lo, const float2* hi) {
    const int pl = g.dWp.div(x), k = x - pl * g.Wp;
    const float f = (k == 0 || 2 * k == g.W) ? 1.f : 2.f;
    float4* dst = R + k * ldx + pl * g.Hp + p0;
#pragma unroll
    for (int e = 0; e < YT; ++e)
      if (e < m)
        dst[e] = make_float4(f * (lo[e].x + lo[e].y), f * (hi[e].x + hi[e].y), f * (lo[e].x - lo[e].y), f * (hi[e].x - hi[e].y));
  });
}

// inverse rows (C2R; the imaginary parts of columns 0 and W/2 meet a zero sine) -> planes in shared
// memory, rows of W | 1 floats
template <int RT, int YT, int NT>
__device__ __forceinline__ void dp_inv_rows(const DpGeom& g, const float4* R, int ldx, const float2* TW, float* out, int P) {
  const int pitch = g.W | 1;
  dp_pass<RT, YT, NT>(reinterpret_cast<const ulonglong2*>(R), ldx, reinterpret_cast<const dp_u64*>(TW), g.ldw, g.Wp,
                  P * g.Hp, g.Wp, [&](int x, int w0, int m, const float2* lo, const float2* hi) {
    const int pl = g.dHp.div(x), p = x - pl * g.Hp;
    float* r0 = out + (pl * g.H + p) * pitch;
    float* r1 = r0 + (g.H - 2 * p) * pitch;
    const bool two = p != 0 && 2 * p != g.H;
#pragma unroll
    for (int e = 0; e < YT; ++e) {
      const int w = w0 + e;
      if (e >= m) continue;
      const bool self_w = w == 0 || 2 * w == g.W;
      r0[w] = lo[e].x + lo[e].y;
      if (!self_w) r0[g.W - w] = lo[e].x - lo[e].y;
      if (two) {
        r1[w] = hi[e].x + hi[e].y;
        if (!self_w) r1[g.W - w] = hi[e].x - hi[e].y;
      }
    }
  });
}

// planes in shared memory (rows of W | 1 floats) -> global memory, times the planes z unless it is null
template <int NT>
__device__ __forceinline__ void dp_store(const DpGeom& g, const float* out, float* __restrict__ dst, const float* __restrict__ z, int P) {
  const int total = P * g.H * g.W, pitch = g.W | 1;
  for (int i0 = threadIdx.x; i0 < total; i0 += 8 * NT) {
    float zv[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int i = i0 + u * NT;
      zv[u] = (z != nullptr && i < total) ? __ldg(z + i) : 1.f;
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int i = i0 + u * NT;
      if (i < total) {
        const int row = g.dW.div(i);
        dst[i] = out[row * pitch + (i - row * g.W)] * zv[u];
      }
    }
  }
}

// Register tiles of a kernel: RT x YT cells in the forward columns, whose epilogue holds the recurrence, and RL x YL in the
// other three passes.  A pass reads 16 (RT + YT / 2) bytes of shared memory for its 2 RT YT packed multiply-adds, so that a
// lane's 16-byte operand (four wavefronts a warp) is what the light passes wait for: eight cells a lane (1 x 8, one operand
// and four broadcast reads of the table) take 8 wavefronts for 16 of them where 2 x 4 takes 10 and 1 x 2 takes 20.  The forward columns have no
// registers left for it, and planes that leave lanes idle want the smaller tiles.  (2 x 8: best for none of 40 shapes.)
template <int RT_, int YT_, int RL_, int YL_> struct DpTiles { static constexpr int RT = RT_, YT = YT_, RL = RL_, YL = YL_; };

// Launch choice of the plane-group kernels: P planes per CTA (a multiple of `unit`; one of `back` is transformed back), the pair of register tiles (dp_pick),
// CTAs per SM, threads, dynamic shared memory.  bytes(g, P, arg): shared memory of P planes.
struct DpChoice { int P, tiles, ctas, threads; size_t smem; double cost; };
DpChoice dp_choose(int H, int W, int C, int B, int unit, int back, size_t limit, size_t (*bytes)(const DpGeom&, int, int), int arg);

constexpr int DP_TILES = 5;
template <class F> auto dp_pick(int tiles, F&& f) {
  switch (tiles) {
    case 0: return f(DpTiles<1, 2, 1, 2>{});
    case 1: return f(DpTiles<1, 2, 1, 4>{});
    case 2: return f(DpTiles<2, 4, 1, 4>{});
    case 3: return f(DpTiles<2, 4, 2, 4>{});
    default: return f(DpTiles<2, 4, 1, 8>{});
  }
}

}  // namespace cssm
