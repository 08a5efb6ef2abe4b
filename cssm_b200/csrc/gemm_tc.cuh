// What the kernels of the 64-channel float32 projections share (csrc/gemm_tc.cu, csrc/gemm_qkv_tconv.cu): raw 128-pixel tiles that
// a loader warp brings by TMA, and converter warps (lane = pixel) that rotate and split them into the A operand in TMEM.
#pragma once
#include <cuda.h>
#include "gemm.cuh"
#include "tc05.cuh"
#include "bf16_ops.cuh"

namespace cssm {

constexpr int TC_BM = 128, TC_K = 64;
constexpr uint32_t TC_RAW = TC_BM * TC_K * 4;                            // one raw tile
constexpr uint32_t TC_ANG = 8 * 32 * 8;                                  // angles of a tile's rows, up to eight: [row][32 pairs]
constexpr uint32_t TC_WANG = 64 * 32 * 8;                                // angles of the columns: [16 pairs of pairs][W]

// Divisions by HW, T and the source-frame divisor.
struct TcGeom {
  FastDiv hw, t, fdiv;
  explicit TcGeom(const GemmArgs& g) : hw(g.HW), t(g.T > 0 ? g.T : 1), fdiv(g.a_fdiv > 1 ? g.a_fdiv : 1) {}
};
__device__ __forceinline__ int tc_src_frame(const GemmArgs& g, const TcGeom& dv, int f) {
  return (g.a_fmul == 0 && g.a_fadd == 0) ? f : dv.fdiv.div(f) * g.a_fmul + g.a_fadd;
}
__device__ __forceinline__ int tc_rope_t(const GemmArgs& g, const TcGeom& dv, int f) { return g.rope_tlast ? g.T - 1 : f - dv.t.div(f) * g.T; }

// RoPE (channels-last A; a tile never crosses a frame, H*W is a multiple of the tile height).  Where tiles are whole image rows of
// 16, 32 or 64 pixels the tables come from shared memory: the columns' angles once per CTA, and with every raw tile those of its
// frame and rows, which the loader adds up for all lanes.  Otherwise every lane reads the tables of its pixel.
__device__ __forceinline__ bool tc_rope_shared(const GemmArgs& g) { return g.rope_t != nullptr && (g.W == 16 || g.W == 32 || g.W == 64); }
__device__ __forceinline__ void tc_rope_columns(const GemmArgs& g, unsigned char* wang, int tid, int threads) {
  for (int i = tid; i < 16 * g.W; i += threads) {
    const int c = i / g.W, w = i - c * g.W;
    reinterpret_cast<float4*>(wang)[i] = __ldg(reinterpret_cast<const float4*>(g.rope_w + w * 32 + 2 * c));
  }
}
// by one warp: rows from px0 on of frame time t
__device__ __forceinline__ void tc_rope_rows(const GemmArgs& g, unsigned char* ang, int t, int px0, int lane) {
  const int wshift = 31 - __clz(g.W), h0 = px0 >> wshift, nrow = TC_BM >> wshift;
  const float2 a = __ldg(g.rope_t + t * 32 + lane);
  for (int r = 0; r < nrow; ++r) {
    const float2 b = __ldg(g.rope_h + (h0 + r) * 32 + lane);
    reinterpret_cast<float2*>(ang)[r * 32 + lane] = make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
  }
}
// bit c: pairs k0 / 2 + 2 c and the next are rotated (most modes rotate the low pairs only)
__device__ __forceinline__ uint32_t tc_rotated(const GemmArgs& g, int k0) {
  uint32_t m = 0;
  if (g.rope_t != nullptr)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int pi = (k0 >> 1) + 2 * c;
      if (g.rope_nz == nullptr || g.rope_nz[pi] != 0.f || g.rope_nz[pi + 1] != 0.f) m |= 1u << c;
    }
  return m;
}
__device__ __forceinline__ void tc_turn(float4 a, float4 w, float (&x)[16], int c) {
  auto turn = [](float tx, float ty, float wx, float wy, float& x, float& y) {
    const float c2 = tx * wx - ty * wy, s2 = tx * wy + ty * wx;
    const float ne = x * c2 - y * s2, no = x * s2 + y * c2;
    x = ne; y = no;
  };
  turn(a.x, a.y, w.x, w.y, x[4 * c], x[4 * c + 1]);
  turn(a.z, a.w, w.z, w.w, x[4 * c + 2], x[4 * c + 3]);
}
// channels [k0, k0 + 16) of the lane's pixel: `row` of the tile, pixel px of its frame at time t
__device__ __forceinline__ void tc_rotate16(const GemmArgs& g, bool shared, uint32_t rot, const unsigned char* ang, const unsigned char* wang,
                                            int row, int t, int px, int k0, float (&v)[16]) {
  if (shared) {
    const float4* an = reinterpret_cast<const float4*>(ang) + (row >> (31 - __clz(g.W))) * 16 + (k0 >> 2);
    const float4* wn = reinterpret_cast<const float4*>(wang) + (k0 >> 2) * g.W + (row & (g.W - 1));
#pragma unroll
    for (int c = 0; c < 4; ++c)
      if (rot >> c & 1) tc_turn(an[c], wn[c * g.W], v, c);
  } else if (rot) {
    const int h = (int)(((float)px + 0.5f) * (1.0f / (float)g.W)), w = px - h * g.W;     // exact for px < 2^22
#pragma unroll
    for (int c = 0; c < 4; ++c)
      if (rot >> c & 1) {
        const int pi = (k0 >> 1) + 2 * c;
        const float4 a = __ldg(reinterpret_cast<const float4*>(g.rope_t + t * 32 + pi));
        const float4 b = __ldg(reinterpret_cast<const float4*>(g.rope_h + h * 32 + pi));
        tc_turn(make_float4(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x, a.z * b.z - a.w * b.w, a.z * b.w + a.w * b.z),
                __ldg(reinterpret_cast<const float4*>(g.rope_w + w * 32 + pi)), v, c);
      }
  }
}

// channels [k0, k0 + 16) of pixel `row`: of a channels-last raw tile (two boxes of 32 channels, 128-byte swizzle) ...
__device__ __forceinline__ void tc_read16_rows(const unsigned char* raw, int row, int k0, float (&v)[16]) {
  const unsigned char* rp = raw + (k0 >> 5) * (TC_BM * 128);
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const float4 x = *reinterpret_cast<const float4*>(rp + tc::sw128_offset(row, ((k0 & 31) >> 2) + c));
    v[4 * c] = x.x; v[4 * c + 1] = x.y; v[4 * c + 2] = x.z; v[4 * c + 3] = x.w;
  }
}
// ... or of planes, times those of the gate behind them
// (returns the sum of the planes' squares where SQ)
template <bool GATE, bool SQ>
__device__ __forceinline__ float tc_read16_planes(const unsigned char* raw, int row, int k0, float (&v)[16]) {
  const float* rp = reinterpret_cast<const float*>(raw) + k0 * TC_BM + row;
  float ss = 0.f;
#pragma unroll
  for (int j = 0; j < 16; ++j) v[j] = rp[j * TC_BM];
  if (SQ) {
#pragma unroll
    for (int j = 0; j < 16; ++j) ss = fmaf(v[j], v[j], ss);
  }
  if (GATE) {
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] *= rp[(TC_K + j) * TC_BM];
  }
  return ss;
}
// hi parts to TMEM columns taddr .. + 15, remainders 32 columns on
__device__ __forceinline__ void tc_split_store16(uint32_t taddr, const float (&v)[16]) {
#pragma unroll
  for (int p = 0; p < 16; p += 8) {                        // eight channels at a time: registers
    uint32_t hi[8], lo[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float h, l;
      tc::split_tf32(v[p + j], h, l);
      hi[j] = __float_as_uint(h); lo[j] = __float_as_uint(l);
    }
    tc::st_32x32b_x8(taddr + p, hi);
    tc::st_32x32b_x8(taddr + 32u + p, lo);
  }
}

// The MMAs of one stage (32 channels in TMEM, hi and lo) into d by half hf of the N rows of B (hi, lo; 128-byte swizzle): the small
// products lo hi, hi lo, and the leading ones.  The accumulator truncates at every MMA, toward zero, so the small products of both
// stages come first and the full sum is truncated eight times instead of 24 (blocks of 64 channels against float64, 32 x 32: additive
// 1.50 -> 0.44, GDN 1.26 -> 0.45 x 1e-6; the joined q, k, v launch 1 % slower, the others not).
template <int N>
__device__ __forceinline__ void tc_mma_small(uint32_t d, uint32_t a, uint64_t b_hi, uint64_t b_lo, int hf, uint32_t idesc) {
  const uint64_t off = (uint64_t)(hf * (N * 128u >> 4));
#pragma unroll
  for (int ks = 0; ks < 4; ++ks) tc::mma_tf32_ts(d, a + 32u + ks * 8u, b_hi + off + ks * 2, idesc, (hf | ks) ? 1u : 0u);
#pragma unroll
  for (int ks = 0; ks < 4; ++ks) tc::mma_tf32_ts(d, a + ks * 8u, b_lo + off + ks * 2, idesc, 1u);
}
template <int N>
__device__ __forceinline__ void tc_mma_lead(uint32_t d, uint32_t a, uint64_t b_hi, int hf, uint32_t idesc) {
#pragma unroll
  for (int ks = 0; ks < 4; ++ks) tc::mma_tf32_ts(d, a + ks * 8u, b_hi + (uint64_t)(hf * (N * 128u >> 4)) + ks * 2, idesc, 1u);
}
// Weights W[k][n0 + n] of a (64, ldn) matrix -> B_hi / B_lo rows n, K-major swizzled
template <int N>
__device__ __forceinline__ void tc_split_weights(const float* Wk, int ldn, int n0, unsigned char* b_hi, unsigned char* b_lo, int tid, int threads) {
  for (int item = tid; item < N * 16; item += threads) {
    const int n = item % N, c = item / N;               // c: 16-byte chunk of 4 k values
    float hi[4], lo[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) tc::split_tf32(Wk[(size_t)(4 * c + e) * ldn + n0 + n], hi[e], lo[e]);
    const uint32_t off = (uint32_t)(c >> 3) * (N * 128u) + tc::sw128_offset(n, c & 7);
    *reinterpret_cast<float4*>(b_hi + off) = make_float4(hi[0], hi[1], hi[2], hi[3]);
    *reinterpret_cast<float4*>(b_lo + off) = make_float4(lo[0], lo[1], lo[2], lo[3]);
  }
}

// The same for three bf16 parts (split3: 24 bits, where two tf32 parts hold 22) and their six products down to 2^-16 of the leading
// one: sixteen channels are eight columns of a part, the parts of a stage sixteen columns apart.
__device__ __forceinline__ void tc_split3_store16(uint32_t taddr, const float (&v)[16]) {
  uint32_t p[3][8];
#pragma unroll
  for (int j = 0; j < 8; ++j) split3(v[2 * j], v[2 * j + 1], p[0][j], p[1][j], p[2][j]);
#pragma unroll
  for (int i = 0; i < 3; ++i) tc::st_32x32b_x8(taddr + 16u * i, p[i]);
}
// b: the first part of B; the others follow N rows on each
template <int N>
__device__ __forceinline__ void tc_mma3(uint32_t d, uint32_t a, uint64_t b, int pa, int pb, int hf, uint32_t idesc, bool first) {
#pragma unroll
  for (int ks = 0; ks < 2; ++ks)
    tc::mma_bf16_ts(d, a + pa * 16u + ks * 8u, b + (uint64_t)(pb * (N * 128 >> 4) + (hf * 2 + ks) * 2), idesc, first && ks == 0 ? 0u : 1u);
}
template <int N>
__device__ __forceinline__ void tc_mma3_small(uint32_t d, uint32_t a, uint64_t b, int hf, uint32_t idesc) {
  constexpr int PA[5] = {2, 0, 1, 1, 0}, PB[5] = {0, 2, 1, 0, 1};
#pragma unroll
  for (int p = 0; p < 5; ++p) tc_mma3<N>(d, a, b, PA[p], PB[p], hf, idesc, (hf | p) == 0);
}
// Weights W[k][n] of a (64, N) matrix times scale[k] -> three parts of N rows, K-major swizzled
template <int N>
__device__ __forceinline__ void tc_split3_weights(const float* Wk, const float* scale, unsigned char* b, int tid, int threads) {
  for (int item = tid; item < N * 16; item += threads) {
    const int n = item % N, c = item / N;               // c: half of a 16-byte chunk, 4 k values
    float w[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) w[e] = Wk[(size_t)(4 * c + e) * N + n] * scale[4 * c + e];
    uint32_t p[3][2];
    split3(w[0], w[1], p[0][0], p[1][0], p[2][0]);
    split3(w[2], w[3], p[0][1], p[1][1], p[2][1]);
#pragma unroll
    for (int i = 0; i < 3; ++i)
      *reinterpret_cast<uint2*>(b + (uint32_t)i * (N * 128u) + tc::sw128_offset(n, c >> 1) + (c & 1) * 8u) = make_uint2(p[i][0], p[i][1]);
  }
}

// Tensor maps of A (and of the gate planes): boxes of 128 rows x 32 channels, 128-byte swizzle, or of 128 pixels x 64 planes.
// They cover all source frames that the tiles name.
bool tc_input_map(const GemmArgs& g, bool a_planar, bool gate, CUtensorMap* map);

}  // namespace cssm
