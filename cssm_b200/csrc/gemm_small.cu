// bf16 GEMM of few rows (one to a few images of the classifier): the latency of one tile counts, not the rate.
//
//   out[m, n] = act( sum_k LN(A)[m, k] * Wt[n, k] + bias[n] ) (+ res[m, n]),  bf16 in, fp32 accumulate.
//
// Tiles of 32 x 32 outputs, 8 warps a CTA, wk = 2, 4 or 8 of them to a tile (8 / wk tiles a CTA): a warp takes every wk-th
// step of 32 k straight from global memory into mma.sync fragments.  A lane's 16-byte loads are eight consecutive k of one
// row; the order of k inside a step is the same for A and Wt, so words x, y are the fragments of one MMA and z, w of the next,
// and nothing passes through shared memory but the partial sums of the wk warps at the end.  All loads of two steps are in
// flight together, those of the weights from before the wait for the previous kernel.
// The rows may be normalised on the way (LN: LayerNorm over K, the whole row being in the fragments of the wk warps), and may
// be the windows of a 3x3 stride-2 conv (CONV).
// mma.sync and not tcgen05: gemm_bf16_kernel spends 8 to 9 us on a launch that these sizes give 1 us of work (barriers and
// TMEM set up and torn down, TMA -> MMA -> epilogue hand-offs of a single 128-row tile, 64 columns of weights and up
// to 36 K blocks in turn on one SM).
#include "kernels.cuh"
#include "bf16_ops.cuh"

namespace cssm {

constexpr int SG_THREADS = 256, SG_PITCH = 40;      // floats per row of a partial tile: rows 8 banks apart

__device__ __forceinline__ void mma_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// NU: steps a warp takes at a time; with LN those of the whole row
template <int wk, int NU, bool LN, bool CONV>
__global__ void __launch_bounds__(SG_THREADS, 2) gemm_small_kernel(const Bf16GemmArgs g, const float* __restrict__ ln_scale,
                                                                const float* __restrict__ ln_bias) {
  __shared__ __align__(16) float part[8][32 * SG_PITCH];
  __shared__ float stat[2][8][32];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gr = lane >> 2, t = lane & 3;
  const int n_tiles = g.N >> 5, tile = blockIdx.x * (8 / wk) + warp / wk, wi = warp % wk;
  const int m0 = (tile / n_tiles) * 32, n0 = (tile % n_tiles) * 32;      // a tile past the end has m0 >= M: loads clamped, no stores
  const int steps = (CONV ? g.Kpad : g.K) >> 5;

  // steps s = wi, wi + wk, ...
  uint4 a[NU][4], b[NU][4];
  const __nv_bfloat16* wp = g.Wt + (size_t)(n0 + gr) * g.ldw + 8 * t;
  auto load_b = [&](int s, uint4 (&v)[4]) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      v[j] = s < steps ? __ldg(reinterpret_cast<const uint4*>(wp + (size_t)(8 * j) * g.ldw + s * 32)) : make_uint4(0u, 0u, 0u, 0u);
  };
#pragma unroll
  for (int u = 0; u < NU; ++u) load_b(wi + u * wk, b[u]);
  // outputs of this thread: 4 columns from 4 (i & 7) of row i >> 3, i = its index in the tile's warps + 32 wk r
  const int lt = wi * 32 + lane, col = n0 + 4 * (lt & 7);
  float4 bias = make_float4(0.f, 0.f, 0.f, 0.f);
  if (g.bias != nullptr) bias = make_float4(__ldg(g.bias + col), __ldg(g.bias + col + 1), __ldg(g.bias + col + 2), __ldg(g.bias + col + 3));
  pdl_sync();

  const __nv_bfloat16* ap[4];
  int h0[4], w0[4];                                   // CONV: window origin
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = min(m0 + gr + 8 * i, g.M - 1);
    if (CONV) {
      const int hw = g.Ho * g.Wo, im = m / hw, px = m - im * hw, ho = px / g.Wo, wo = px - ho * g.Wo;
      h0[i] = ho * 2 - g.pad_h;
      w0[i] = wo * 2 - g.pad_w;
      ap[i] = g.A + (size_t)im * g.Hi * g.Wi * g.Cin + 8 * t;
    } else {
      ap[i] = g.A + (size_t)m * g.lda + 8 * t;
    }
  }
  auto load_a = [&](int s, uint4 (&v)[4]) {
    if (CONV) {
      // conv_tma == 2: two K blocks of 64 per kernel row, [column 0 | column 1] and [column 2 | zeros]
      int ti, tj, c0;
      if (g.conv_tma == 2) { ti = s >> 2; tj = s & 3; c0 = 0; }
      else { const int k = s * 32, tap = k / g.Cin; ti = tap / 3; tj = tap - 3 * ti; c0 = k - tap * g.Cin; }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int h = h0[i] + ti, w = w0[i] + tj;
        const bool in = s < steps && h >= 0 && h < g.Hi && w >= 0 && w < g.Wi && tj < 3 && ti < 3;
        v[i] = in ? __ldg(reinterpret_cast<const uint4*>(ap[i] + ((size_t)h * g.Wi + w) * g.Cin + c0)) : make_uint4(0u, 0u, 0u, 0u);
      }
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) v[i] = s < steps ? __ldg(reinterpret_cast<const uint4*>(ap[i] + s * 32)) : make_uint4(0u, 0u, 0u, 0u);
    }
  };
#pragma unroll
  for (int u = 0; u < NU; ++u) load_a(wi + u * wk, a[u]);
  constexpr int OUT = 8 / wk;                         // outputs of a thread, in fours
  uint2 res[OUT];
#pragma unroll
  for (int r = 0; r < OUT; ++r) {
    const int i = lt + 32 * wk * r, m = m0 + (i >> 3);
    res[r] = (g.res != nullptr && m < g.M) ? __ldg(reinterpret_cast<const uint2*>(g.res + (size_t)m * g.ldr + col)) : make_uint2(0u, 0u);
  }
  if (LN) {
    // the row's wk warps exchange their sums of x, then those of (x - mean)^2
    const float inv = 1.0f / (float)g.K;
    float mean[4], rstd[4];
#pragma unroll
    for (int pass = 0; pass < 2; ++pass) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float s = 0.f;
#pragma unroll
        for (int u = 0; u < NU; ++u) {
          float f[8];
          unpack8(a[u][i], f);
          if (pass == 0) {
#pragma unroll
            for (int e = 0; e < 8; ++e) s += f[e];
          } else if (wi + u * wk < steps) {
#pragma unroll
            for (int e = 0; e < 8; ++e) { const float d = f[e] - mean[i]; s = fmaf(d, d, s); }
          }
        }
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        if (t == 0) stat[pass][warp][gr + 8 * i] = s;
      }
      __syncthreads();
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float s = 0.f;
#pragma unroll
        for (int q = 0; q < wk; ++q) s += stat[pass][warp - wi + q][gr + 8 * i];
        if (pass == 0) mean[i] = s * inv; else rstd[i] = rsqrtf(s * inv + 1e-6f);
      }
    }
#pragma unroll
    for (int u = 0; u < NU; ++u) {
      const int k = min(wi + u * wk, steps - 1) * 32 + 8 * t;
      float sc[8], bi[8];
#pragma unroll
      for (int e = 0; e < 8; e += 4) {
        const float4 s4 = __ldg(reinterpret_cast<const float4*>(ln_scale + k + e)), b4 = __ldg(reinterpret_cast<const float4*>(ln_bias + k + e));
        sc[e] = s4.x; sc[e + 1] = s4.y; sc[e + 2] = s4.z; sc[e + 3] = s4.w;
        bi[e] = b4.x; bi[e + 1] = b4.y; bi[e + 2] = b4.z; bi[e + 3] = b4.w;
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float f[8];
        unpack8(a[u][i], f);
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] = fmaf((f[e] - mean[i]) * rstd[i], sc[e], bi[e]);
        if (wi + u * wk < steps) a[u][i] = pack8(f);
      }
    }
  }

  float acc[2][4][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.f;
#pragma unroll 1
  for (int s = wi;; ) {
#pragma unroll
    for (int u = 0; u < NU; ++u)
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          mma_16816(acc[i][j], a[u][2 * i].x, a[u][2 * i + 1].x, a[u][2 * i].y, a[u][2 * i + 1].y, b[u][j].x, b[u][j].y);
          mma_16816(acc[i][j], a[u][2 * i].z, a[u][2 * i + 1].z, a[u][2 * i].w, a[u][2 * i + 1].w, b[u][j].z, b[u][j].w);
        }
    s += NU * wk;
    if (LN || s >= steps) break;
#pragma unroll
    for (int u = 0; u < NU; ++u) { load_b(s + u * wk, b[u]); load_a(s + u * wk, a[u]); }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float* p = part[warp] + (16 * i + gr) * SG_PITCH + 8 * j + 2 * t;
      *reinterpret_cast<float2*>(p) = make_float2(acc[i][j][0], acc[i][j][1]);
      *reinterpret_cast<float2*>(p + 8 * SG_PITCH) = make_float2(acc[i][j][2], acc[i][j][3]);
    }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < OUT; ++r) {
    const int i = lt + 32 * wk * r, row = i >> 3, m = m0 + row;
    if (m >= g.M) continue;
    float4 v = bias;
#pragma unroll
    for (int q = 0; q < wk; ++q) {
      const float4 p = *reinterpret_cast<const float4*>(part[warp - wi + q] + row * SG_PITCH + 4 * (i & 7));
      v.x += p.x; v.y += p.y; v.z += p.z; v.w += p.w;
    }
    if (g.act == 1) { gelu_tanh_x2(v.x, v.y); gelu_tanh_x2(v.z, v.w); }
    else if (g.act == 2) { silu_tanh_x2(v.x, v.y); silu_tanh_x2(v.z, v.w); }
    const float2 r0 = bf16x2_to_float2(res[r].x), r1 = bf16x2_to_float2(res[r].y);
    if (g.res != nullptr) { v.x += r0.x; v.y += r0.y; v.z += r1.x; v.w += r1.y; }
    *reinterpret_cast<uint2*>(g.out + (size_t)m * g.ldo + col) = make_uint2(float2_to_bf16x2(v.x, v.y), float2_to_bf16x2(v.z, v.w));
  }
}

static int small_split(int steps) { return steps >= 8 ? 8 : steps >= 4 ? 4 : 2; }

// Arguments as launch_gemm_bf16 has validated and completed them (Kpad, conv_tma).
bool gemm_small_supported(const Bf16GemmArgs& g) {
  const bool conv = g.ksz > 0;
  if (g.N % 32 != 0 || (conv ? g.conv_tma == 0 || (g.conv_tma == 1 && g.Cin % 32 != 0) : g.K % 32 != 0)) return false;
  const long long rows = (long long)g.M * (g.whole > 1 ? g.whole : 1);
  const long long tiles = (rows + 31) / 32 * (g.N / 32), steps = (conv ? g.Kpad : g.K) / 32;
  // Up to 16 warps (two rounds of a CTA) an SM, a conv, whose rows are gathered, 12.  us a launch here / gemm_bf16_kernel, at
  // 16: 1176 x 256 x 256 6.2 / 8.3, 784 x 1536 -> 384 12.3 / 16.4, 784 x 1024 -> 256 at 11 8.2 / 12.7; at 21: 784 x 256 -> 512
  // 8.3 / 8.3, 1568 x 128 -> 512 9.3 / 8.2; at 32: 1176 x 256 -> 512 10.3 / 8.3.  Conv at 11: 784 x 1152 -> 256 12.3 / 14.4; at 16:
  // 784 x 2304 -> 384 26 / 23.  With the LayerNorms of fc1 the pass of one 224-pixel image goes from 358 to 256 us, of four from 375 to 316.
  return tiles * small_split((int)steps) <= (conv ? 12 : 16) * (long long)sm_count();
}

// LayerNorm on the way: the row in one step a warp (with two the fragments and their float32 values do not fit 128 registers:
// K = 384 7.4 us a launch, against 2.6 and 3 for LayerNorm and GEMM)
bool gemm_small_ln_supported(int M, int N, int K, int whole, const float* scale, const float* bias) {
  Bf16GemmArgs g = {};
  g.M = M; g.N = N; g.K = K; g.whole = whole;
  return K % 32 == 0 && K <= 32 * small_split(K / 32) && aligned16(scale) && aligned16(bias) && gemm_small_supported(g);
}

template <int WK>
static int launch_v(const Bf16GemmArgs& g, const float* ln_scale, const float* ln_bias, cudaStream_t st) {
  const int per = 8 / WK, tiles = (g.M + 31) / 32 * (g.N / 32);
  const bool one = g.K <= 32 * WK;                    // one step a warp
  auto kern = g.ksz > 0 ? gemm_small_kernel<WK, 2, false, true>
              : ln_scale == nullptr ? (one ? gemm_small_kernel<WK, 1, false, false> : gemm_small_kernel<WK, 2, false, false>)
                                    : gemm_small_kernel<WK, 1, true, false>;
  launch_k(kern, (unsigned)((tiles + per - 1) / per), SG_THREADS, 0, st, g, ln_scale, ln_bias);
  return check_launch();
}

int launch_gemm_small(const Bf16GemmArgs& g, const float* ln_scale, const float* ln_bias, cudaStream_t st) {
  const int wk = small_split((g.ksz > 0 ? g.Kpad : g.K) / 32);
  return wk == 8 ? launch_v<8>(g, ln_scale, ln_bias, st) : wk == 4 ? launch_v<4>(g, ln_scale, ln_bias, st) : launch_v<2>(g, ln_scale, ln_bias, st);
}

}  // namespace cssm
