// tcgen05 / TMEM GEMM of the float32 channel projections, any K, N and plane size.
//
// Every float32 operand is split into three bfloat16 parts, x = x0 + x1 + x2 (8 significant bits
// each: the sum is exact to float32's own 24), and the product is taken as the six partial products
// whose weight reaches 2^-16 of the leading one (00, 01, 10, 11, 02, 20), accumulated in float32 in
// TMEM.  What is dropped is below 2^-24 of |a||b|.  A bf16 MMA runs at twice the tf32 rate, so six of them
// cost what three tf32 passes cost, in three quarters of the shared memory.  The accumulator truncates
// at every MMA, so with more than one K block the 00 products have accumulators of their own and the five
// small ones another (24 truncations of the full sum at K = 384 instead of 144: relative error 2.2e-6 before).
// The truncations all go toward zero, so the error of one accumulator grows like the number of MMAs added to it
// (0.56e-7 of the 2-norm for every K block of 64), that of float32 FMAs like its root (1.37e-7 sqrt(K blocks)).
// Above six K blocks the 00 products are therefore dealt out to several accumulators (WIDE) of at most
// 2 sqrt(K blocks) each, which the epilogue adds in registers, rounding to nearest.  Error against float64 (1e-7)
// with one leading accumulator / so / with FMAs: K = 512 4.5 / 2.2 / 3.9, 1024 9.5 / 4.5 / 5.5, 2048 20 / 6.2 / 7.8,
// 4096 42 / 9.6 / 11; it costs less than 1 % (96 x 14 x 14 x 1024, whole block: 1965 -> 1974 us).
//
// Persistent kernel, one CTA per SM, 544 threads, warp-specialised:
//   warps 0-7  producers : 128-row x 64-k A blocks (of K <= 32 only the half that the MMAs read) from global memory (channels-last rows with RoPE
//                          applied, or planar planes times scale and gate), fetched one block ahead
//                          into registers, split, and written into the 128-byte-swizzled K-major
//                          operand layout of the ring; with streamed weights also the B blocks;
//   warp  8    MMA issuer: one lane issues 6 x (K block / 16) tcgen05.mma per block into one of two
//                          TMEM accumulators and commits to mbarriers;
//   warps 9-16 epilogue  : tcgen05.ld (lane = pixel row; two warps per TMEM lane quadrant, half of the
//                          32-column chunks each), 1/rms, bias, activation; planar stores (coalesced
//                          over pixels) or channels-last rows through a per-warp TMA tensor store.
// RES: the whole (K, BN) weight tile is split once per CTA and stays in shared memory (the ring then
// carries A only); without it the producers split the weight block of every stage again, unless the caller had the weights
// split beforehand (wsplit): then bulk copies bring the blocks, which halves what the producers do (float32 mixers of the
// classifier, 33 images of 256 pixels: a pass 823 -> 752 us).
// Rows are flat pixels m = frame * HW + px, so a tile may cross frames and HW may be anything.
// Every mbarrier wait is bounded; on expiry the kernel records an error code and winds down.
//
// Bound: the producers (about 300 instructions a thread and tile, twice that with RoPE; a clock trace of
// one CTA shows the MMA warp waiting for them), not memory: at K = 64 it reaches 0.6 of the HBM rate.
// Against the CUDA-core GEMM that covered these sizes before (batch x frames, plane, channels):
// in_proj 48 x 8 x 14^2, 256 -> 512: 884 -> 211 us; in_proj + B_k/B_v + qkv of 12 x 8 x 28^2, 64: 271 -> 56 us;
// out_proj 33 x 16^2, 256 -> 256: 121 -> 36 us; 16 x 8 x 56^2, 32 -> 64: 150 -> 67 us, 32 -> 32: 134 -> 37 us.
#include <cuda.h>
#include <cuda_bf16.h>
#include <math.h>
#include <string.h>
#include "kernels.cuh"
#include "bf16_ops.cuh"
#include "gemm.cuh"
#include "tc05.cuh"

namespace cssm {

__device__ int g_split_error = 0;

// 8 producer warps, 1 MMA warp, 8 epilogue warps (with 16 producer warps 72 registers a thread are left
// and the kernel is slower throughout).
constexpr int GS_PROD = 256;
constexpr int GS_THREADS = GS_PROD + 32 + 256;
constexpr int GS_MMA_WARP = GS_PROD / 32;
constexpr int GS_BM = 128, GS_BK = 64;
constexpr uint32_t GS_A_PART = GS_BM * 128u;           // one bf16 part of an A block
constexpr uint32_t GS_A_BYTES = 3u * GS_A_PART;
constexpr int GS_SS = 8;             // row-sum buffers (producers run at most five tiles ahead of the epilogue)

// streaming loads that leave the L1 (a few KB beside the shared memory in use) to the RoPE tables
__device__ __forceinline__ void ld_stream4(const float* p, float* v) {
  asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "l"(p));
}

template <int V> struct Int { static constexpr int value = V; };

struct SplitGeom {
  int BN, n_tiles, m_tiles, kblocks, stages;
  int nl;                             // leading accumulators beside that of the small partial products (0: one for all)
  int lead;                           // WIDE: K blocks of one leading accumulator
  int bufs;                           // WIDE: accumulator sets, 2 (the epilogue drains one while the MMAs fill the
                                      // other) or 1; otherwise 2
  FastDiv hw, w, t, fdiv;             // divisions by HW, W, T and the source-frame divisor
};

// The arguments once more, for the path that takes their address: with the address of g and q themselves the
// block 16 x 8 x 56 x 56 x 32 took 398 instead of 393 us.
struct SplitArgs { GemmArgs g; SplitGeom q; };

// eight consecutive k values -> one 16-byte chunk in each of the three parts
__device__ __forceinline__ void store_split8(unsigned char* base, uint32_t off, uint32_t part, const float (&v)[8]) {
  uint4 a, b, c;
  split3(v[0], v[1], a.x, b.x, c.x);
  split3(v[2], v[3], a.y, b.y, c.y);
  split3(v[4], v[5], a.z, b.z, c.z);
  split3(v[6], v[7], a.w, b.w, c.w);
  *reinterpret_cast<uint4*>(base + off) = a;
  *reinterpret_cast<uint4*>(base + part + off) = b;
  *reinterpret_cast<uint4*>(base + 2 * part + off) = c;
}
__device__ __forceinline__ void mma_f16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                        uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}

// Columns [n, n + 32) of output row m once more, by float32 FMAs over k: for results that are not finite.  An
// infinity, or a value above the largest bfloat16 (3.39e38), has no finite parts: the partial products give
// inf - inf where the sum itself is infinite, or even finite.
template <bool A_PLANAR>
__device__ __noinline__ void split_row_fma(const SplitArgs& a, int m, int n, float rinv) {
  const GemmArgs& g = a.g;
  const SplitGeom& q = a.q;
  const int fo = q.hw.div(m), px = m - fo * g.HW, tt = fo - q.t.div(fo) * g.T;
  const int fr = (g.a_fmul != 0 || g.a_fadd != 0) ? q.fdiv.div(fo) * g.a_fmul + g.a_fadd : fo;
#pragma unroll 1
  for (const int end = min(n + 32, g.N); n < end; ++n) {
    const float* w = g.Wk + n;
    float v = 0.f;
    if (A_PLANAR) {
      const float* ap = g.A + ((size_t)fr * g.a_planes + g.a_plane0) * g.HW + px;
      const float* gp = g.gate ? g.gate + ((size_t)(g.g_compact ? fo : fr) * g.g_planes + g.g_plane0) * g.HW + px : nullptr;
      for (int k = 0; k < g.K; ++k) {
        float x = ap[(size_t)k * g.HW];
        if (g.rms_scale != nullptr) x *= rinv * g.rms_scale[k];
        if (gp != nullptr) x *= gp[(size_t)k * g.HW];
        v = fmaf(x, w[(size_t)k * g.N], v);
      }
    } else {
      const float* ap = g.A + ((size_t)fr * g.HW + px) * g.K;
      const int t = g.rope_tlast ? g.T - 1 : tt, h = q.w.div(px), wi = px - h * g.W, n2 = g.K >> 1;
      for (int k = 0; k < g.K; k += 2) {
        float x = ap[k], y = ap[k + 1];
        if (g.rope_t != nullptr && (g.rope_nz == nullptr || g.rope_nz[k >> 1] != 0.f)) {
          const float2 ct = g.rope_t[t * n2 + (k >> 1)], ch = g.rope_h[h * n2 + (k >> 1)], cw = g.rope_w[wi * n2 + (k >> 1)];
          const float cx = ct.x * ch.x - ct.y * ch.y, sx = ct.x * ch.y + ct.y * ch.x;
          const float c2 = cx * cw.x - sx * cw.y, s2 = cx * cw.y + sx * cw.x;
          const float ne = x * c2 - y * s2;
          y = x * s2 + y * c2;
          x = ne;
        }
        v = fmaf(x, w[(size_t)k * g.N], v);
        v = fmaf(y, w[(size_t)(k + 1) * g.N], v);
      }
    }
    if (g.bias != nullptr) v += g.bias[n];
    if (A_PLANAR) {
      g.out[(size_t)m * g.N + n] = g.sub != nullptr ? v - g.sub[(size_t)m * g.N + n] : v;
    } else {
      if (n >= g.act_n0 && g.z_last_only && tt != g.T - 1) continue;
      if (n >= g.act_n0 && g.out_act != 0) v = g.out_act == 1 ? silu_f(v) : sigmoid_f(v);
      g.out[((size_t)fo * g.o_planes + g.o_plane0 + n) * g.HW + px] = v;
    }
  }
}

// One 16-byte chunk per thread and part: rows n of 32-row groups, [group][K block][part][32 rows x 128 bytes], 128-byte swizzle
__global__ void __launch_bounds__(256) split_weights_kernel(int K, const float* __restrict__ w0, int N0, unsigned char* __restrict__ out0,
                                                            const float* __restrict__ w1, int N1, unsigned char* __restrict__ out1,
                                                            int items0, int items) {
  pdl_sync();
  int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= items) return;
  const bool second = i >= items0;
  const float* w = second ? w1 : w0;
  const int N = second ? N1 : N0;
  unsigned char* out = second ? out1 : out0;
  if (second) i -= items0;
  const int kchunks = (K + GS_BK - 1) / GS_BK * 8, n = i % ((N + 31) / 32 * 32), ck = i / ((N + 31) / 32 * 32), kb = ck >> 3;
  float v[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) v[e] = n < N && ck * 8 + e < K ? __ldg(w + (size_t)(ck * 8 + e) * N + n) : 0.f;
  store_split8(out + ((size_t)(n >> 5) * (kchunks >> 3) + kb) * 3 * 4096, tc::sw128_offset(n & 31, ck & 7), 4096, v);
}

size_t split_weights_bytes(int K, int N) {
  const int kblocks = (K + GS_BK - 1) / GS_BK;
  return kblocks < 4 ? 0 : (size_t)((N + 31) / 32) * kblocks * 3 * 4096;
}

int launch_split_weights(int K, const float* w0, int N0, void* out0, const float* w1, int N1, void* out1, cudaStream_t st) {
  const int kchunks = (K + GS_BK - 1) / GS_BK * 8, items0 = (N0 + 31) / 32 * 32 * kchunks, items = items0 + (N1 + 31) / 32 * 32 * kchunks;
  launch_k(split_weights_kernel, (items + 255) / 256, 256, 0, st, K, w0, N0, (unsigned char*)out0, w1, N1, (unsigned char*)out1, items0, items);
  return check_launch();
}

// GATE: planar A times the gate planes.  WIDE: more than one leading accumulator (nl > 1).
// PRE (channels-last A): weights split beforehand.  Planar A without gate planes tests wsplit at run time, with gate planes there never is
// one: where the test is not needed it costs (GDN 100 x 2 x 14 x 14 x 384 1577 us a pass with it in the gated form, 1556 without;
// gated 1 x 2 x 14 x 14 x 384 62.1 / 60.7 in the channels-last one), and planar A is not better off with a variant of its own.
template <bool A_PLANAR, bool RES, bool GATE, bool WIDE, bool PRE = false>
__global__ void __launch_bounds__(GS_THREADS, 1)
gemm_split_kernel(const GemmArgs g, const SplitGeom q, const __grid_constant__ CUtensorMap omap,
                  const __grid_constant__ SplitArgs again) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  // operand tiles need 1024-byte alignment (swizzle atoms); the launch adds 1024 bytes of slack
  unsigned char* smem = smem_raw + ((1024u - (tc::smem_u32(smem_raw) & 1023u)) & 1023u);
  const uint32_t sbase = tc::smem_u32(smem);
  const uint32_t BN = (uint32_t)q.BN, b_part = BN * 128u, b_block = 3u * b_part;
  const int NS = q.stages, kblocks = q.kblocks;
  const bool pre_split = (PRE || (A_PLANAR && !RES && !GATE)) && g.wsplit != nullptr;
  const uint32_t res_bytes = RES ? (uint32_t)kblocks * b_block : 0u;
  const uint32_t stage_bytes = GS_A_BYTES + (RES ? 0u : b_block);
  unsigned char* ring = smem + res_bytes;
  unsigned char* stg = ring + (uint32_t)NS * stage_bytes;         // 8 x 4 KB when the output is channels-last
  // RES: bias of the CTA's N tile; else 32 floats per epilogue warp, filled for every 32-column chunk.
  // (The bias itself is read by scalars: it may sit at any 4-byte offset of a parameter buffer.)
  float* bias_s = reinterpret_cast<float*>(stg + (A_PLANAR ? 8u * 4096u : 0u));
  // (barriers before the row sums, which not every launch has: with their address depending on that, the short launches of 392 to
  // 5880 rows and 288 to 512 channels took 2 to 5 % of the ungated block's pass longer)
  uint64_t* bars = reinterpret_cast<uint64_t*>(bias_s + 256);
  float* ss_s = bias_s + 256 + 32;                                // [GS_SS][2][128] row sums (RMS prologue alone has room for them)
  uint64_t* full = bars;           // [4] block written (8 producer warps)
  uint64_t* empty = bars + 4;      // [4] block consumed (tcgen05.commit)
  uint64_t* accfull = bars + 8;    // [2] accumulator set complete (tcgen05.commit)
  uint64_t* accempty = bars + 10;  // [2] accumulator set drained (8 epilogue warps)
  uint64_t* done = bars + 12;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 13);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int num_tiles = q.m_tiles * q.n_tiles;
  const int bufs = WIDE ? q.bufs : 2;
  const uint32_t acc_cols = WIDE ? (1u + (uint32_t)q.nl) * BN : (q.nl ? 2u * BN : BN);      // of one set: [small | leading 0 | ...]
  uint32_t tmem_cols = 32;
  while (tmem_cols < (uint32_t)bufs * acc_cols) tmem_cols <<= 1;

  if (tid == 0) {
    for (int s = 0; s < NS; ++s) { tc::mbar_init(&full[s], GS_PROD / 32 + (pre_split ? 1 : 0)); tc::mbar_init(&empty[s], 1); }
    for (int a = 0; a < 2; ++a) { tc::mbar_init(&accfull[a], 1); tc::mbar_init(&accempty[a], 8); }
    tc::mbar_init(done, 1);
    tc::fence_mbar_init();
  }
  if (warp == GS_MMA_WARP) {
    tc::tmem_alloc(tmem_slot, tmem_cols);
    tc::tmem_relinquish();
  }
  // one 8-k chunk of weight row n (columns of the (K, N) matrix), zero outside the matrix
  auto load_w8 = [&](int n, int k0, float (&v)[8]) {
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int k = k0 + e;
      float w = (n < g.N && k < g.K) ? __ldg(g.Wk + (size_t)k * g.N + n) : 0.f;
      if (A_PLANAR && g.rms_scale != nullptr && k < g.K) w *= __ldg(g.rms_scale + k);
      v[e] = w;
    }
  };
  const int n_first = (blockIdx.x % q.n_tiles) * q.BN;            // RES: the N tile of this CTA
  if (RES) {
    for (int item = tid; item < q.BN * kblocks * 8; item += GS_THREADS) {
      const int n = item % q.BN, ck = item / q.BN;                // ck: 8-k chunk over all K blocks
      float v[8];
      load_w8(n_first + n, ck * 8, v);
      store_split8(smem + (uint32_t)(ck >> 3) * b_block, tc::sw128_offset(n, ck & 7), b_part, v);
    }
    for (int n = tid; n < q.BN; n += GS_THREADS) bias_s[n] = (g.bias && n_first + n < g.N) ? g.bias[n_first + n] : 0.f;
  }
  tc::fence_proxy_async();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  pdl_sync();

  if (warp < GS_MMA_WARP) {
    // ================================ producers ================================
    // channels-last: item i of a thread is the 4-k chunk (lane & 7) + 8 (i >> 2) of row prow0 + 32 (i & 3), so
    // a warp load covers four rows x 128 contiguous bytes.  Most RoPE modes rotate the low channel pairs
    // only: with this order they are the first half of the items of six lanes in eight, not all items of
    // three.  The four rows of a warp are four apart, which keeps its 8-byte stores free of conflicts.
    // planar: thread = (pixel row tid & 127, k half tid >> 7).
    float pre[32], gpre[GATE ? 32 : 1];
    const int chunk = lane & 7, prow0 = (lane >> 3) * 4 + (warp & 3) + 16 * (warp >> 2);
    // the lane's two chunks inside a part, rows prow0 (+ 32 r)
    const uint32_t dst0 = tc::sw128_offset(prow0, chunk >> 1) + (chunk & 1) * 8;
    const uint32_t dst1 = tc::sw128_offset(prow0, (chunk >> 1) + 4) + (chunk & 1) * 8;
    const int prow = tid & 127, kh = tid >> 7, kw = g.K <= 32 ? 16 : 32;      // planar: k values of a thread
    const bool rope = !A_PLANAR && g.rope_t != nullptr;
    const bool remap = g.a_fmul != 0 || g.a_fadd != 0;
    auto fetch = [&](int tile, int kb) {
      const int m0 = (tile / q.n_tiles) * GS_BM, k0 = kb * GS_BK;
      if constexpr (!A_PLANAR) {
        if (!remap && m0 + GS_BM <= g.M && k0 + GS_BK <= g.K) {      // whole block, rows one after another
          const float* p = g.A + (size_t)(m0 + prow0) * g.K + k0 + chunk * 4;
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            ld_stream4(p, pre + 4 * r);
            ld_stream4(p + 32, pre + 16 + 4 * r);
            p += 32 * g.K;
          }
          return;
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const int m = m0 + prow0 + 32 * r;
          size_t row = (size_t)m;
          if (remap) {
            const int fo = q.hw.div(m);
            row = (size_t)(q.fdiv.div(fo) * g.a_fmul + g.a_fadd) * g.HW + (m - fo * g.HW);
          }
          const float* p = g.A + row * g.K + k0 + chunk * 4;
#pragma unroll
          for (int hf = 0; hf < 2; ++hf) {
            if (hf == 1 && k0 + 32 >= g.K) continue;                 // (the MMAs of such a block end before its second half)
            float* v = pre + 16 * hf + 4 * r;
            if (m < g.M && k0 + (chunk + 8 * hf) * 4 < g.K) ld_stream4(p + 32 * hf, v);
            else v[0] = v[1] = v[2] = v[3] = 0.f;
          }
        }
      } else {
        const int m = m0 + prow, kk = k0 + kh * kw;
        const int nk = m < g.M ? min(g.K - kk, kw) : 0;    // values of this thread from kk on
        const int fo = q.hw.div(min(m, g.M - 1)), px = min(m, g.M - 1) - fo * g.HW;
        const int fr = remap ? q.fdiv.div(fo) * g.a_fmul + g.a_fadd : fo;
        const float* ap = g.A + ((size_t)fr * g.a_planes + g.a_plane0 + kk) * g.HW + px;
#pragma unroll
        for (int j = 0; j < 32; ++j) pre[j] = j < nk ? __ldg(ap + (size_t)j * g.HW) : 0.f;
        if constexpr (GATE) {
          const float* gp = g.gate + ((size_t)(g.g_compact ? fo : fr) * g.g_planes + g.g_plane0 + kk) * g.HW + px;
#pragma unroll
          for (int j = 0; j < 32; ++j) gpre[j] = j < nk ? __ldg(gp + (size_t)j * g.HW) : 0.f;
        }
      }
    };
    int tile = blockIdx.x, kb = 0, it = 0, tcnt = 0, rot_kb = -1;
    float ss = 0.f;
    bool rot[2] = {false, false};       // this lane's chunk in either half of the block holds rotated pairs
    if (tile < num_tiles) fetch(tile, 0);
    while (tile < num_tiles) {
      const int s = it % NS;
      const int m0 = (tile / q.n_tiles) * GS_BM, k0 = kb * GS_BK;
      int ntile = tile, nkb = kb + 1;
      if (nkb == kblocks) { nkb = 0; ntile += gridDim.x; }
      unsigned char* a_s = ring + (uint32_t)s * stage_bytes;
      if constexpr (!A_PLANAR) {
        if (rope && rot_kb != kb) {
          rot_kb = kb;
#pragma unroll
          for (int hf = 0; hf < 2; ++hf) {
            const int k = k0 + (chunk + 8 * hf) * 4;
            rot[hf] = k < g.K && (g.rope_nz == nullptr || __ldg(g.rope_nz + (k >> 1)) != 0.f ||
                                  __ldg(g.rope_nz + (k >> 1) + 1) != 0.f);
          }
        }
        if (rot[0] || rot[1]) {
          const int n2 = g.K >> 1, pi = (k0 >> 1) + 2 * chunk;
          const int fr0 = q.hw.div(m0), px0 = m0 - fr0 * g.HW;
          const int t0 = g.rope_tlast ? g.T - 1 : fr0 - q.t.div(fr0) * g.T;
          const bool crosses = px0 + GS_BM > g.HW;            // the tile runs into the next frame(s)
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            int px = px0 + prow0 + 32 * r, t = t0;
            if (crosses && px >= g.HW) {
              const int m = min(m0 + prow0 + 32 * r, g.M - 1), fr = q.hw.div(m);
              px = m - fr * g.HW;
              if (!g.rope_tlast) t = fr - q.t.div(fr) * g.T;
            }
            const int h = q.w.div(px), w = px - h * g.W;
            const float2* pt = g.rope_t + t * n2 + pi;
            const float2* ph = g.rope_h + h * n2 + pi;
            const float2* pw = g.rope_w + w * n2 + pi;
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
              if (!rot[hf]) continue;
              // two pairs per 16-byte table load (K % 4 == 0)
              const float4 ct = __ldg(reinterpret_cast<const float4*>(pt + 16 * hf));
              const float4 ch = __ldg(reinterpret_cast<const float4*>(ph + 16 * hf));
              const float4 cw = __ldg(reinterpret_cast<const float4*>(pw + 16 * hf));
              float* x = pre + 16 * hf + 4 * r;
              // (cos, sin) of the summed angle, then the rotation of one pair
              auto turn = [](float tx, float ty, float hx, float hy, float wx, float wy, float& u, float& v) {
                const float cx = tx * hx - ty * hy, sx = tx * hy + ty * hx;
                const float c2 = cx * wx - sx * wy, s2 = cx * wy + sx * wx;
                const float ne = u * c2 - v * s2, no = u * s2 + v * c2;
                u = ne; v = no;
              };
              turn(ct.x, ct.y, ch.x, ch.y, cw.x, cw.y, x[0], x[1]);
              turn(ct.z, ct.w, ch.z, ch.w, cw.z, cw.w, x[2], x[3]);
            }
          }
        }
        // warp-uniform exit: the lanes of a warp meet again at the __syncwarp before the arrive
        if (__any_sync(0xffffffffu, !tc::mbar_wait(&empty[s], ((it / NS) & 1) ^ 1))) { atomicExch(&g_split_error, 1); break; }
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          if (hf == 1 && k0 + 32 >= g.K) continue;
          unsigned char* dst = a_s + (hf ? dst1 : dst0);
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            const float* x = pre + 16 * hf + 4 * r;
            uint2 a, b, c;
            split3(x[0], x[1], a.x, b.x, c.x);
            split3(x[2], x[3], a.y, b.y, c.y);
            *reinterpret_cast<uint2*>(dst + r * 4096) = a;                       // 32 rows = 4096 bytes on
            *reinterpret_cast<uint2*>(dst + r * 4096 + GS_A_PART) = b;
            *reinterpret_cast<uint2*>(dst + r * 4096 + 2 * GS_A_PART) = c;
          }
        }
        if (ntile < num_tiles) fetch(ntile, nkb);
      } else {
        if (g.rms_scale != nullptr) {
          // the sum of squares of this part of the row; 1/rms is a row factor, applied to the accumulator
#pragma unroll
          for (int j = 0; j < 32; ++j) ss = fmaf(pre[j], pre[j], ss);
        }
        if (__any_sync(0xffffffffu, !tc::mbar_wait(&empty[s], ((it / NS) & 1) ^ 1))) { atomicExch(&g_split_error, 1); break; }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          if (8 * c >= kw) continue;
          float v[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) v[e] = GATE ? pre[8 * c + e] * gpre[GATE ? 8 * c + e : 0] : pre[8 * c + e];
          store_split8(a_s, tc::sw128_offset(prow, kh * (kw >> 3) + c), GS_A_PART, v);
        }
        if (g.rms_scale != nullptr && nkb == 0) { ss_s[((tcnt % GS_SS) * 2 + kh) * 128 + prow] = ss; ss = 0.f; }
        if (ntile < num_tiles) fetch(ntile, nkb);
      }
      if (pre_split) {
        if (tid == 0) {                                 // (it has waited for the stage above)
          unsigned char* b_s = a_s + GS_A_BYTES;
          const int grp0 = (tile % q.n_tiles) * (q.BN >> 5), grps = min(q.BN >> 5, ((g.N + 31) >> 5) - grp0);
          tc::mbar_expect_tx(&full[s], (uint32_t)grps * 3u * 4096u);
          const unsigned char* src = static_cast<const unsigned char*>(g.wsplit) + ((size_t)grp0 * kblocks + kb) * 3 * 4096;
          for (int i = 0; i < grps; ++i)
            for (int p = 0; p < 3; ++p)
              tc::bulk_g2s(b_s + p * b_part + i * 4096, src + ((size_t)i * kblocks * 3 + p) * 4096, 4096, &full[s]);
        }
      } else if (!RES) {
        unsigned char* b_s = a_s + GS_A_BYTES;
        const int n0 = (tile % q.n_tiles) * q.BN;
        for (int item = tid; item < q.BN * 8; item += GS_PROD) {
          const int n = item % q.BN, c = item / q.BN;
          float v[8];
          load_w8(n0 + n, k0 + c * 8, v);
          store_split8(b_s, tc::sw128_offset(n, c), b_part, v);
        }
      }
      tc::fence_proxy_async();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&full[s]);
      if (nkb == 0) ++tcnt;
      tile = ntile; kb = nkb; ++it;
    }
  } else if (warp == GS_MMA_WARP) {
    // ================================ MMA issuer ================================
    // The whole warp walks the loop, one lane issues (elect_one).
    const uint32_t idesc = tc::make_idesc_bf16(GS_BM, BN);
    // (A part, B part) of the six partial products, smallest first
    constexpr int PA[6] = {2, 0, 1, 1, 0, 0}, PB[6] = {0, 2, 1, 0, 1, 0};
    int s = 0, sph = 0, ac = 0, aph = 1;
    bool ok = true;
    for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
      if (__any_sync(0xffffffffu, !tc::mbar_wait(&accempty[ac], aph))) { atomicExch(&g_split_error, 2); ok = false; break; }
      tc::fence_after_sync();
      const uint32_t d = tmem_base + (uint32_t)ac * acc_cols;
      uint32_t d00 = WIDE || !q.nl ? d : d + BN;
      int left = 0;                                     // WIDE: K blocks that still go to the leading accumulator d00
      for (int kb = 0; kb < kblocks; ++kb) {
        if (__any_sync(0xffffffffu, !tc::mbar_wait(&full[s], sph))) { atomicExch(&g_split_error, 2); ok = false; break; }
        tc::fence_after_sync();
        const uint32_t a_s = sbase + res_bytes + (uint32_t)s * stage_bytes;
        const uint32_t b_s = RES ? sbase + (uint32_t)kb * b_block : a_s + GS_A_BYTES;
        const uint64_t ad0 = tc::make_desc_sw128(a_s), bd0 = tc::make_desc_sw128(b_s);
        const uint64_t bp = (uint64_t)(b_part >> 4);
        const uint64_t bd[3] = {bd0, bd0 + bp, bd0 + 2 * bp};
        const uint32_t first = kb == 0 ? 0u : 1u;
        uint32_t first00 = q.nl ? first : 1u;           // (one accumulator: the small products came before)
        if (WIDE) {
          first00 = left == 0 ? 0u : 1u;
          if (left == 0) { d00 += BN; left = q.lead; }
          --left;
        }
        auto issue = [&](auto steps) {
          constexpr int KS = decltype(steps)::value;
#pragma unroll
          for (int p = 0; p < 6; ++p)
#pragma unroll
            for (int ks = 0; ks < KS; ++ks)
              mma_f16(p == 5 ? d00 : d, ad0 + PA[p] * (GS_A_PART >> 4) + ks * 2, bd[PB[p]] + ks * 2, idesc,
                      p == 5 && ks == 0 ? first00 : (p | ks ? 1u : first));
        };
        const int krem = g.K - kb * GS_BK;
        if (tc::elect_one()) {
          if (krem > 48) issue(Int<4>());
          else if (krem > 32) issue(Int<3>());
          else if (krem > 16) issue(Int<2>());
          else issue(Int<1>());
          tc::commit(&empty[s]);
          if (kb + 1 == kblocks) tc::commit(&accfull[ac]);
        }
        __syncwarp();
        if (++s == NS) { s = 0; sph ^= 1; }
      }
      if (++ac == bufs) { ac = 0; aph ^= 1; }
    }
    // nothing of this warp's tensor work may be in flight when TMEM is freed
    if (tc::elect_one()) tc::commit(done);
    __syncwarp();
    if (!tc::mbar_wait(done, 0) && ok) atomicExch(&g_split_error, 3);
    __syncwarp();
  } else {
    // ================================ epilogue ================================
    const int quad = warp & 3;                          // TMEM lane quadrant this warp may read
    const int half = (warp - (GS_MMA_WARP + 1)) >> 2;   // even or odd 32-column chunks
    const int row = quad * 32 + lane;
    unsigned char* my_stg = stg + (uint32_t)(warp - (GS_MMA_WARP + 1)) * 4096u;
    int tcnt = 0;
    for (int tile = blockIdx.x; tile < num_tiles; tile += gridDim.x, ++tcnt) {
      const int ac = tcnt & (bufs - 1), ph = (tcnt >> (bufs - 1)) & 1;
      const int m0 = (tile / q.n_tiles) * GS_BM, n0 = (tile % q.n_tiles) * q.BN;
      const int m = m0 + row;
      int fr = 0, px = 0;
      bool zrow = true;                                 // this row's z columns are wanted
      if (!A_PLANAR) {
        fr = q.hw.div(min(m, g.M - 1)); px = m - fr * g.HW;
        zrow = !g.z_last_only || fr - q.t.div(fr) * g.T == g.T - 1;
      }
      if (__any_sync(0xffffffffu, !tc::mbar_wait(&accfull[ac], ph))) { atomicExch(&g_split_error, 4); break; }
      tc::fence_after_sync();
      float rinv = 1.f;
      if (A_PLANAR && g.rms_scale != nullptr) {
        const float* sp = ss_s + (tcnt % GS_SS) * 256 + row;
        rinv = rsqrtf((sp[0] + sp[128]) / (float)g.K + 1e-6f);
      }
      const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)ac * acc_cols;
      float odd = 0.f;                                  // NaN once a result of the row is not finite
#pragma unroll 1
      for (int cc = half; cc * 32 < q.BN; cc += 2) {
        const int n = n0 + cc * 32;
        if (n >= g.N) break;
        const bool zcols = n >= g.act_n0;               // all 32 columns are activated ones
        if (!A_PLANAR && zcols && g.z_last_only && !__any_sync(0xffffffffu, zrow)) continue;
        const float* bias_c = bias_s + (RES ? cc * 32 : (warp - (GS_MMA_WARP + 1)) * 32);
        if (!RES) {
          const float b = (g.bias && n + lane < g.N) ? __ldg(g.bias + n + lane) : 0.f;
          __syncwarp();                                 // the chunk before has been read
          bias_s[(warp - (GS_MMA_WARP + 1)) * 32 + lane] = b;
          __syncwarp();
        }
        float v[32];
        {
          uint32_t r[32];
          tc::ld_32x32b_x32(taddr + cc * 32, r);
          tc::wait_ld();
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
        }
        for (int l = 1; l <= (WIDE ? q.nl : q.nl ? 1 : 0); ++l) {
#pragma unroll
          for (int hf = 0; hf < 2; ++hf) {
            uint32_t r[16];
            tc::ld_32x32b_x16(taddr + l * BN + cc * 32 + hf * 16, r);
            tc::wait_ld();
#pragma unroll
            for (int j = 0; j < 16; ++j) v[hf * 16 + j] += __uint_as_float(r[j]);
          }
        }
        // (16 packed FMAs a thread and 32 columns: the same block 393 -> 395 us)
        unsigned long long od[2] = {pk2(odd, 0.f), 0ull};
#pragma unroll
        for (int j = 0; j < 32; j += 2) od[(j >> 1) & 1] = fma2(pk2(v[j], v[j + 1]), 0ull, od[(j >> 1) & 1]);
        float o0, o1, o2, o3;
        upk2(od[0], o0, o1); upk2(od[1], o2, o3);
        odd = (o0 + o1) + (o2 + o3);
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
          const float4 b = *reinterpret_cast<const float4*>(bias_c + j);
          v[j] = fmaf(v[j], rinv, b.x);         v[j + 1] = fmaf(v[j + 1], rinv, b.y);
          v[j + 2] = fmaf(v[j + 2], rinv, b.z); v[j + 3] = fmaf(v[j + 3], rinv, b.w);
        }
        if (!A_PLANAR) {
          if (g.out_act != 0 && n + 32 > g.act_n0) {
            // (a branch on the kind inside the loops: 82 -> 137 us at K = 64, N = 128, 524 K rows)
            if (!zcols) {
#pragma unroll
              for (int j = 0; j < 32; ++j) {
                const float sg = sigmoid_f(v[j]);
                if (n + j >= g.act_n0) v[j] = g.out_act == 1 ? v[j] * sg : sg;
              }
            } else if (g.out_act == 1) {
#pragma unroll
              for (int j = 0; j < 32; ++j) v[j] = silu_f(v[j]);
            } else {
#pragma unroll
              for (int j = 0; j < 32; ++j) v[j] = sigmoid_f(v[j]);
            }
          }
          // planar: lanes are consecutive pixels, so every column is a coalesced store
          if (m < g.M) {
            float* op = g.out + ((size_t)fr * g.o_planes + g.o_plane0 + n) * g.HW + px;
            const int nw = zrow ? g.N - n : min(g.N, g.act_n0) - n;     // columns of this row to store
            if (nw >= 32) {
#pragma unroll
              for (int j = 0; j < 32; ++j) op[(size_t)j * g.HW] = v[j];
            } else {
#pragma unroll
              for (int j = 0; j < 32; ++j)
                if (j < nw) op[(size_t)j * g.HW] = v[j];
            }
          }
        } else {
          if (g.sub != nullptr && m < g.M) {
            const float4* sp = reinterpret_cast<const float4*>(g.sub + (size_t)m * g.N + n);
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
              if (n + j >= g.N) continue;
              const float4 sv = __ldg(sp + (j >> 2));
              v[j] -= sv.x; v[j + 1] -= sv.y; v[j + 2] -= sv.z; v[j + 3] -= sv.w;
            }
          }
          // 32 rows x 32 columns in the 128-byte swizzle, one TMA store per warp; rows beyond M and
          // columns beyond N are clipped by the tensor map
          if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
          __syncwarp();
#pragma unroll
          for (int j = 0; j < 32; j += 4)
            *reinterpret_cast<float4*>(my_stg + tc::sw128_offset(lane, j >> 2)) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
          tc::fence_proxy_async();
          __syncwarp();
          if (lane == 0) {
            tc::tma_store_2d(&omap, my_stg, n, m0 + quad * 32);
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          }
        }
      }
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&accempty[ac]);
      if (__any_sync(0xffffffffu, odd != odd)) {
        if (A_PLANAR) {                                 // the TMA stores of this tile go first
          if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
          asm volatile("fence.proxy.async;" ::: "memory");
          __syncwarp();
        }
        if (odd != odd && m < g.M)
          for (int cc = half; cc * 32 < q.BN; cc += 2) split_row_fma<A_PLANAR>(again, m, n0 + cc * 32, rinv);
        __syncwarp();
      }
    }
    // shared memory must outlive the last TMA stores that read it
    if (A_PLANAR && lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == GS_MMA_WARP) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem_base, tmem_cols);
  }
}

int launch_gemm_split(const GemmArgs& g, bool a_planar, cudaStream_t st) {
  if (g.M <= 0 || g.N <= 0 || g.K <= 0 || g.HW <= 0) return CSSM_ERR_DIMS;
  if (g.K % 4 != 0 || g.N % 4 != 0 || g.mul != nullptr) return CSSM_ERR_UNSUPPORTED;
  SplitGeom q;
  memset(&q, 0, sizeof(q));
  q.kblocks = (g.K + GS_BK - 1) / GS_BK;
  q.m_tiles = (g.M + GS_BM - 1) / GS_BM;
  q.hw = FastDiv(g.HW); q.w = FastDiv(g.W > 0 ? g.W : 1); q.t = FastDiv(g.T > 0 ? g.T : 1);
  q.fdiv = FastDiv(g.a_fdiv > 1 ? g.a_fdiv : 1);
  constexpr size_t LIMIT = 227 * 1024;
  // The RMS prologue's row sums; two and three K blocks ask for their room in any case: 8 KB less and the CTAs of an overlapped launch
  // find room beside those of the transforms on some SMs, and 128-column tiles of 128 channels fit (ungated block, us a pass without / with:
  // 54 x 14 x 14 x 96 32.2 / 31.1, 40 x 14 x 14 x 128 30.2 / 28.9, 120 53.3 / 51.7; one block gains without: 10 x 14 x 14 x 32 15.5 / 16.5).
  const bool sums = g.rms_scale != nullptr || q.kblocks == 2 || q.kblocks == 3;
  const size_t fixed = 1024 + 1024 + 128 + (a_planar ? 8 * 4096 + (sums ? GS_SS * 1024 : 0) : 0);   // slack, bias, barriers, staging, sums
  if (g.wsplit != nullptr && (g.rms_scale != nullptr || g.gate != nullptr || !aligned16(g.wsplit))) return CSSM_ERR_UNSUPPORTED;
  auto round32 = [](int v) { return (v + 31) / 32 * 32; };
  auto res_size = [&](int bn) { return (size_t)q.kblocks * 3 * bn * 128; };
  // Weights resident when a tile of at least 64 columns (or all of N) leaves room for two A stages:
  // every CTA then splits its weights once.  Otherwise 128-column tiles with the weights streamed.
  // The leading accumulators and the one of the small products of a tile share the 512 columns of TMEM.
  q.nl = q.kblocks > 1 ? 1 : 0;
  q.lead = q.kblocks;
  if (q.kblocks > 6) {
    const int most = (int)(2.0 * sqrt((double)q.kblocks)) > 6 ? (int)(2.0 * sqrt((double)q.kblocks)) : 6;
    q.nl = (q.kblocks + most - 1) / most;
    if (q.nl > 15) q.nl = 15;
    q.lead = (q.kblocks + q.nl - 1) / q.nl;
  }
  const bool wide = q.nl > 1;
  const int bn_tmem = 512 / (1 + q.nl) / 32 * 32;
  // Planar A, weights split by the producers: tiles of 96 or 128 columns, by rounds over the SMs, a tile of bn columns taking as long
  // as bn + 30 of them.  us a pass of the ungated block, K = N, 96- / 128-column tiles: 384 channels, 5880 rows 83 / 64, 13916
  // 135 / 151, 29988 313 / 295; 448 channels, 20972 288 / 300, 55860 689 / 697; 512 channels, 5880 105 / 119, 13916 245 / 206.
  const int sms = sm_count();
  auto rounds = [&](int bn) { return (((long long)q.m_tiles * ((g.N + bn - 1) / bn) + sms - 1) / sms) * (bn + 30); };
  int nt = q.nl > 0 ? (g.N + 127) / 128 : (g.N + 255) / 256;
  while (round32((g.N + nt - 1) / nt) > 32 && res_size(round32((g.N + nt - 1) / nt)) + 2 * GS_A_BYTES + fixed > LIMIT) ++nt;
  q.BN = round32((g.N + nt - 1) / nt);
  const bool res = !wide && g.wsplit == nullptr && (q.BN >= 64 || nt == 1) && res_size(q.BN) + 2 * GS_A_BYTES + fixed <= LIMIT;
  if (!res) {
    // (the row sums of the RMS prologue leave no room for two stages of 128 columns)
    auto width = [&](int most) {
      most = most < bn_tmem ? most : bn_tmem;
      const int n = (g.N + most - 1) / most;
      return round32((g.N + n - 1) / n);
    };
    q.BN = width(g.rms_scale != nullptr ? 96 : 128);
    if (a_planar && g.wsplit == nullptr && rounds(width(96)) < rounds(q.BN)) q.BN = width(96);
    nt = (g.N + q.BN - 1) / q.BN;
  }
  cudaError_t e;
  // few row tiles: narrower column tiles until two thirds of the SMs have one (each CTA then splits
  // fewer weights too; the row tile is split once more per column tile, which idle SMs do for free)
  for (int k = nt + 1; q.BN > 32 && q.m_tiles * ((g.N + q.BN - 1) / q.BN) * 3 < sms * 2; ++k)
    q.BN = round32((g.N + k - 1) / k);
  q.n_tiles = (g.N + q.BN - 1) / q.BN;
  q.bufs = 2 * (1 + q.nl) * q.BN <= 512 ? 2 : 1;
  const size_t stage = GS_A_BYTES + (res ? 0 : (size_t)3 * q.BN * 128);
  const size_t base = (res ? res_size(q.BN) : 0) + fixed;
  q.stages = 4;
  while (q.stages > 1 && base + q.stages * stage > LIMIT) --q.stages;
  if (base + q.stages * stage > LIMIT) return CSSM_ERR_UNSUPPORTED;
  const size_t smem = base + q.stages * stage;
  const long long tiles = (long long)q.m_tiles * q.n_tiles;
  if (tiles > 0x7fffffffLL) return CSSM_ERR_DIMS;
  // a multiple of n_tiles, so that a CTA keeps one N tile (resident weights, bias)
  int grid = (int)(tiles < sms ? tiles : sms);
  if (res && grid > q.n_tiles) grid -= grid % q.n_tiles;
  if (res && grid < q.n_tiles) return CSSM_ERR_UNSUPPORTED;
  CUtensorMap map;
  memset(&map, 0, sizeof(map));
  if (a_planar) {
    const tc::EncodeTiledFn enc = tc::encode_fn();
    const cuuint64_t dims[2] = {(cuuint64_t)g.N, (cuuint64_t)g.M}, strides[1] = {(cuuint64_t)g.N * 4};
    const cuuint32_t box[2] = {32, 32}, es[2] = {1, 1};
    if (enc == nullptr ||
        enc(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, g.out, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return CSSM_ERR_CUDA;
  }
  const bool gate = g.gate != nullptr;
  auto kern = a_planar ? (gate ? (res ? gemm_split_kernel<true, true, true, false> : gemm_split_kernel<true, false, true, false>)
                               : (res ? gemm_split_kernel<true, true, false, false> : gemm_split_kernel<true, false, false, false>))
                       : (res ? gemm_split_kernel<false, true, false, false> : gemm_split_kernel<false, false, false, false>);
  if (wide)
    kern = a_planar ? (gate ? gemm_split_kernel<true, false, true, true> : gemm_split_kernel<true, false, false, true>)
                    : gemm_split_kernel<false, false, false, true>;
  if (g.wsplit != nullptr && !a_planar)
    kern = wide ? gemm_split_kernel<false, false, false, true, true> : gemm_split_kernel<false, false, false, false, true>;
  e = func_smem(kern, smem);
  if (e != cudaSuccess) { set_cuda_error(e); return CSSM_ERR_CUDA; }
  launch_k(kern, grid, GS_THREADS, smem, st, g, q, map, SplitArgs{g, q});
  return check_launch();
}

int read_split_error(int* out, int clear) {
  cudaError_t e = cudaMemcpyFromSymbol(out, g_split_error, sizeof(int));
  if (e == cudaSuccess && clear && *out != 0) {
    const int zero = 0;
    e = cudaMemcpyToSymbol(g_split_error, &zero, sizeof(int));
  }
  if (e != cudaSuccess) { set_cuda_error(e); return CSSM_ERR_CUDA; }
  return CSSM_OK;
}

}  // namespace cssm
