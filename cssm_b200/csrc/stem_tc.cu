// Second and later stem layers (3x3 'SAME' conv of C to C channels, softplus, LayerNorm, 2x2 max-pool) on the tensor cores,
// C = 32 or 64: an implicit GEMM in float32-equivalent precision, three bfloat16 parts a value and six partial products as
// in csrc/gemm_split.cu.
//
// A CTA (eight warps, two CTAs per SM) makes one tile of 16 x 8 conv pixels:
//   all warps   read the 18 x 10 input pixels (zero outside the image), split them once and write the parts as
//               [16-byte channel chunk][pixel], the K-major layout without swizzle: eight neighbouring pixels are one
//               core matrix, so a tap of the window is the same operand 16 bytes (a column) or 160 bytes (a row) further
//               on, and no tap is copied;
//   warp 1      streams the split weights (stem_split_weights) through a ring, 32 channels of one tap a stage (bulk copies);
//   warp 0      issues the MMAs, M = 128: A0 B0 into one of two leading accumulators (taps 0-4, 5-8), A0 [B1 B2],
//               A1 [B0 B1] and A2 B0 into two accumulators of small products next to one another;
//   warps 0-3   lane = pixel: sum of the accumulators, bias, softplus, LayerNorm of the lane's own C values, then the
//               maximum over the window, the lanes of a window keeping a quarter of the channels each.
// Bound: the MMAs' operand reads (per 16 k: four A tiles of 4 KB and 384 weight rows of 32 bytes, about 224 clocks) and the
// chain load -> split -> 36 k steps -> epilogue of one tile.  A lane owning two channels of eight pixels on the FMA pipes
// (the kernel before) read a weight for every eight FMAs.
#include <string.h>
#include "kernels.cuh"
#include "bf16_ops.cuh"
#include "tc05.cuh"
#include "stem.cuh"

namespace cssm {

__device__ int g_stem_error = 0;

constexpr int ST_THREADS = 256, ST_TW = 8, ST_TH = 16, ST_PW = ST_TW + 2, ST_PH = ST_TH + 2;
constexpr int ST_PIX = ST_PW * ST_PH + 1;      // rows of a chunk; odd: a warp's stores of eight chunks meet no bank conflict
constexpr int ST_RING = 3;

template <int C>
struct StemTc {
  static constexpr int CH = C / 8, STAGES = 9 * (C / 32);
  static constexpr uint32_t STAGE_BYTES = 4u * 3u * C * 16u, PART = (uint32_t)CH * ST_PIX * 16u;
  static constexpr uint32_t RING_OFF = 0, A_OFF = ST_RING * STAGE_BYTES, VEC_OFF = A_OFF + 3u * PART;
  static constexpr uint32_t BAR_OFF = VEC_OFF + 3u * C * 4u, TOTAL = BAR_OFF + 128u;
  static constexpr uint32_t TMEM = 4u * C;     // leading 0, leading 1, small, small
};

// x -> three bf16 parts for a pair of values, packed (low half = first value)
__device__ __forceinline__ void stem_split3(float x, float y, uint32_t& p0, uint32_t& p1, uint32_t& p2) {
  p0 = float2_to_bf16x2(x, y);
  const cf r = mk(x, y) - mk(__uint_as_float(p0 << 16), __uint_as_float(p0 & 0xffff0000u));
  p1 = float2_to_bf16x2(r.x, r.y);
  const cf u = r - mk(__uint_as_float(p1 << 16), __uint_as_float(p1 & 0xffff0000u));
  p2 = float2_to_bf16x2(u.x, u.y);
}
__device__ __forceinline__ void stem_split8(const float (&v)[8], uint4& a, uint4& b, uint4& c) {
  stem_split3(v[0], v[1], a.x, b.x, c.x);
  stem_split3(v[2], v[3], a.y, b.y, c.y);
  stem_split3(v[4], v[5], a.z, b.z, c.z);
  stem_split3(v[6], v[7], a.w, b.w, c.w);
}

// weights (3,3,C,C) -> [tap][32-channel half][8-channel chunk 0..3][part][n] of 16 bytes
__global__ void __launch_bounds__(128) stem_split_weights(const float* __restrict__ wk, uint4* __restrict__ out, int C) {
  pdl_sync();
  const int item = blockIdx.x * 128 + threadIdx.x, n = item % C, kc = item / C;      // kc: 8-k chunk over all taps
  if (kc >= 9 * (C / 8)) return;
  float v[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) v[e] = __ldg(wk + (size_t)(kc * 8 + e) * C + n);
  uint4 a, b, c;
  stem_split8(v, a, b, c);
  uint4* o = out + (size_t)kc * 3 * C + n;
  o[0] = a; o[C] = b; o[2 * C] = c;
}

// K-major operand without swizzle: core matrices of 8 rows x 16 bytes, `lbo` bytes apart along K, `sbo` along M / N
__device__ __forceinline__ uint64_t desc_k(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) | ((uint64_t)1 << 46);
}
__device__ __forceinline__ void stem_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ uint32_t stem_idesc(uint32_t M, uint32_t N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((N >> 3) << 17) | ((M >> 4) << 24);
}

// One conv output by float32 FMAs: where the partial products are not finite (an input or weight above the largest
// bfloat16 has no finite parts)
__device__ __noinline__ float stem_conv_fma(const StemArgs& a, int n, int h, int w, int c) {
  float v = a.bk[c];
  for (int tap = 0; tap < 9; ++tap) {
    const int hh = h + tap / 3 - 1, ww = w + tap % 3 - 1;
    if (hh < 0 || hh >= a.Hin || ww < 0 || ww >= a.Win) continue;
    const float* xp = a.x + (((size_t)n * a.Hin + hh) * a.Win + ww) * a.Cin;
    const float* wp = a.wk + (size_t)tap * a.Cin * a.C + c;
    for (int k = 0; k < a.Cin; ++k) v = fmaf(xp[k], wp[(size_t)k * a.C], v);
  }
  return v;
}

template <int C>
__global__ void __launch_bounds__(ST_THREADS, 2)
stem_layer_tc_kernel(const __grid_constant__ StemArgs a, const unsigned char* __restrict__ wsplit, int tiles_x, int tiles_y) {
  using L = StemTc<C>;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ int s_bad;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  float* vec = reinterpret_cast<float*>(smem + L::VEC_OFF);               // bias, scale, lnbias
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + L::BAR_OFF);
  uint64_t* empty = full + ST_RING;
  uint64_t* accfull = empty + ST_RING;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(accfull + 1);
  if (tid == 0) {
    for (int s = 0; s < ST_RING; ++s) { tc::mbar_init(&full[s], 1); tc::mbar_init(&empty[s], 1); }
    tc::mbar_init(accfull, 1);
    tc::fence_mbar_init();
    s_bad = 0;
  }
  if (warp == 0) {
    tc::tmem_alloc(tmem_slot, L::TMEM);
    tc::tmem_relinquish();
  }
  for (int i = tid; i < C; i += ST_THREADS) { vec[i] = a.bk[i]; vec[C + i] = a.scale[i]; vec[2 * C + i] = a.bias[i]; }
  const int tx = blockIdx.x % tiles_x, ty = (blockIdx.x / tiles_x) % tiles_y, n = blockIdx.x / (tiles_x * tiles_y);
  const int x0 = tx * ST_TW, y0 = ty * ST_TH;
  __syncthreads();
  pdl_sync();
  const uint32_t sbase = tc::smem_u32(smem);
  auto load_stage = [&](int st) {
    tc::mbar_expect_tx(&full[st % ST_RING], L::STAGE_BYTES);
    tc::bulk_g2s(smem + L::RING_OFF + (st % ST_RING) * L::STAGE_BYTES, wsplit + (size_t)st * L::STAGE_BYTES, L::STAGE_BYTES,
                 &full[st % ST_RING]);
  };
  if (warp == 1 && lane == 0)
    for (int st = 0; st < ST_RING; ++st) load_stage(st);

  // ---- input pixels -> three bf16 parts ----
  constexpr int ITEMS = ST_PW * ST_PH * L::CH, BATCH = 3;
  for (int i0 = tid; i0 < ITEMS; i0 += BATCH * ST_THREADS) {
    float v[BATCH][8];
#pragma unroll
    for (int u = 0; u < BATCH; ++u) {
      const int i = i0 + u * ST_THREADS, c = i % L::CH, px = i / L::CH, hh = y0 - 1 + px / ST_PW, ww = x0 - 1 + px % ST_PW;
      float4 p = make_float4(0.f, 0.f, 0.f, 0.f), r = p;
      if (i < ITEMS && hh >= 0 && hh < a.Hin && ww >= 0 && ww < a.Win) {
        const float4* xp = reinterpret_cast<const float4*>(a.x + (((size_t)n * a.Hin + hh) * a.Win + ww) * C) + 2 * c;
        p = __ldg(xp); r = __ldg(xp + 1);
      }
      v[u][0] = p.x; v[u][1] = p.y; v[u][2] = p.z; v[u][3] = p.w; v[u][4] = r.x; v[u][5] = r.y; v[u][6] = r.z; v[u][7] = r.w;
    }
#pragma unroll
    for (int u = 0; u < BATCH; ++u) {
      const int i = i0 + u * ST_THREADS;
      if (i < ITEMS) {
        uint4 p0, p1, p2;
        stem_split8(v[u], p0, p1, p2);
        unsigned char* d = smem + L::A_OFF + ((uint32_t)(i % L::CH) * ST_PIX + i / L::CH) * 16u;
        *reinterpret_cast<uint4*>(d) = p0;
        *reinterpret_cast<uint4*>(d + L::PART) = p1;
        *reinterpret_cast<uint4*>(d + 2 * L::PART) = p2;
      }
    }
  }
  tc::fence_proxy_async();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = *tmem_slot;

  if (warp == 1 && lane == 0) {
    for (int st = ST_RING; st < L::STAGES; ++st) {
      if (!tc::mbar_wait(&empty[st % ST_RING], ((st / ST_RING) & 1) ^ 1)) { atomicExch(&g_stem_error, 1); s_bad = 1; break; }
      load_stage(st);
    }
  }
  if (warp == 0) {
    // the whole warp walks the loop, one lane issues (elect_one)
    constexpr uint32_t ALBO = ST_PIX * 16u, ASBO = ST_PW * 16u, BLBO = 3u * C * 16u;
    const uint32_t id1 = stem_idesc(128, C), id2 = stem_idesc(128, 2 * C);
    for (int st = 0; st < L::STAGES; ++st) {
      if (__any_sync(0xffffffffu, !tc::mbar_wait_spin(&full[st % ST_RING], (st / ST_RING) & 1))) { atomicExch(&g_stem_error, 2); s_bad = 1; break; }
      tc::fence_after_sync();
      const int tap = st / (C / 32), half = st % (C / 32);
      const uint32_t bs = sbase + L::RING_OFF + (st % ST_RING) * L::STAGE_BYTES;
      const uint32_t as = sbase + L::A_OFF + (uint32_t)(half * 4 * ST_PIX + (tap / 3) * ST_PW + tap % 3) * 16u;
      const uint32_t lead = tmem + (tap < 5 ? 0u : (uint32_t)C), small = tmem + 2u * C;
      const bool first_lead = half == 0 && (tap == 0 || tap == 5);
      if (tc::elect_one()) {
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) {
          const uint32_t ak = as + 2u * ks * ALBO, bk = bs + 2u * ks * BLBO;
          const uint64_t a0 = desc_k(ak, ALBO, ASBO), a1 = desc_k(ak + L::PART, ALBO, ASBO), a2 = desc_k(ak + 2 * L::PART, ALBO, ASBO);
          const uint64_t b0 = desc_k(bk, BLBO, 128), b1 = desc_k(bk + C * 16u, BLBO, 128);
          stem_mma(lead, a0, b0, id1, !(first_lead && ks == 0));
          stem_mma(small, a0, b1, id2, !(st == 0 && ks == 0));       // [01 02]
          stem_mma(small, a1, b0, id2, 1);                           // [10 11]
          stem_mma(small, a2, b0, id1, 1);                           // [20]
        }
        tc::commit(&empty[st % ST_RING]);
      }
      __syncwarp();
    }
    if (tc::elect_one()) tc::commit(accfull);
    __syncwarp();
  }
  __syncwarp();

  // ---- epilogue: lane = pixel, warps 0-3 ----
  if (warp < 4) {
    const bool ok = !__any_sync(0xffffffffu, !tc::mbar_wait(accfull, 0));
    if (!ok) { atomicExch(&g_stem_error, 3); s_bad = 1; }
    tc::fence_after_sync();
    const int h = y0 + warp * 4 + (lane >> 3), w = x0 + (lane & 7);
    const uint32_t t0 = tmem + ((uint32_t)(warp * 32) << 16);
    float v[C];
#pragma unroll
    for (int c = 0; c < C; c += 16) {
      uint32_t r[16], s[16];
      tc::ld_32x32b_x16(t0 + c, r);
      tc::ld_32x32b_x16(t0 + C + c, s);
      tc::wait_ld();
#pragma unroll
      for (int j = 0; j < 16; ++j) v[c + j] = __uint_as_float(r[j]) + __uint_as_float(s[j]);
      tc::ld_32x32b_x16(t0 + 2 * C + c, r);
      tc::ld_32x32b_x16(t0 + 3 * C + c, s);
      tc::wait_ld();
#pragma unroll
      for (int j = 0; j < 16; ++j) v[c + j] = (v[c + j] + (__uint_as_float(r[j]) + __uint_as_float(s[j]))) + vec[c + j];
    }
    const bool inb = h < a.Hin && w < a.Win;                       // else 'SAME' pool padding on odd sizes
    float z = 0.f;
#pragma unroll
    for (int c = 0; c < C; ++c) z = fmaf(v[c], 0.f, z);
    if (inb && !(z == 0.f)) {
#pragma unroll
      for (int c = 0; c < C; ++c) v[c] = stem_conv_fma(a, n, h, w, c);
    }
    // softplus, LayerNorm (moments of the values minus the pixel's first channel)
    float s = 0.f, ss = 0.f;
    const float vref = softplus_f(v[0]);
#pragma unroll
    for (int c = 0; c < C; ++c) {
      v[c] = softplus_f(v[c]) - vref;
      s += v[c]; ss = fmaf(v[c], v[c], ss);
    }
    const float mean = s / (float)C, rinv = rsqrtf(fmaxf(ss / (float)C - mean * mean, 0.f) + 1e-6f);
#pragma unroll
    for (int c = 0; c < C; ++c) v[c] = inb ? (v[c] - mean) * rinv * vec[C + c] + vec[2 * C + c] : -INFINITY;
    // 2x2 maximum: columns are lanes xor 1, rows lanes xor 8; each exchange leaves a lane half of its channels
    const int odd = lane & 1, low = (lane >> 3) & 1;
    float u[C / 2], q[C / 4];
#pragma unroll
    for (int j = 0; j < C / 2; ++j) {
      const float got = __shfl_xor_sync(0xffffffffu, odd ? v[j] : v[C / 2 + j], 1);
      u[j] = fmaxf(odd ? v[C / 2 + j] : v[j], got);
    }
#pragma unroll
    for (int j = 0; j < C / 4; ++j) {
      const float got = __shfl_xor_sync(0xffffffffu, low ? u[j] : u[C / 4 + j], 8);
      q[j] = fmaxf(low ? u[C / 4 + j] : u[j], got);
    }
    const int ho = h >> 1, wo = w >> 1;
    if (ok && !*reinterpret_cast<volatile int*>(&s_bad) && ho < a.Ho && wo < a.Wo) {
      float4* o = reinterpret_cast<float4*>(a.out + (((size_t)n * a.Ho + ho) * a.Wo + wo) * C + odd * (C / 2) + low * (C / 4));
#pragma unroll
      for (int j = 0; j < C / 4; j += 4) o[j / 4] = make_float4(q[j], q[j + 1], q[j + 2], q[j + 3]);
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  // error path only: weight copies that may still be in flight get a bounded time (~1 ms) to land
  if (s_bad)
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
  if (warp == 0) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem, L::TMEM);
  }
}

size_t stem_tc_scratch_bytes(int C) { return (size_t)9 * C * C * 6; }

bool stem_tc_supported(const StemArgs& a) {
  return a.Cin == a.C && (a.C == 32 || a.C == 64) && aligned16(a.x) && aligned16(a.out) &&
         (long long)a.N * ((a.Hin + ST_TH - 1) / ST_TH) * ((a.Win + ST_TW - 1) / ST_TW) < (1LL << 31);
}

int launch_stem_split_weights(const float* wk, void* scratch, int C, cudaStream_t st) {
  launch_k(stem_split_weights, (9 * (C / 8) * C + 127) / 128, 128, 0, st, wk, (uint4*)scratch, C);
  return check_launch();
}

template <int C>
static int launch_v(const StemArgs& a, const void* scratch, cudaStream_t st) {
  const int tx = (a.Win + ST_TW - 1) / ST_TW, ty = (a.Hin + ST_TH - 1) / ST_TH;
  const cudaError_t e = func_smem(stem_layer_tc_kernel<C>, StemTc<C>::TOTAL);
  if (e != cudaSuccess) { set_cuda_error(e); return CSSM_ERR_CUDA; }
  launch_k(stem_layer_tc_kernel<C>, (unsigned)(a.N * tx * ty), ST_THREADS, StemTc<C>::TOTAL, st, a, (const unsigned char*)scratch, tx, ty);
  return check_launch();
}

int launch_stem_layer_tc(const StemArgs& a, const void* scratch, cudaStream_t st) {
  if (!stem_tc_supported(a) || !aligned16(scratch)) return CSSM_ERR_UNSUPPORTED;
  return a.C == 64 ? launch_v<64>(a, scratch, st) : launch_v<32>(a, scratch, st);
}

int read_stem_error(int* out, int clear) {
  cudaError_t e = cudaMemcpyFromSymbol(out, g_stem_error, sizeof(int));
  if (e == cudaSuccess && clear && *out != 0) {
    const int zero = 0;
    e = cudaMemcpyToSymbol(g_stem_error, &zero, sizeof(int));
  }
  if (e != cudaSuccess) { set_cuda_error(e); return CSSM_ERR_CUDA; }
  return CSSM_OK;
}

}  // namespace cssm
