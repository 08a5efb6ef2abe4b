// q, k, v projection of the GDN block at 64 channels with the causal temporal conv, SiLU and input gates behind it: the conv's
// history stays in TMEM.
//
//   out[b, t, n, px] = silu(b_t[n] + sum_j w_j[n] s[b, t - 3 + j, n, px]) * gate,   s = A W + bias (frames before 0: nothing)
//
// The tcgen05 GEMM of csrc/gemm_tc.cu (3 x TF32, producers / MMA warp / epilogue) with another order of the tiles: a CTA takes 128
// pixels and half of the 192 columns through t = 0 .. T - 1.  Its accumulators, 96 columns each, are a ring of five in
// TMEM: the epilogue of step t reads those of t - 3 .. t, while the MMAs of t + 1 fill the fifth.  So the projected planes
// never go to memory and back for the conv (6.4 GB of 128 x 8 x 64 x 64 x 64).  The price is that each tile of A is split
// twice, once for either half of the columns (all 192 would need 768 columns of TMEM for the history).
#include "kernels.cuh"
#include "gemm.cuh"
#include "tc05.cuh"

namespace cssm {

__device__ int g_qt_error = 0;

constexpr int QT_THREADS = 544, QT_MMA_WARP = 8, QT_N = 96, QT_RING = 5, QT_BM = 128;
constexpr uint32_t QT_A_HALF = 2u * QT_BM * 128u, QT_B_HALF = 2u * QT_N * 128u;
constexpr uint32_t QT_A_OFF = 2u * QT_B_HALF, QT_TAB_OFF = QT_A_OFF + 4u * QT_A_HALF;      // two stages of hi, lo
constexpr uint32_t QT_BAR_OFF = QT_TAB_OFF + 8u * QT_N * 4u, QT_SMEM = QT_BAR_OFF + 128u;   // tables: w[4][96], constants[4][96]
static_assert(QT_SMEM + 1024 <= 227 * 1024, "one CTA per SM");

struct QkvTconvGemmArgs {
  GemmArgs g;                                   // M, HW, A, source frames, RoPE, Wk (64, 192), bias, out (3C planes a frame), T
  const float* wt[3]; const float* bt[3]; int kt;
  const float2* bkv;                            // (frames, HW) {B_k, B_v} or nullptr
  int seqs;                                     // 2 * clips * HW / 128
};

__global__ void __launch_bounds__(QT_THREADS, 1) gemm_qkv_tconv_kernel(const __grid_constant__ QkvTconvGemmArgs a) {
  const GemmArgs& g = a.g;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned char* smem = smem_raw + ((1024u - (tc::smem_u32(smem_raw) & 1023u)) & 1023u);
  const uint32_t sbase = tc::smem_u32(smem);
  float* wtab = reinterpret_cast<float*>(smem + QT_TAB_OFF);      // [tap][column], tap 3 = the current frame
  float* ctab = wtab + 4 * QT_N;                                  // [min(t, 3)][column]: b_t + bias * sum of the taps in use
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + QT_BAR_OFF);
  uint64_t* full = bars;          // [2] A stage written (8 warps)
  uint64_t* empty = bars + 2;     // [2] A stage consumed
  uint64_t* accfull = bars + 4;   // [2] accumulator of step n, n & 1
  uint64_t* accempty = bars + 6;  // [2] epilogue of step n is through (8 warps)
  uint64_t* done = bars + 8;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 9);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int half = blockIdx.x & 1, n0 = half * QT_N;              // the grid is even: a CTA keeps its half of the columns

  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      tc::mbar_init(&full[i], 8); tc::mbar_init(&empty[i], 1);
      tc::mbar_init(&accfull[i], 1); tc::mbar_init(&accempty[i], 8);
    }
    tc::mbar_init(done, 1);
    tc::fence_mbar_init();
  }
  if (warp == QT_MMA_WARP) {
    tc::tmem_alloc(tmem_slot, 512);
    tc::tmem_relinquish();
  }
  for (int item = tid; item < QT_N * 16; item += QT_THREADS) {
    const int n = item % QT_N, c = item / QT_N;                   // c: 16-byte chunk of 4 k values
    float hi[4], lo[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) tc::split_tf32(g.Wk[(size_t)(4 * c + e) * 192 + n0 + n], hi[e], lo[e]);
    const uint32_t off = (uint32_t)(c >> 3) * (QT_N * 128u) + tc::sw128_offset(n, c & 7);
    *reinterpret_cast<float4*>(smem + off) = make_float4(hi[0], hi[1], hi[2], hi[3]);
    *reinterpret_cast<float4*>(smem + QT_B_HALF + off) = make_float4(lo[0], lo[1], lo[2], lo[3]);
  }
  for (int n = tid; n < QT_N; n += QT_THREADS) {
    const int grp = (n0 + n) >> 6, c = (n0 + n) & 63;
    const float* wp = grp == 0 ? a.wt[0] : grp == 1 ? a.wt[1] : a.wt[2];
    const float bt = (grp == 0 ? a.bt[0] : grp == 1 ? a.bt[1] : a.bt[2])[c], b = g.bias[n0 + n];
    float sum = 0.f;
    for (int j = 3; j >= 0; --j) {                                // newest first; fewer taps than four: zeros before them
      const int i = j - (4 - a.kt);
      const float w = i >= 0 ? wp[(size_t)i * 64 + c] : 0.f;
      wtab[j * QT_N + n] = w;
      sum += w;
      ctab[(3 - j) * QT_N + n] = fmaf(b, sum, bt);
    }
  }
  tc::fence_proxy_async();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  pdl_sync();

  const int blocks = g.HW / QT_BM, T = g.T;                       // pixel blocks of a frame
  // source frame of frame f, pixel block of sequence s
  auto src_frame = [&](int f) { return g.a_fmul == 0 && g.a_fadd == 0 ? f : (g.a_fdiv > 1 ? f / g.a_fdiv : f) * g.a_fmul + g.a_fadd; };

  if (warp < 8) {
    // ================================ producers ================================
    // item r: chunk (tid & 7) + 8 (r >> 2) of row (tid >> 3) + 32 (r & 3), as in gemm_tc_kernel; `pre` holds the next step's tile
    float4 pre[8];
    const int chunk = tid & 7, rsub = tid >> 3;
    const uint32_t dst0 = tc::sw128_offset(rsub, chunk);
    bool rot[2] = {false, false};
    if (g.rope_t != nullptr)
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        const int pi = 2 * (chunk + 8 * hf);
        rot[hf] = g.rope_nz == nullptr || g.rope_nz[pi] != 0.f || g.rope_nz[pi + 1] != 0.f;
      }
    const float invW = 1.0f / (float)g.W;
    auto fetch = [&](int s, int t) {
      const int pb = s >> 1, b = pb / blocks, px0 = (pb - b * blocks) * QT_BM;
      const float* a0 = g.A + ((size_t)src_frame(b * T + t) * g.HW + px0 + rsub) * 64 + chunk * 4;
#pragma unroll
      for (int r = 0; r < 8; ++r) pre[r] = __ldg(reinterpret_cast<const float4*>(a0 + (size_t)(r & 3) * 32 * 64 + (r >> 2) * 32));
    };
    int it = 0;
    bool ok = true;
    if ((int)blockIdx.x < a.seqs) fetch(blockIdx.x, 0);
    for (int s = blockIdx.x; s < a.seqs && ok; s += gridDim.x) {
      const int pb = s >> 1, px0 = (pb - pb / blocks * blocks) * QT_BM;
      for (int t = 0; t < T; ++t, ++it) {
        const int st = it & 1;
        float4 cur[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) cur[r] = pre[r];
        if (t + 1 < T) fetch(s, t + 1);
        else if (s + (int)gridDim.x < a.seqs) fetch(s + gridDim.x, 0);
        if (__any_sync(0xffffffffu, !tc::mbar_wait(&empty[st], ((it >> 1) & 1) ^ 1))) { atomicExch(&g_qt_error, 1); ok = false; break; }
        unsigned char* a_hi = smem + QT_A_OFF + (uint32_t)st * 2u * QT_A_HALF + dst0;
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          float4 v = cur[r];
          if (rot[r >> 2]) {
            const int px = px0 + rsub + 32 * (r & 3), pi = 2 * (chunk + 8 * (r >> 2));
            const int h = (int)(((float)px + 0.5f) * invW), w = px - h * g.W;             // exact for px < 2^22
            const float4 ct = __ldg(reinterpret_cast<const float4*>(g.rope_t + t * 32 + pi));
            const float4 ch = __ldg(reinterpret_cast<const float4*>(g.rope_h + h * 32 + pi));
            const float4 cw = __ldg(reinterpret_cast<const float4*>(g.rope_w + w * 32 + pi));
            auto turn = [](float tx, float ty, float hx, float hy, float wx, float wy, float& x, float& y) {
              const float cx = tx * hx - ty * hy, sx = tx * hy + ty * hx;
              const float c2 = cx * wx - sx * wy, s2 = cx * wy + sx * wx;
              const float ne = x * c2 - y * s2, no = x * s2 + y * c2;
              x = ne; y = no;
            };
            turn(ct.x, ct.y, ch.x, ch.y, cw.x, cw.y, v.x, v.y);
            turn(ct.z, ct.w, ch.z, ch.w, cw.z, cw.w, v.z, v.w);
          }
          float4 h4, l4;
          tc::split_tf32(v.x, h4.x, l4.x); tc::split_tf32(v.y, h4.y, l4.y);
          tc::split_tf32(v.z, h4.z, l4.z); tc::split_tf32(v.w, h4.w, l4.w);
          unsigned char* d = a_hi + (r & 3) * 4096 + (r >> 2) * (QT_BM * 128);            // 32 rows = 4096 bytes on
          *reinterpret_cast<float4*>(d) = h4;
          *reinterpret_cast<float4*>(d + QT_A_HALF) = l4;
        }
        tc::fence_proxy_async();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&full[st]);
      }
    }
  } else if (warp == QT_MMA_WARP) {
    // ================================ MMA issuer ================================
    // The whole warp walks the loop, one lane issues (elect_one).
    const uint32_t idesc = tc::make_idesc_tf32(QT_BM, QT_N);
    const int mine = a.seqs > (int)blockIdx.x ? (a.seqs - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x * T : 0;
    bool ok = true;
    int slot = 0;
    for (int n = 0; n < mine; ++n) {
      // the accumulator of step n - 5 was last read by the epilogue of step n - 2
      if (__any_sync(0xffffffffu, !tc::mbar_wait(&accempty[n & 1], ((n >> 1) & 1) ^ 1) || !tc::mbar_wait(&full[n & 1], (n >> 1) & 1))) {
        atomicExch(&g_qt_error, 2); ok = false; break;
      }
      tc::fence_after_sync();
      const uint32_t a_hi = sbase + QT_A_OFF + (uint32_t)(n & 1) * 2u * QT_A_HALF, a_lo = a_hi + QT_A_HALF;
      const uint32_t d = tmem_base + (uint32_t)slot * QT_N;
      if (++slot == QT_RING) slot = 0;
      if (tc::elect_one()) {
#pragma unroll
        for (int pass = 0; pass < 3; ++pass) {
          const uint64_t ad = tc::make_desc_sw128(pass == 1 ? a_lo : a_hi), bd = tc::make_desc_sw128(pass == 2 ? sbase + QT_B_HALF : sbase);
#pragma unroll
          for (int ks = 0; ks < 8; ++ks)
            tc::mma_tf32(d, ad + (ks >> 2) * (QT_BM * 128u >> 4) + (ks & 3) * 2, bd + (ks >> 2) * (QT_N * 128u >> 4) + (ks & 3) * 2, idesc, (pass | ks) ? 1u : 0u);
        }
        tc::commit(&empty[n & 1]);
        tc::commit(&accfull[n & 1]);
      }
      __syncwarp();
    }
    // nothing of this warp's tensor work may be in flight when TMEM is freed
    if (tc::elect_one()) tc::commit(done);
    __syncwarp();
    if (!tc::mbar_wait(done, 0) && ok) atomicExch(&g_qt_error, 3);
    __syncwarp();
  } else {
    // ================================ epilogue ================================
    const int q = warp & 3, part = (warp - (QT_MMA_WARP + 1)) >> 2;          // TMEM lane quadrant; 48 of the 96 columns
    const uint32_t tlane = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)part * 48u;
    int n = 0, slot = 0;
    bool ok = true;
    for (int s = blockIdx.x; s < a.seqs && ok; s += gridDim.x) {
      const int pb = s >> 1, b = pb / blocks, px = (pb - b * blocks) * QT_BM + q * 32 + lane;
      for (int t = 0; t < T; ++t, ++n) {
        const size_t frame = (size_t)b * T + t;
        const float2 gv = a.bkv != nullptr ? __ldg(a.bkv + frame * g.HW + px) : make_float2(1.f, 1.f);
        if (__any_sync(0xffffffffu, !tc::mbar_wait(&accfull[n & 1], (n >> 1) & 1))) { atomicExch(&g_qt_error, 4); ok = false; break; }
        tc::fence_after_sync();
        // earlier frames of this clip under the taps (frames further back may hold anything: no product with a zero tap)
        const int back = t < a.kt - 1 ? t : a.kt - 1;
        uint32_t sl[4];                                                     // ring slots of t, t - 1, t - 2, t - 3
#pragma unroll
        for (int d = 0; d < 4; ++d) sl[d] = (uint32_t)(slot >= d ? slot - d : slot - d + QT_RING) * QT_N;
        if (++slot == QT_RING) slot = 0;
#pragma unroll 1
        for (int pc = 0; pc < 3; ++pc) {
          const int c0 = part * 48 + pc * 16;
          float v[16];
#pragma unroll
          for (int j = 0; j < 16; j += 4) {
            const float4 c = *reinterpret_cast<const float4*>(ctab + back * QT_N + c0 + j);
            v[j] = c.x; v[j + 1] = c.y; v[j + 2] = c.z; v[j + 3] = c.w;
          }
          auto tap = [&](const uint32_t (&r)[16], int d) {
#pragma unroll
            for (int j = 0; j < 16; j += 4) {
              const float4 w = *reinterpret_cast<const float4*>(wtab + (3 - d) * QT_N + c0 + j);
              v[j] = fmaf(w.x, __uint_as_float(r[j]), v[j]);             v[j + 1] = fmaf(w.y, __uint_as_float(r[j + 1]), v[j + 1]);
              v[j + 2] = fmaf(w.z, __uint_as_float(r[j + 2]), v[j + 2]); v[j + 3] = fmaf(w.w, __uint_as_float(r[j + 3]), v[j + 3]);
            }
          };
          uint32_t r0[16], r1[16];
          tc::ld_32x32b_x16(tlane + sl[0] + pc * 16, r0);
          if (back >= 1) tc::ld_32x32b_x16(tlane + sl[1] + pc * 16, r1);
          tc::wait_ld();
          tap(r0, 0);
          if (back >= 1) tap(r1, 1);
          if (back >= 2) {
            tc::ld_32x32b_x16(tlane + sl[2] + pc * 16, r0);
            if (back >= 3) tc::ld_32x32b_x16(tlane + sl[3] + pc * 16, r1);
            tc::wait_ld();
            tap(r0, 2);
            if (back >= 3) tap(r1, 3);
          }
          const int col = n0 + c0;
          const float gate = col < 64 ? 1.f : col < 128 ? gv.x : gv.y;
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] = silu_f(v[j]) * gate;
          float* op = g.out + (frame * 192 + col) * g.HW + px;
#pragma unroll
          for (int j = 0; j < 16; ++j) op[(size_t)j * g.HW] = v[j];
        }
        tc::fence_before_sync();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&accempty[n & 1]);
      }
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == QT_MMA_WARP) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem_base, 512);
  }
}

static long long sequences(const GemmArgs& g) { return 2LL * (g.M / g.HW / g.T) * (g.HW / QT_BM); }

// g: the projection as launch_gemm takes it; kt: taps of the conv on its output
bool gemm_qkv_tconv_supported(const GemmArgs& g, int kt) {
  if (g.K != 64 || g.N != 192 || g.HW % QT_BM != 0 || g.T <= 0 || g.M % g.HW != 0 || g.M / g.HW % g.T != 0 || kt < 1 || kt > 4 ||
      g.bias == nullptr || g.o_planes != 192 || g.o_plane0 != 0)
    return false;
  // A sequence of T steps is the unit of work and cannot be split.  From two for every SM on the joined launch is ahead wherever the
  // last round ends (three rounds for the work of 2.05 included).  GDN block, us a pass, two launches / this one: 32x32, T = 8, 19
  // clips (304 sequences) 306 / 288, 20 310 / 294, 23 331 / 310, 27 380 / 331, 28 412 / 382, 38 533 / 478, 120 1463 / 1263; T = 1, 19
  // clips 82.8 / 71.7; T = 32, 19 1046 / 1001; 64x64, T = 8, 5 clips (320) 460 / 439, 10 874 / 816; 16x16, T = 4, 80 clips (320) 260 / 248.
  return sequences(g) >= 2 * sm_count() && sequences(g) < (1LL << 31) && sm_count() > 1;
}

int launch_gemm_qkv_tconv(const GemmArgs& g, const QkvTconvArgs& t, cudaStream_t st) {
  if (!gemm_qkv_tconv_supported(g, t.kt) || t.C != 64) return CSSM_ERR_UNSUPPORTED;
  QkvTconvGemmArgs a = {};
  a.g = g;
  for (int i = 0; i < 3; ++i) { a.wt[i] = t.wt[i]; a.bt[i] = t.bt[i]; }
  a.kt = t.kt; a.bkv = t.bkv;
  const int sms = sm_count() & ~1;
  a.seqs = (int)sequences(g);
  const cudaError_t e = func_smem(gemm_qkv_tconv_kernel, QT_SMEM + 1024);
  if (e != cudaSuccess) { set_cuda_error(e); return CSSM_ERR_CUDA; }
  launch_k(gemm_qkv_tconv_kernel, sms, QT_THREADS, QT_SMEM + 1024, st, a);
  return check_launch();
}

int read_qt_error(int* out, int clear) {
  cudaError_t e = cudaMemcpyFromSymbol(out, g_qt_error, sizeof(int));
  if (e == cudaSuccess && clear && *out != 0) {
    const int zero = 0;
    e = cudaMemcpyToSymbol(g_qt_error, &zero, sizeof(int));
  }
  if (e != cudaSuccess) { set_cuda_error(e); return CSSM_ERR_CUDA; }
  return CSSM_OK;
}

}  // namespace cssm
