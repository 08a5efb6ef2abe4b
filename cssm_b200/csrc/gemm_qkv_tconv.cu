// q, k, v projection of the GDN block at 64 channels with the causal temporal conv, SiLU and input gates behind it: the conv's
// history stays in TMEM.
//
//   out[b, t, n, px] = silu(b_t[n] + sum_j w_j[n] s[b, t - 3 + j, n, px]) * gate,   s = A W + bias (frames before 0: nothing)
//
// The tcgen05 GEMM of csrc/gemm_tc.cu (3 x TF32, raw tiles by TMA, A in TMEM) with another order of the tiles: a CTA takes 128
// pixels and one of q, k and v (64 columns) through t = 0 .. T - 1.  Its accumulators, 64 columns each, are a ring of five in
// TMEM: the epilogue of step t reads those of t - 3 .. t, while the MMAs of t + 1 fill the fifth; the other 128 columns are the A operand.
// So the projected planes never go to memory and back for the conv (6.4 GB of 128 x 8 x 64 x 64 x 64).  The price is that each tile
// of A is split three times, once for each of q, k and v (all 192 columns would need 768 of TMEM for the history); the CTAs of the three
// run side by side, so HBM sees it once.
// Bound: the epilogue's issue slots and special functions.  With halves of 96 columns, A in shared memory and eight epilogue warps the epilogue's reads
// of the taps waited for the MMAs' reads of A, and two warps a scheduler could not hide the special functions behind them.
#include "kernels.cuh"
#include "gemm_tc.cuh"
#include "bf16_ops.cuh"

namespace cssm {

__device__ int g_qt_error = 0;

constexpr int QT_CONV = 8, QT_EPI = 16;                           // converter and epilogue warps
constexpr int QT_MMA_WARP = QT_CONV, QT_LOAD_WARP = QT_CONV + 1, QT_EPI_WARP = QT_CONV + 2, QT_THREADS = (QT_CONV + 2 + QT_EPI) * 32;
constexpr int QT_N = 64, QT_RING = 5, QT_NRAW = 3;
constexpr uint32_t QT_B_HALF = 2u * QT_N * 128u;
constexpr uint32_t QT_RAW_OFF = 2u * QT_B_HALF, QT_TAB_OFF = QT_RAW_OFF + QT_NRAW * TC_RAW;
constexpr uint32_t QT_ANG_OFF = QT_TAB_OFF + 8u * QT_N * 4u, QT_WANG_OFF = QT_ANG_OFF + QT_NRAW * TC_ANG;      // tables: w[4][64], constants[4][64]
constexpr uint32_t QT_BAR_OFF = QT_WANG_OFF + TC_WANG, QT_SMEM = QT_BAR_OFF + 256u;
static_assert(QT_SMEM + 1024 <= 227 * 1024, "one CTA per SM");

struct QkvTconvGemmArgs {
  GemmArgs g;                                   // M, HW, A, source frames, RoPE, Wk (64, 192), bias, out (3C planes a frame), T
  const float* wt[3]; const float* bt[3]; int kt;
  const float2* bkv;                            // (frames, HW) {B_k, B_v} or nullptr
  int seqs;                                     // 3 * clips * HW / 128
  FastDiv blocks;                               // by the pixel blocks of a frame
};

template <int V> struct QtInt { static constexpr int value = V; };

__global__ void __launch_bounds__(QT_THREADS, 1) gemm_qkv_tconv_kernel(const __grid_constant__ QkvTconvGemmArgs a, const TcGeom dv,
                                                                       const __grid_constant__ CUtensorMap amap) {
  const GemmArgs& g = a.g;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned char* smem = smem_raw + ((1024u - (tc::smem_u32(smem_raw) & 1023u)) & 1023u);
  const uint32_t sbase = tc::smem_u32(smem);
  float* wtab = reinterpret_cast<float*>(smem + QT_TAB_OFF);      // [tap][column], tap 3 = the current frame
  float* ctab = wtab + 4 * QT_N;                                  // [min(t, 3)][column]: b_t + bias * sum of the taps in use
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + QT_BAR_OFF);
  uint64_t* raw_full = bars;       // [3] raw tile landed
  uint64_t* raw_empty = bars + 3;  // [3] and read (8 converter warps)
  uint64_t* full = bars + 6;       // [2] A stage (half of the channels) written (4 warps)
  uint64_t* empty = bars + 8;      // [2] A stage consumed
  uint64_t* accfull = bars + 10;   // [2] accumulator of step n, n & 1
  uint64_t* accempty = bars + 12;  // [2] epilogue of step n is through (8 warps)
  uint64_t* done = bars + 14;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 15);
  __shared__ int s_bad;            // a bounded wait expired
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int part3 = blockIdx.x % 3;                               // q, k or v: the grid is a multiple of three, a CTA keeps its own
  const bool rope_s = tc_rope_shared(g);

  if (tid == 0) {
    for (int i = 0; i < QT_NRAW; ++i) { tc::mbar_init(&raw_full[i], rope_s ? 2 : 1); tc::mbar_init(&raw_empty[i], QT_CONV); }
    for (int i = 0; i < 2; ++i) {
      tc::mbar_init(&full[i], QT_CONV / 2); tc::mbar_init(&empty[i], 1);
      tc::mbar_init(&accfull[i], 1); tc::mbar_init(&accempty[i], QT_EPI / 2);
    }
    tc::mbar_init(done, 1);
    tc::fence_mbar_init();
    s_bad = 0;
  }
  if (warp == QT_MMA_WARP) {
    tc::tmem_alloc(tmem_slot, 512);
    tc::tmem_relinquish();
  }
  tc_split_weights<QT_N>(g.Wk, 192, part3 * QT_N, smem, smem + QT_B_HALF, tid, QT_THREADS);
  if (rope_s) tc_rope_columns(g, smem + QT_WANG_OFF, tid, QT_THREADS);
  for (int n = tid; n < QT_N; n += QT_THREADS) {
    const float* wp = part3 == 0 ? a.wt[0] : part3 == 1 ? a.wt[1] : a.wt[2];
    const float bt = (part3 == 0 ? a.bt[0] : part3 == 1 ? a.bt[1] : a.bt[2])[n], b = g.bias[part3 * QT_N + n];
    float sum = 0.f;
    for (int j = 3; j >= 0; --j) {                                // newest first; fewer taps than four: zeros before them
      const int i = j - (4 - a.kt);
      const float w = i >= 0 ? wp[(size_t)i * 64 + n] : 0.f;
      wtab[j * QT_N + n] = w;
      sum += w;
      ctab[(3 - j) * QT_N + n] = fmaf(b, sum, bt);
    }
  }
  tc::fence_proxy_async();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem_base = *tmem_slot, tmem_a = tmem_base + QT_RING * QT_N;
  pdl_sync();
  // all lanes of a warp agree; a wait that expires is recorded
  auto wait = [&](uint64_t* bar, uint32_t phase, int code) {
    const bool ok = !__any_sync(0xffffffffu, !tc::mbar_wait(bar, phase));
    if (!ok) { if (lane == 0) atomicExch(&g_qt_error, code); s_bad = 1; }
    return ok;
  };

  const int T = g.T;
  // sequence s: q, k or v s % 3 of pixel block s / 3 of the clips
  auto clip_of = [&](int s, int& px0) {
    const int pb = s / 3, b = a.blocks.div(pb);
    px0 = (pb - b * (g.HW / TC_BM)) * TC_BM;
    return b;
  };

  if (warp < QT_CONV) {
    // ================================ converters ================================
    const int q = warp & 3, hf = warp >> 2, row = q * 32 + lane;             // lane quadrant, half of the channels
    const uint32_t tdst = tmem_a + ((uint32_t)(q * 32) << 16) + (uint32_t)(hf * 64);
    const uint32_t rot[2] = {tc_rotated(g, hf * 32), tc_rotated(g, hf * 32 + 16)};
    int n = 0, rs = 0;
    uint32_t rph = 0;
    bool ok = true;
    for (int s = blockIdx.x; s < a.seqs && ok; s += gridDim.x) {
      int px0;
      clip_of(s, px0);
      for (int t = 0; t < T; ++t, ++n) {
        const unsigned char* raw = smem + QT_RAW_OFF + rs * TC_RAW;
        if (!(ok = wait(&raw_full[rs], rph, 1))) break;
#pragma unroll
        for (int sl = 0; sl < 2; ++sl) {
          const int k0 = hf * 32 + sl * 16;
          float v[16];
          tc_read16_rows(raw, row, k0, v);
          tc_rotate16(g, rope_s, rot[sl], smem + QT_ANG_OFF + rs * TC_ANG, smem + QT_WANG_OFF, row, t, px0 + row, k0, v);
          if (sl == 1) {
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&raw_empty[rs]);
          } else {
            if (!(ok = wait(&empty[hf], (n & 1) ^ 1, 1))) break;
            tc::fence_after_sync();
          }
          tc_split_store16(tdst + sl * 16u, v);
        }
        if (!ok) break;
        tc::wait_st();
        tc::fence_before_sync();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&full[hf]);
        if (++rs == QT_NRAW) { rs = 0; rph ^= 1; }
      }
    }
  } else if (warp == QT_LOAD_WARP) {
    // ================================ loader ================================
    int rs = 0;
    uint32_t rph = 0;
    bool ok = true;
    for (int s = blockIdx.x; s < a.seqs && ok; s += gridDim.x) {
      int px0;
      const int b = clip_of(s, px0);
      for (int t = 0; t < T; ++t) {
        const int r0 = tc_src_frame(g, dv, b * T + t) * g.HW + px0;
        if (!(ok = wait(&raw_empty[rs], rph ^ 1, 5))) break;
        if (tc::elect_one()) {
          unsigned char* raw = smem + QT_RAW_OFF + rs * TC_RAW;
          tc::mbar_expect_tx(&raw_full[rs], TC_RAW);
          tc::tma_load_2d(raw, &amap, 0, r0, &raw_full[rs]);
          tc::tma_load_2d(raw + TC_BM * 128, &amap, 32, r0, &raw_full[rs]);
        }
        __syncwarp();
        if (rope_s) {
          tc_rope_rows(g, smem + QT_ANG_OFF + rs * TC_ANG, t, px0, lane);
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(&raw_full[rs]);
        }
        if (++rs == QT_NRAW) { rs = 0; rph ^= 1; }
      }
    }
  } else if (warp == QT_MMA_WARP) {
    // ================================ MMA issuer ================================
    // The whole warp walks the loop, one lane issues (elect_one).
    const uint32_t idesc = tc::make_idesc_tf32(TC_BM, QT_N);
    const uint64_t b_hi = tc::make_desc_sw128(sbase), b_lo = tc::make_desc_sw128(sbase + QT_B_HALF);
    const int mine = a.seqs > (int)blockIdx.x ? (a.seqs - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x * T : 0;
    bool ok = true;
    int slot = 0;
    for (int n = 0; n < mine && ok; ++n) {
      // the accumulator of step n - 5 was last read by the epilogue of step n - 2
      if (!(ok = wait(&accempty[n & 1], ((n >> 1) & 1) ^ 1, 2))) break;
      const uint32_t d = tmem_base + (uint32_t)slot * QT_N;
      if (++slot == QT_RING) slot = 0;
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        if (!(ok = wait(&full[hf], n & 1, 2))) break;
        tc::fence_after_sync();
        if (tc::elect_one()) tc_mma_small<QT_N>(d, tmem_a + hf * 64u, b_hi, b_lo, hf, idesc);
        __syncwarp();
      }
      if (ok && tc::elect_one()) {
        tc_mma_lead<QT_N>(d, tmem_a, b_hi, 0, idesc);
        tc::commit(&empty[0]);
        tc_mma_lead<QT_N>(d, tmem_a + 64u, b_hi, 1, idesc);
        tc::commit(&empty[1]);
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
    // Two groups of eight warps take every other step, so that one loads while the other is at its special functions.  Half of the columns
    // a warp, eight at a time: the frames under the four taps are requested together, one wait.
    constexpr int PART = QT_N / 2;
    const int q = warp & 3, grp = (warp - QT_EPI_WARP) >> 3, part = ((warp - QT_EPI_WARP) >> 2) & 1;      // q: TMEM lane quadrant
    const uint32_t tlane = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(part * PART);
    int n = grp, slot = grp, t = grp, s = blockIdx.x;
    bool ok = true;
    while (ok) {
      while (t >= T && s < a.seqs) { t -= T; s += gridDim.x; }
      if (s >= a.seqs) break;
      int px;
      const int b = clip_of(s, px);
      px += q * 32 + lane;
      {
        const size_t frame = (size_t)b * T + t;
        const float2 gv = a.bkv != nullptr && part3 != 0 ? __ldg(a.bkv + frame * g.HW + px) : make_float2(1.f, 1.f);
        if (!(ok = wait(&accfull[n & 1], (n >> 1) & 1, 4))) break;
        tc::fence_after_sync();
        // earlier frames of this clip under the taps (frames further back may hold anything: no product with a zero tap)
        const int back = t < a.kt - 1 ? t : a.kt - 1;
        uint32_t sl[4];                                                     // ring slots of t, t - 1, t - 2, t - 3
#pragma unroll
        for (int d = 0; d < 4; ++d) sl[d] = (uint32_t)(slot >= d ? slot - d : slot - d + QT_RING) * QT_N;
        const float gate = part3 == 0 ? 1.f : part3 == 1 ? gv.x : gv.y;
        float* op = g.out + (frame * 192 + part3 * QT_N + part * PART) * g.HW + px;
        // eight columns from pc on: taps of frames t - BACK .. t
        auto chunk = [&](auto BACK, int pc) {
          constexpr int NB = decltype(BACK)::value;
          const int c0 = part * PART + pc;
          uint32_t r[NB + 1][8];
#pragma unroll
          for (int d = 0; d <= NB; ++d) tc::ld_32x32b_x8(tlane + sl[d] + pc, r[d]);
          typedef unsigned long long u64;
          u64 v[4];
#pragma unroll
          for (int j = 0; j < 4; j += 2) {
            const ulonglong2 c = *reinterpret_cast<const ulonglong2*>(ctab + NB * QT_N + c0 + 2 * j);
            v[j] = c.x; v[j + 1] = c.y;
          }
          tc::wait_ld();
#pragma unroll
          for (int d = 0; d <= NB; ++d)
#pragma unroll
            for (int j = 0; j < 4; j += 2) {
              const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(wtab + (3 - d) * QT_N + c0 + 2 * j);
              v[j] = fma2(w.x, pk2(__uint_as_float(r[d][2 * j]), __uint_as_float(r[d][2 * j + 1])), v[j]);
              v[j + 1] = fma2(w.y, pk2(__uint_as_float(r[d][2 * j + 2]), __uint_as_float(r[d][2 * j + 3])), v[j + 1]);
            }
          const u64 g2 = pk2(gate, gate);
          float o[8];
#pragma unroll
          for (int j = 0; j < 4; ++j) upk2(mul2(mul2(v[j], sigmoid_x2(v[j])), g2), o[2 * j], o[2 * j + 1]);
#pragma unroll
          for (int j = 0; j < 8; ++j) op[(size_t)j * g.HW] = o[j];
          op += (size_t)8 * g.HW;
        };
#pragma unroll 1
        for (int pc = 0; pc < PART; pc += 8) {
          if (back == 3) chunk(QtInt<3>(), pc);
          else if (back == 0) chunk(QtInt<0>(), pc);
          else if (back == 1) chunk(QtInt<1>(), pc);
          else chunk(QtInt<2>(), pc);
        }
        tc::fence_before_sync();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&accempty[n & 1]);
      }
      n += 2; t += 2;
      slot += 2;
      if (slot >= QT_RING) slot -= QT_RING;
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  // error path only: give copies that may still be in flight a bounded time (~1 ms) to land
  if (s_bad)
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
  if (warp == QT_MMA_WARP) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem_base, 512);
  }
}

static long long sequences(const GemmArgs& g) { return 3LL * (g.M / g.HW / g.T) * (g.HW / TC_BM); }

// g: the projection as launch_gemm takes it; kt: taps of the conv on its output
bool gemm_qkv_tconv_supported(const GemmArgs& g, int kt) {
  if (g.K != 64 || g.N != 192 || g.HW % TC_BM != 0 || g.T <= 0 || g.M % g.HW != 0 || g.M / g.HW % g.T != 0 || kt < 1 || kt > 4 ||
      g.bias == nullptr || g.o_planes != 192 || g.o_plane0 != 0 || !aligned16(g.A))
    return false;
  // A sequence of T steps is the unit of work and cannot be split: with few of them most SMs are idle for T steps.  The joined launch is
  // ahead from two sequences for three SMs on, and at up to four steps always (one launch less).  GDN block, us a pass, two launches / this
  // one: 32x32, T = 8, 4 clips (96 sequences) 112 / 98, 19 271 / 249, 62 734 / 620; T = 32, 4 312 / 287, 19 972 / 867; T = 1, 19 79 / 68; 64x64,
  // T = 8, 2 clips (192) 343 / 336, T = 32 1273 / 1250; 16x16, T = 32, 16 clips (96) 546 / 529; below: 16x16, T = 8, 4 clips 122 / 123, T =
  // 32, 12 clips 501 / 512, T = 4, one clip 78.8 / 78.5; 32x32, T = 32, one clip 236 / 238.  With halves of 96 columns 32x32, T = 8, 19
  // clips took 288, 62 694.
  return (g.T <= 4 || 3 * sequences(g) >= 2 * (sm_count() / 3 * 3)) && sequences(g) < (1LL << 31) && sm_count() > 2;
}

int launch_gemm_qkv_tconv(const GemmArgs& g, const QkvTconvArgs& t, cudaStream_t st) {
  if (!gemm_qkv_tconv_supported(g, t.kt) || t.C != 64) return CSSM_ERR_UNSUPPORTED;
  QkvTconvGemmArgs a = {};
  a.g = g;
  for (int i = 0; i < 3; ++i) { a.wt[i] = t.wt[i]; a.bt[i] = t.bt[i]; }
  a.kt = t.kt; a.bkv = t.bkv;
  a.seqs = (int)sequences(g);
  const int sms = sm_count() / 3 * 3, grid = a.seqs < sms ? a.seqs : sms;       // multiples of three
  a.blocks = FastDiv(g.HW / TC_BM);
  CUtensorMap amap;
  if (!tc_input_map(g, false, false, &amap)) return CSSM_ERR_CUDA;
  const cudaError_t e = func_smem(gemm_qkv_tconv_kernel, QT_SMEM + 1024);
  if (e != cudaSuccess) { set_cuda_error(e); return CSSM_ERR_CUDA; }
  launch_k(gemm_qkv_tconv_kernel, grid, QT_THREADS, QT_SMEM + 1024, st, a, TcGeom(g), amap);
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
