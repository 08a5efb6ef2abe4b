// tcgen05 / TMEM GEMM for the K = 64 channel projections in fp32-equivalent precision
// (3 x TF32: A_lo*B_hi + A_hi*B_lo + A_hi*B_hi, accumulated in fp32 in TMEM; with the RMS prologue six products of three bf16 parts).
//
// Persistent kernel, one CTA per SM, 26 warps (18 where a second tensor is subtracted):
//   loader, 1 warp       : TMA copies of 128-pixel A tiles as they lie in memory (channels-last rows, or planar planes and
//                          their gate planes) into a ring of raw tiles, and the angles of the tile's frame and rows;
//   converters, 16 or 8  : lane = pixel, 16 of the 64 channels at a time: read the raw tile, apply RoPE or the gate, split every
//                          value into tf32 hi + remainder and write both to TMEM (tcgen05.st), where the MMAs read their A operand;
//                          a stage is half of the channels;
//   MMA issuer, 1 warp   : 24 tcgen05.mma (M128 x N x K8, bf16 K16; A in TMEM, B in shared memory) per tile into one of two TMEM
//                          accumulators, commits to mbarriers;
//   epilogue, 8 or 16    : tcgen05.ld the accumulator (lane = pixel; two or four warps per TMEM lane
//                          quadrant, a share of the columns each), add bias / activation, store
//                          planar (coalesced over pixels) or channels-last rows.
// The weight tile (both halves of the split) is prepared once per CTA and stays in shared memory.
// With A in shared memory the MMAs' operand reads (6 to 8 KB an instruction) and the converters' stores shared its one port, and the
// converters, which loaded A through the L1 as well and so kept the rotation tables out of it, set the pace: a clock trace had them
// at 2000 clocks a tile without RoPE and 2800 to 3700 with it, of 3700 to 5000 in all.  4.2 M rows, us: 64 -> 128 columns 631 -> 429, planes
// -> 64 435 -> 359, 64 -> 64 with sigmoid 472 -> 330 (rows of repeated frames 619 -> 345), planes under RMS and gate 706 (gemm_split) ->
// 507; HBM's copy rate allows 493, 328, 328 (164) and 493.  98 K rows of 64 -> 128 + 64 in place 137 -> 110.
// Bound now: HBM for the planes, issue slots (65 to 70 % busy) where little is read.
// Every mbarrier wait is bounded; on expiry the kernel records an error code and winds down.
#include <cuda.h>
#include <string.h>
#include "kernels.cuh"
#include "gemm_tc.cuh"
#include "bf16_ops.cuh"
#include "stem.cuh"

namespace cssm {

__device__ int g_tc_error = 0;

// Forms of the epilogue: plain; ZLAST: the output columns from act_n0 on (the z half of the in_proj) are only produced for the
// last frame of every clip (last-frame-only forward); MUL: the first g.mul_n output columns multiply planes in place; SUB: the
// channels-last tensor g.sub is subtracted from the rows.  Compile-time variants, so that the plain one carries no extra test.
// RMS (planar A, 64 columns): a <- a * rsqrt(mean_k a^2 + eps) * scale[k]; the scale goes into the weights, the row factor to the accumulator.
// Its operands are three bf16 parts, all 24 bits of a float32, as gemm_split_kernel has them (two tf32 parts hold 22): error of the launch
// against float64 1.1e-7 of the 2-norm, 2.0e-7 with two tf32 parts, at the same time (4.2 M rows 507 us, 1 M 135); gemm_split_kernel 1.2e-7,
// 701.
enum TcForm { TC_PLAIN, TC_ZLAST, TC_MUL, TC_SUB, TC_RMS };
// Warps: converters, MMA issuer, loader, epilogue.  A wide planar output has more to store than to convert (with sixteen converters and
// eight epilogue warps: 4.2 M rows to 128 columns 491 us, 429 so; DeltaNet 32x32, whose 192 columns multiply planes, 462 and 415 a pass).
// SUB reads a second tensor behind the accumulator: eight of each, whose registers hold the row to come (26 warps cannot: 12 x 8 x 64 x 64
// NoGate 218 us a pass, 128 x 8 x 32 x 32 600; so 205 and 562).
template <int N, bool A_PLANAR, TcForm FORM> constexpr int tc_conv = (FORM == TC_SUB || (!A_PLANAR && N > 64)) ? 8 : 16;
template <int N, bool A_PLANAR, TcForm FORM> constexpr int tc_epi = FORM == TC_SUB ? 8 : 24 - tc_conv<N, A_PLANAR, FORM>;
template <int N, bool A_PLANAR, TcForm FORM> constexpr int tc_threads = (tc_conv<N, A_PLANAR, FORM> + tc_epi<N, A_PLANAR, FORM> + 2) * 32;

// One output of a planar A under the RMS prologue by float32 FMAs over k: for results that are not finite (the products are taken
// before the row factor, and an infinity has no finite parts).
__device__ __noinline__ float tc_planar_fma(const GemmArgs& g, const TcGeom& dv, int m, int n, float rinv) {
  const int fo = dv.hw.div(m), px = m - fo * g.HW, fr = tc_src_frame(g, dv, fo);
  const float* ap = g.A + ((size_t)fr * g.a_planes + g.a_plane0) * g.HW + px;
  const float* gp = g.gate ? g.gate + ((size_t)(g.g_compact ? fo : fr) * g.g_planes + g.g_plane0) * g.HW + px : nullptr;
  float v = 0.f;
  for (int k = 0; k < TC_K; ++k) {
    float x = ap[(size_t)k * g.HW] * (rinv * g.rms_scale[k]);
    if (gp != nullptr) x *= gp[(size_t)k * g.HW];
    v = fmaf(x, g.Wk[(size_t)k * g.N + n], v);
  }
  return g.bias != nullptr ? v + g.bias[n] : v;
}

// STG = true: the epilogue stages 16 KB chunks (128 pixels x 32 output columns) in shared memory, one chunk buffer per half of the
// epilogue warps, and writes each chunk with one TMA tensor store (channels-last output, N <= 128); else it stores from registers.
template <int N, bool GATE, bool STG, bool RMS = false>
struct TcSmem {
  static constexpr int NT = N == 192 ? 1 : 2;                            // tiles of A in TMEM, two stages of 64 columns each
  static constexpr int NRAW = GATE ? 2 : N == 192 ? 3 : 4;          // raw tiles in flight
  static constexpr uint32_t RAW_BYTES = GATE ? 2u * TC_RAW : TC_RAW;
  static constexpr uint32_t B_HALF = 2u * N * 128u;
  static constexpr uint32_t B_OFF = 0;
  static constexpr uint32_t RAW_OFF = 2u * B_HALF;                       // after B_hi, B_lo
  static constexpr uint32_t OUT_OFF = RAW_OFF + NRAW * RAW_BYTES;        // 2 x 16 KB when STG
  static constexpr uint32_t BIAS_OFF = OUT_OFF + (STG ? 2u * 16384u : 0u);
  static constexpr uint32_t ANG_OFF = BIAS_OFF + N * 4u;                 // angles of a raw tile's rows: [NRAW][8 rows][32 pairs]
  static constexpr uint32_t WANG_OFF = ANG_OFF + (STG ? 0u : NRAW * TC_ANG);
  static constexpr uint32_t BAR_OFF = WANG_OFF + (STG ? 0u : TC_WANG);
  static constexpr uint32_t SS_OFF = BAR_OFF + 256u;                     // RMS: [4 tiles][4 parts of the channels][128] sums of squares
  static constexpr uint32_t TOTAL = SS_OFF + (RMS ? 4u * 4u * 128u * 4u : 0u);
  static_assert(TOTAL + 1024u <= 227u * 1024u, "one CTA per SM");
};

template <int N, bool A_PLANAR, bool GATE, bool STG, TcForm FORM = TC_PLAIN>
__global__ void __launch_bounds__((tc_threads<N, A_PLANAR, FORM>), 1)
gemm_tc_kernel(const __grid_constant__ GemmArgs g, const __grid_constant__ TcGeom dv, int num_tiles, const __grid_constant__ CUtensorMap amap, const __grid_constant__ CUtensorMap gmap,
               const __grid_constant__ CUtensorMap omap) {
  // tile schedule: round-robin over the CTAs
  const int t_first = blockIdx.x, t_step = gridDim.x, t_end = num_tiles;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  // operand tiles need 1024-byte alignment (swizzle atoms); the launch adds 1024 bytes of slack
  unsigned char* smem = smem_raw + ((1024u - (tc::smem_u32(smem_raw) & 1023u)) & 1023u);
  using L = TcSmem<N, GATE, STG, FORM == TC_RMS>;
  constexpr int CONV = tc_conv<N, A_PLANAR, FORM>, EPI = tc_epi<N, A_PLANAR, FORM>, THREADS = tc_threads<N, A_PLANAR, FORM>;
  constexpr int MMA_WARP = CONV, LOAD_WARP = CONV + 1, EPI_WARP = CONV + 2;
  constexpr int NT = L::NT, NST = 2 * NT, NRAW = L::NRAW;
  const uint32_t sbase = tc::smem_u32(smem);
  float* bias_s = reinterpret_cast<float*>(smem + L::BIAS_OFF);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BAR_OFF);
  uint64_t* raw_full = bars;           // [4] raw tile landed
  uint64_t* raw_empty = bars + 4;      // [4] and read (all converter warps)
  uint64_t* full = bars + 8;           // [4] A stage written (half of the converter warps)
  uint64_t* empty = bars + 12;         // [4] A stage consumed (tcgen05.commit)
  uint64_t* accfull = bars + 16;       // [2] accumulator complete (tcgen05.commit)
  uint64_t* accempty = bars + 18;      // [2] accumulator drained (all epilogue warps)
  uint64_t* done = bars + 20;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 21);
  __shared__ int s_bad;                // a bounded wait expired

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  const bool rope_s = !A_PLANAR && tc_rope_shared(g);
  if (tid == 0) {
    for (int i = 0; i < NRAW; ++i) { tc::mbar_init(&raw_full[i], rope_s ? 2 : 1); tc::mbar_init(&raw_empty[i], CONV); }
    for (int i = 0; i < NST; ++i) { tc::mbar_init(&full[i], CONV / 2); tc::mbar_init(&empty[i], 1); }
    for (int i = 0; i < 2; ++i) { tc::mbar_init(&accfull[i], 1); tc::mbar_init(&accempty[i], EPI); }
    tc::mbar_init(done, 1);
    tc::fence_mbar_init();
    s_bad = 0;
  }
  if (warp == MMA_WARP) {
    tc::tmem_alloc(tmem_slot, 512);
    tc::tmem_relinquish();
  }
  if constexpr (FORM == TC_RMS) tc_split3_weights<N>(g.Wk, g.rms_scale, smem + L::B_OFF, tid, THREADS);
  else tc_split_weights<N>(g.Wk, g.N, 0, smem + L::B_OFF, smem + L::B_OFF + L::B_HALF, tid, THREADS);
  if (rope_s) tc_rope_columns(g, smem + L::WANG_OFF, tid, THREADS);
  for (int n = tid; n < N; n += THREADS) bias_s[n] = g.bias ? g.bias[n] : 0.f;
  tc::fence_proxy_async();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem_a = tmem_base + 2u * N;            // stages of 64 columns: 32 channels hi, 32 lo
  pdl_sync();
  // all lanes of a warp agree; a wait that expires is recorded
  auto wait = [&](uint64_t* bar, uint32_t phase, int code) {
    const bool ok = !__any_sync(0xffffffffu, !tc::mbar_wait(bar, phase));
    if (!ok) { if (lane == 0) atomicExch(&g_tc_error, code); s_bad = 1; }
    return ok;
  };

  if (warp < CONV) {
    // ================================ converters ================================
    // channels 32 hf + 16 sl .. + 15 of the quadrant's pixels; of eight warps each has both sl
    const int q = warp & 3, grp = warp >> 2, hf = CONV == 16 ? grp >> 1 : grp, sl0 = CONV == 16 ? grp & 1 : 0;
    const int row = q * 32 + lane;
    const uint32_t tdst = tmem_a + ((uint32_t)(q * 32) << 16) + (uint32_t)(hf * 64);
    uint32_t rot[16 / CONV];
#pragma unroll
    for (int i = 0; i < 16 / CONV; ++i) rot[i] = A_PLANAR ? 0u : tc_rotated(g, hf * 32 + (sl0 + i) * 16);
    int it = 0;
    for (int tile = t_first; tile < t_end; tile += t_step, ++it) {
      const int rs = it % NRAW, s = (it % NT) * 2 + hf;
      const unsigned char* raw = smem + L::RAW_OFF + rs * L::RAW_BYTES;
      int t = 0, px = 0;
      if (!A_PLANAR && !rope_s && g.rope_t != nullptr) {
        const int m0 = tile * TC_BM, fr = dv.hw.div(m0);
        px = m0 - fr * g.HW + row;
        t = tc_rope_t(g, dv, fr);
      }
      if (!wait(&raw_full[rs], (it / NRAW) & 1, 1)) break;
      bool ok = true;
#pragma unroll
      for (int i = 0; i < 16 / CONV; ++i) {
        const int sl = sl0 + i, k0 = hf * 32 + sl * 16;
        float v[16], ss = 0.f;
        if (!A_PLANAR) {
          tc_read16_rows(raw, row, k0, v);
          tc_rotate16(g, rope_s, rot[i], smem + L::ANG_OFF + rs * TC_ANG, smem + L::WANG_OFF, row, t, px, k0, v);
        } else {
          ss = tc_read16_planes<GATE, FORM == TC_RMS>(raw, row, k0, v);
        }
        if (i == 16 / CONV - 1) {
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(&raw_empty[rs]);
        }
        if (i == 0) {
          if (!(ok = wait(&empty[s], ((it / NT) & 1) ^ 1, 1))) break;
          tc::fence_after_sync();
          // (the epilogue of the tile four back is through: the MMAs of the one two back, which this stage waited for, began after it)
          if (FORM == TC_RMS) reinterpret_cast<float*>(smem + L::SS_OFF)[((it & 3) * 4 + grp) * 128 + row] = ss;
        }
        if constexpr (FORM == TC_RMS) tc_split3_store16(tdst + (uint32_t)(it % NT) * 128u + sl * 8u, v);
        else tc_split_store16(tdst + (uint32_t)(it % NT) * 128u + sl * 16u, v);
      }
      if (!ok) break;
      tc::wait_st();
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&full[s]);
    }
  } else if (warp == LOAD_WARP) {
    // ================================ loader ================================
    int it = 0;
    for (int tile = t_first; tile < t_end; tile += t_step, ++it) {
      const int rs = it % NRAW;
      const int m0 = tile * TC_BM, fo = dv.hw.div(m0), px0 = m0 - fo * g.HW, fr = tc_src_frame(g, dv, fo);
      if (!wait(&raw_empty[rs], ((it / NRAW) & 1) ^ 1, 5)) break;
      if (tc::elect_one()) {
        unsigned char* raw = smem + L::RAW_OFF + rs * L::RAW_BYTES;
        tc::mbar_expect_tx(&raw_full[rs], L::RAW_BYTES);
        if (!A_PLANAR) {
          tc::tma_load_2d(raw, &amap, 0, fr * g.HW + px0, &raw_full[rs]);
          tc::tma_load_2d(raw + TC_BM * 128, &amap, 32, fr * g.HW + px0, &raw_full[rs]);
        } else {
          tc::tma_load_3d(raw, &amap, px0, g.a_plane0, fr, &raw_full[rs]);
          if (GATE) tc::tma_load_3d(raw + TC_RAW, &gmap, px0, g.g_plane0, g.g_compact ? fo : fr, &raw_full[rs]);
        }
      }
      __syncwarp();
      if (rope_s) {
        tc_rope_rows(g, smem + L::ANG_OFF + rs * TC_ANG, tc_rope_t(g, dv, fo), px0, lane);
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&raw_full[rs]);
      }
    }
  } else if (warp == MMA_WARP) {
    // ================================ MMA issuer ================================
    // The whole warp walks the loop, one lane issues (elect_one).
    const uint32_t idesc = FORM == TC_RMS ? tc::make_idesc_bf16(TC_BM, N) : tc::make_idesc_tf32(TC_BM, N);
    const uint64_t b_hi = tc::make_desc_sw128(sbase + L::B_OFF), b_lo = tc::make_desc_sw128(sbase + L::B_OFF + L::B_HALF);
    int it = 0;
    bool ok = true;
    for (int tile = t_first; tile < t_end && ok; tile += t_step, ++it) {
      const int ac = it & 1, ph = (it >> 1) & 1;              // accumulator and its phase
      if (!(ok = wait(&accempty[ac], ph ^ 1, 2))) break;
      const uint32_t d = tmem_base + (uint32_t)ac * N;
      const int s = (it % NT) * 2;
      const uint32_t a = tmem_a + (uint32_t)s * 64u;
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        if (!(ok = wait(&full[s + hf], (it / NT) & 1, 2))) break;
        tc::fence_after_sync();
        if (tc::elect_one()) {
          if constexpr (FORM == TC_RMS) tc_mma3_small<N>(d, a + hf * 64u, b_hi, hf, idesc);
          else tc_mma_small<N>(d, a + hf * 64u, b_hi, b_lo, hf, idesc);
        }
        __syncwarp();
      }
      if (ok && tc::elect_one()) {
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          if constexpr (FORM == TC_RMS) tc_mma3<N>(d, a + hf * 64u, b_hi, 0, 0, hf, idesc, false);
          else tc_mma_lead<N>(d, a + hf * 64u, b_hi, hf, idesc);
          tc::commit(&empty[s + hf]);
        }
        tc::commit(&accfull[ac]);
      }
      __syncwarp();
    }
    // nothing of this warp's tensor work may be in flight when TMEM is freed
    if (tc::elect_one()) tc::commit(done);
    __syncwarp();
    if (!tc::mbar_wait(done, 0) && ok) atomicExch(&g_tc_error, 3);
    __syncwarp();
  } else {
    // ================================ epilogue ================================
    const int q = warp & 3;                 // TMEM lane quadrant this warp may read
    // (Two groups of warps with an accumulator and every other tile each, as in gemm_qkv_tconv_kernel, were no faster here: DeltaNet 32x32
    // 415 -> 427 us a pass, the gate projection of 64x64 GDN 347 -> 397.)
    const int half = (warp - EPI_WARP) >> 2;      // which half (of eight warps) or quarter (of sixteen) of the N columns
    constexpr int CH = EPI == 16 ? 16 : 32, COLS = N / (EPI / 4);
    const int row = q * 32 + lane;
    int it = 0;
    for (int tile = t_first; tile < t_end; tile += t_step, ++it) {
      const int s = it & 1, ph = (it >> 1) & 1;
      // SUB (one chunk a half): the row to subtract is in flight while the accumulator is waited for
      float4 sv[FORM == TC_SUB ? CH / 4 : 1];
      if constexpr (FORM == TC_SUB) {
        static_assert(COLS == CH && STG, "one chunk");
        const float4* sp = reinterpret_cast<const float4*>(g.sub + (size_t)(tile * TC_BM + row) * g.N + half * COLS);
#pragma unroll
        for (int j = 0; j < CH / 4; ++j) sv[j] = __ldg(sp + j);
      }
      bool ok = tc::mbar_wait(&accfull[s], ph);
      if (STG) {
        // the named barriers below need all 128 threads of the half: make the exit uniform
        uint32_t all_ok;
        asm volatile(
            "{\n\t.reg .pred p, q;\n\t"
            "setp.ne.u32 p, %1, 0;\n\t"
            "bar.red.and.pred q, %2, 128, p;\n\t"
            "selp.u32 %0, 1, 0, q;\n\t}"
            : "=r"(all_ok) : "r"((uint32_t)ok), "r"(1 + half) : "memory");
        ok = all_ok != 0;
      } else {
        ok = !__any_sync(0xffffffffu, !ok);
      }
      if (!ok) { atomicExch(&g_tc_error, 4); s_bad = 1; break; }
      tc::fence_after_sync();
      const int m = tile * TC_BM + row, fr = dv.hw.div(tile * TC_BM), px = m - fr * g.HW;
      const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)s * N;
      float rinv = 1.f;
      if (FORM == TC_RMS) {
        const float* sp = reinterpret_cast<const float*>(smem + L::SS_OFF) + (it & 3) * 512 + row;
        rinv = rsqrtf(((sp[0] + sp[128]) + (sp[256] + sp[384])) * (1.0f / TC_K) + 1e-6f);
      }
#pragma unroll 1
      for (int c0 = half * COLS; c0 < (half + 1) * COLS; c0 += CH) {
        if (FORM == TC_ZLAST && c0 >= g.act_n0 && fr - dv.t.div(fr) * g.T != g.T - 1) continue;   // tile-uniform
        uint32_t r[CH];
        if constexpr (CH == 32) tc::ld_32x32b_x32(taddr + c0, r);
        else tc::ld_32x32b_x16(taddr + c0, r);
        tc::wait_ld();
        if (STG) {
          // this half's 128 threads share two 16 KB staging chunks and named barrier 1 + half
          const int grp_tid = tid - (EPI_WARP + 4 * half) * 32;      // 0..127
          float* stg = reinterpret_cast<float*>(smem + L::OUT_OFF) + half * 4096;
          // the TMA store that last read this chunk buffer must have drained it
          if (grp_tid == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
          asm volatile("bar.sync %0, 128;" ::"r"(1 + half) : "memory");
          const float* bs = bias_s + c0;
          {
            // chunk layout [pixel][32 columns] in the 128-byte swizzle the tensor map expects
            float vals[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) vals[j] = FORM == TC_RMS ? fmaf(__uint_as_float(r[j]), rinv, bs[j]) : __uint_as_float(r[j]) + bs[j];
            if (FORM == TC_SUB) {
#pragma unroll
              for (int j = 0; j < 32; j += 4) {
                const float4 u = sv[j >> 2];
                vals[j] -= u.x; vals[j + 1] -= u.y; vals[j + 2] -= u.z; vals[j + 3] -= u.w;
              }
            }
#pragma unroll
            for (int j = 0; j < 32; j += 4)
              *reinterpret_cast<float4*>(reinterpret_cast<unsigned char*>(stg) +
                                         tc::sw128_offset(row, j >> 2)) =
                  make_float4(vals[j], vals[j + 1], vals[j + 2], vals[j + 3]);
            if (FORM == TC_RMS) {
              // not finite, though the normalised row may be: again by FMAs
              float odd = 0.f;
#pragma unroll
              for (int j = 0; j < 32; ++j) odd = fmaf(vals[j], 0.f, odd);
              if (odd != 0.f)
                for (int j = 0; j < 32; ++j)
                  *reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(stg) + tc::sw128_offset(row, j >> 2) + (j & 3) * 4) =
                      tc_planar_fma(g, dv, m, c0 + j, rinv);
            }
          }
          tc::fence_proxy_async();
          asm volatile("bar.sync %0, 128;" ::"r"(1 + half) : "memory");
          if (grp_tid == 0) {
            tc::tma_store_2d(&omap, stg, c0, tile * TC_BM);
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          }
          continue;
        }
        // planar output: lanes = consecutive pixels -> 128-byte coalesced stores per column.
        // All values are finished in registers before the first store: the stores go
        // through a generic pointer, so bias loads placed between them could not be hoisted.
        float* op = g.out + ((size_t)fr * g.o_planes + g.o_plane0 + c0) * g.HW + px;
        float vals[CH];
#pragma unroll
        for (int j = 0; j < CH; ++j) vals[j] = __uint_as_float(r[j]) + bias_s[c0 + j];
        if (g.out_act == 1 && c0 >= g.act_n0) {
#pragma unroll
          for (int j = 0; j < CH; j += 2) {
            const unsigned long long x = pk2(vals[j], vals[j + 1]);
            upk2(mul2(x, sigmoid_x2(x)), vals[j], vals[j + 1]);
          }
        } else if (g.out_act == 2 && c0 >= g.act_n0) {
#pragma unroll
          for (int j = 0; j < CH; j += 2) upk2(sigmoid_x2(pk2(vals[j], vals[j + 1])), vals[j], vals[j + 1]);
        }
        if (FORM == TC_MUL && c0 < g.mul_n) {
          op = g.mul + ((size_t)fr * g.mul_planes + g.mul_plane0 + c0) * g.HW + px;
          float old[CH];
#pragma unroll
          for (int j = 0; j < CH; ++j) old[j] = op[(size_t)j * g.HW];
#pragma unroll
          for (int j = 0; j < CH; ++j) vals[j] *= old[j];
        }
#pragma unroll
        for (int j = 0; j < CH; ++j) op[(size_t)j * g.HW] = vals[j];
      }
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&accempty[s]);
    }
    // shared memory must outlive the last TMA stores that read it
    if (STG) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
  }
  tc::fence_before_sync();
  __syncthreads();
  // error path only: give copies that may still be in flight a bounded time (~1 ms) to land
  if (s_bad)
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
  if (warp == MMA_WARP) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem_base, 512);
  }
}

bool gemm_tc_in_place(int K, int N, int HW, int mul_n) {
  return K == TC_K && (N == 128 || N == 192) && HW % TC_BM == 0 && mul_n % 32 == 0;
}

// Whether this kernel takes the problem (else gemm_split_kernel, csrc/gemm_split.cu): 64 channels, tiles inside one frame, 16-byte
// aligned tensors; the RMS prologue for 64 columns.
bool gemm_tc_supported(const GemmArgs& g, bool a_planar) {
  if (g.rms_scale != nullptr && !(a_planar && g.N == 64 && g.sub == nullptr)) return false;
  if (g.K != TC_K || (g.N != 64 && g.N != 128 && g.N != 192)) return false;
  if (g.HW % TC_BM != 0 || g.M % TC_BM != 0) return false;
  if (g.out_act != 0 && g.act_n0 % 32 != 0) return false;
  if (g.mul != nullptr && !gemm_tc_in_place(g.K, g.N, g.HW, g.mul_n)) return false;
  if (a_planar && (g.N == 192 || (g.sub != nullptr && g.N != 64))) return false;
  if (!aligned16(g.A) || (a_planar && (!aligned16(g.out) || (g.gate != nullptr && !aligned16(g.gate))))) return false;      // TMA
  return true;
}

// Tensor map of the channels-last output for the TMA stores: 16 KB boxes of 128 pixels x 32 columns.
static bool make_out_map(const GemmArgs& g, CUtensorMap* map) {
  const tc::EncodeTiledFn enc = tc::encode_fn();
  if (!enc) return false;
  const cuuint32_t es[2] = {1, 1};
  const cuuint64_t dims[2] = {(cuuint64_t)g.N, (cuuint64_t)g.M};
  const cuuint64_t strides[1] = {(cuuint64_t)g.N * 4};
  const cuuint32_t box[2] = {32, 128};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, g.out, dims, strides, box, es,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
             CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// (the rows of a channels-last A are those of its source frames, which may be fewer or more than the output's)
bool tc_input_map(const GemmArgs& g, bool a_planar, bool gate, CUtensorMap* map) {
  const tc::EncodeTiledFn enc = tc::encode_fn();
  if (!enc) return false;
  const int fo = g.M / g.HW;                                       // output frames; their last source frame
  const bool remap = (g.a_fmul != 0 || g.a_fadd != 0) && !(gate && g.g_compact);
  const cuuint64_t frames = remap ? (cuuint64_t)((g.a_fdiv > 1 ? (fo - 1) / g.a_fdiv : fo - 1) * (long long)g.a_fmul + g.a_fadd + 1) : (cuuint64_t)fo;
  const cuuint32_t es[3] = {1, 1, 1};
  CUresult r;
  if (!a_planar) {
    const cuuint64_t dims[2] = {TC_K, frames * g.HW};
    const cuuint64_t strides[1] = {TC_K * 4};
    const cuuint32_t box[2] = {32, TC_BM};
    r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(g.A), dims, strides, box, es,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
            CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  } else {
    const int planes = gate ? g.g_planes : g.a_planes;
    const cuuint64_t dims[3] = {(cuuint64_t)g.HW, (cuuint64_t)planes, frames};
    const cuuint64_t strides[2] = {(cuuint64_t)g.HW * 4, (cuuint64_t)planes * g.HW * 4};
    const cuuint32_t box[3] = {TC_BM, TC_K, 1};
    r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(gate ? g.gate : g.A), dims, strides, box, es,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
            CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  }
  return r == CUDA_SUCCESS;
}

template <int N, bool A_PLANAR, bool GATE, bool STG, TcForm FORM>
static int launch_tc_v(const GemmArgs& g, const CUtensorMap& omap, cudaStream_t st) {
  const int num_tiles = g.M / TC_BM;
  const int sms = sm_count();
  cudaError_t e;
  const int grid = num_tiles < sms ? num_tiles : sms;
  const size_t smem = TcSmem<N, GATE, STG, FORM == TC_RMS>::TOTAL + 1024;      // slack for the 1024-byte alignment
  e = func_smem(gemm_tc_kernel<N, A_PLANAR, GATE, STG, FORM>, smem);
  if (e != cudaSuccess) { set_cuda_error(e); return CSSM_ERR_CUDA; }
  CUtensorMap amap, gmap;
  memset(&gmap, 0, sizeof(gmap));
  if (!tc_input_map(g, A_PLANAR, false, &amap) || (GATE && !tc_input_map(g, true, true, &gmap))) return CSSM_ERR_CUDA;
  // Planes of 64x64: the 64 planes of a tile lie 1 MB apart in all, which neighbouring SMs share (NoGate's output
  // projection of 48 x 4 frames: 104 us in grid order, 139 with the CTAs where SMs came free); 8 x 4 frames and less, and
  // smaller planes, gain more by the early start.  Channels-last input: the second projection of the same rows.
  const PdlOff alone(N == 64 && num_tiles > 8 * sms && (!A_PLANAR || g.HW >= 4096));
  const TcGeom dv(g);
  launch_k(gemm_tc_kernel<N, A_PLANAR, GATE, STG, FORM>, grid, tc_threads<N, A_PLANAR, FORM>, smem, st, g, dv, num_tiles, amap, gmap, omap);
  return check_launch();
}

template <int N, bool A_PLANAR, TcForm FORM = TC_PLAIN>
static int launch_tc(const GemmArgs& g, cudaStream_t st) {
  CUtensorMap map;
  memset(&map, 0, sizeof(map));
  if constexpr (!A_PLANAR) {
    // (planar output: TMA stores measured slower than direct ones, 2.1 against 1.44 ms on an in_proj of 4.2 M rows)
    return launch_tc_v<N, false, false, false, FORM>(g, map, st);
  } else {
    if (!make_out_map(g, &map)) return CSSM_ERR_CUDA;
    return g.gate != nullptr ? launch_tc_v<N, true, true, true, FORM>(g, map, st) : launch_tc_v<N, true, false, true, FORM>(g, map, st);
  }
}

int launch_gemm_tc(const GemmArgs& g, bool a_planar, cudaStream_t st) {
  if (!gemm_tc_supported(g, a_planar)) return CSSM_ERR_UNSUPPORTED;
  if (a_planar)
    return g.N == 128 ? launch_tc<128, true>(g, st) : g.sub != nullptr ? launch_tc<64, true, TC_SUB>(g, st)
                          : g.rms_scale != nullptr ? launch_tc<64, true, TC_RMS>(g, st) : launch_tc<64, true>(g, st);
  if (g.z_last_only && g.N == 128) return launch_tc<128, false, TC_ZLAST>(g, st);
  if (g.mul != nullptr) return g.N == 192 ? launch_tc<192, false, TC_MUL>(g, st) : launch_tc<128, false, TC_MUL>(g, st);
  return g.N == 192 ? launch_tc<192, false>(g, st) : g.N == 128 ? launch_tc<128, false>(g, st) : launch_tc<64, false>(g, st);
}

int read_tc_error(int* out, int clear) {
  cudaError_t e = cudaMemcpyFromSymbol(out, g_tc_error, sizeof(int));
  if (e == cudaSuccess && clear && *out != 0) {
    const int zero = 0;
    e = cudaMemcpyToSymbol(g_tc_error, &zero, sizeof(int));
  }
  if (e != cudaSuccess) { set_cuda_error(e); return CSSM_ERR_CUDA; }
  return CSSM_OK;
}

}  // namespace cssm

extern "C" {
int cssm_device_error(int* out, int clear) {
  if (!out) return CSSM_ERR_NULL;
  int a = 0, b = 0;
  int rc = cssm::read_tc_error(&a, clear), a2 = 0;
  if (rc == CSSM_OK) rc = cssm::read_split_error(&a2, clear);
  if (rc != CSSM_OK) return rc;
  a |= a2;
  rc = cssm::read_qt_error(&a2, clear);
  if (rc != CSSM_OK) return rc;
  a |= a2;
  rc = cssm::read_stem_error(&a2, clear);
  if (rc != CSSM_OK) return rc;
  a |= a2;
  rc = cssm::read_spec_error(&b, clear);
  if (rc != CSSM_OK) return rc;
  int b2 = 0;
  rc = cssm::read_p32_error(&b2, clear);
  if (rc != CSSM_OK) return rc;
  b |= b2;
  rc = cssm::read_p64_error(&b2, clear);
  if (rc != CSSM_OK) return rc;
  b |= b2;
  int c = 0, m = 0;
  rc = cssm::read_bf16_error(&c, clear);
  if (rc != CSSM_OK) return rc;
  rc = cssm::read_mlp_error(&m, clear);
  // low byte: fp32 tensor-core GEMMs and stem, next byte: fused spectral kernels, third: bf16 GEMM, fourth: fused MLP
  *out = a | (b << 8) | (c << 16) | (m << 24);
  return rc;
}
}
