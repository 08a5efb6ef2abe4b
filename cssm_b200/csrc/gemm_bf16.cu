// bf16 tcgen05 / TMEM GEMM with a K loop, for the channel contractions of the CSSM-SHViT model
// (Dense layers with K = 64 ... 1536, and the 3x3 stride-2 ConvBN layers as implicit GEMMs).
//
//   out[m, n] = act( sum_k A[m, k] * Wt[n, k] + bias[n] ) (+ res[m, n]),  bf16 in, fp32 accumulate.
//
// Persistent kernel, one CTA per SM, 18 warps (14 in the im2col form), warp-specialised:
//   warp 0     TMA producer: one lane issues cp.async.bulk.tensor loads of the A tile (128 rows x
//              64 k, plain mode) and the weight tile (BN rows x 64 k) of every K block into a
//              ring of 128-byte-swizzled K-major operand tiles (as many stages as there is room for, at most eight);
//   warp 1     MMA issuer: one lane issues 4 tcgen05.mma.kind::f16 (M128 x BN x K16) per K block
//              into one of four TMEM accumulators (BN <= 128; two for wider single tiles);
//              tcgen05.commit frees the stage / publishes the accumulator;
//   warps 2-17 epilogue, four warps per TMEM lane quadrant: tcgen05.ld (lane = output row), bias (from shared
//              memory), GELU / SiLU, residual; each half (two warps per quadrant) owns every other tile and half of the
//              accumulators.  Without a residual by TMA a warp has its 32 rows of every other box of 64 columns, a 4 KB
//              staging slot in the 128-byte swizzle and TMA tensor stores of its own and waits for no other warp.  With
//              one, and in conv mode, the half shares boxes of 128 rows x 64 columns in a ring of two to four slots
//              (a warp 32 of the columns) with a barrier before the store; the residual box is fetched by TMA into the
//              slot it will be staged in, two boxes ahead, and added in place (N a multiple of 64; otherwise direct
//              16-byte loads and stores).  The im2col form has eight epilogue warps;
//   4 more     im2col producers (conv mode only): eight consecutive lanes fetch the eight 16-byte
//              channel chunks of one output pixel's K block from the channels-last input (zero
//              outside the image), four pixels per warp instruction, and write them in the same
//              swizzled layout; the loads of the next two K blocks are in flight meanwhile.
// With eight warps, a barrier a box and the bias read from global memory behind every accumulator load the epilogue was a chain of
// waits (GELU, 128 x 256 tiles: issue slots 40 % busy, special-function pipe 37 %, most stalls on loads and barriers).  M x K -> N, us:
// 401408 x 128 -> 512 GELU 152 -> 107, 100352 x 256 -> 1024 GELU 94 -> 75, 100352 x 256 -> 512 SiLU 55 -> 45, 25088 x 384 -> 1536 GELU
// 49 -> 41, 25088 x 1536 -> 384 + residual 50 -> 47; sixteen warps alone 148, 90, 53, 47, 48.
// Every mbarrier wait is bounded; on expiry the kernel records an error code (cssm_device_error)
// and winds down.  No multicast, no cluster: each CTA loads its own tiles.
#include <cuda.h>
#include <cuda_bf16.h>
#include <string.h>
#include "kernels.cuh"
#include "tc05.cuh"
#include "bf16_ops.cuh"
#include "gemm_bf16_room.h"

namespace cssm {

__device__ int g_bf16_error = 0;

// Epilogue warps: sixteen; eight beside the gathering warps of the im2col form, which need the registers.
template <bool IM2COL> constexpr int gb_epi_warps = IM2COL ? 8 : 16;
template <bool IM2COL> constexpr int gb_threads = (2 + gb_epi_warps<IM2COL> + (IM2COL ? 4 : 0)) * 32;

__device__ __forceinline__ uint32_t make_idesc_bf16(uint32_t M, uint32_t N) {
  uint32_t d = 0;
  d |= 1u << 4;            // D format: f32
  d |= 1u << 7;            // A format: bf16
  d |= 1u << 10;           // B format: bf16
  d |= (N >> 3) << 17;     // N / 8
  d |= (M >> 4) << 24;     // M / 16
  return d;
}
__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc,
                                         uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}

// RTMA (with TMA_OUT): the residual boxes come by TMA into the staging slots.
// ROWS (with TMA_OUT, plain GEMMs): every epilogue warp stages and stores boxes of its own 32 rows.
template <bool IM2COL, bool TMA_OUT, bool RTMA, bool ROWS = false>
__global__ void __launch_bounds__(gb_threads<IM2COL>, 1)
gemm_bf16_kernel(const Bf16GemmArgs g, const __grid_constant__ CUtensorMap amap,
                 const __grid_constant__ CUtensorMap bmap, const __grid_constant__ CUtensorMap omap,
                 const __grid_constant__ CUtensorMap rmap) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned char* smem = smem_raw + ((1024u - (tc::smem_u32(smem_raw) & 1023u)) & 1023u);
  const uint32_t sbase = tc::smem_u32(smem);
  const uint32_t BN = (uint32_t)g.BN;
  // wres: the whole weight matrix (one N tile, all K blocks) stays in shared memory for the life of
  // the CTA and the ring carries only the A tiles
  const bool wres = g.wres != 0;
  const uint32_t wres_bytes = wres ? (uint32_t)(g.Kpad / GB_BK) * BN * 128u : 0u;
  const uint32_t stage_bytes = GB_A_BYTES + (wres ? 0u : BN * 128u);
  const int NS = g.stages;                                  // ring depth (3 when BN = 256 and TMA_OUT)
  unsigned char* ring = smem + wres_bytes;
  unsigned char* out_s = ring + (uint32_t)NS * stage_bytes; // TMA_OUT: 2 x ostg staging boxes of 16 KB
  uint64_t* bars = reinterpret_cast<uint64_t*>(out_s + (TMA_OUT ? (uint32_t)(2 * g.ostg) * 16384u : 0u));
  uint64_t* full = bars;                        // [8] operands landed
  uint64_t* empty = bars + GB_MAX_STAGES;       // [8] stage consumed
  uint64_t* accfull = bars + 2 * GB_MAX_STAGES; // [4] accumulator complete
  uint64_t* accempty = accfull + 4;             // [4] accumulator drained
  uint64_t* resfull = accempty + 4;             // [2][4] residual box landed in its staging slot
  uint64_t* done = resfull + 8;
  uint64_t* wfull = done + 1;                   // resident weights landed
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(wfull + 1);
  float* bias_s = reinterpret_cast<float*>(bars + GB_BAR_BYTES / 8);      // the bias, where it fits (g.bias_n values)
  const int NACC = g.nacc;                                  // TMEM accumulators: 4 of BN <= 128 columns, else 2

  constexpr int EW = gb_epi_warps<IM2COL>, HALF_THREADS = EW * 16, CW = EW / 8;      // CW: warps of a half and lane quadrant
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n_tiles = g.N / g.BN;
  const int m_tiles = g.conv_tma ? g.tiles_w * g.tiles_h * ((g.Bimg + g.Bbox - 1) / g.Bbox) : (g.M + GB_BM - 1) / GB_BM;
  const int num_tiles = m_tiles * n_tiles;
  const int kblocks = g.Kpad / GB_BK;
  uint32_t tmem_cols = 32;
  while (tmem_cols < (uint32_t)NACC * BN) tmem_cols <<= 1;

  if (tid == 0) {
    for (int s = 0; s < NS; ++s) {
      tc::mbar_init(&full[s], IM2COL ? 1 + 4 : 1);      // TMA lane + one lane per producer warp
      tc::mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 4; ++a) {
      tc::mbar_init(&accfull[a], 1);
      // one lane per warp of the half that drains the accumulator
      tc::mbar_init(&accempty[a], EW / 2);
    }
    for (int a = 0; a < 8; ++a) tc::mbar_init(&resfull[a], 1);
    tc::mbar_init(done, 1);
    tc::mbar_init(wfull, 1);
    tc::fence_mbar_init();
  }
  for (int i = tid; i < g.bias_n; i += gb_threads<IM2COL>) bias_s[i] = __ldg(g.bias + i);      // (as the weights: no wait)
  if (warp == 1) {
    tc::tmem_alloc(tmem_slot, tmem_cols);
    tc::tmem_relinquish();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  bool bad = false;

  if (warp == 0) {
    // ================================ TMA producer ================================
    // The whole warp walks the loop with counters in place of divisions, one lane issues (elect_one): a lane that divided its way to every box
    // was itself what the 3x3 convs waited for (780 of 980 clocks a K block).
    // Weights do not depend on the kernel before this one: the resident ones, or the weight tiles of
    // the first ring round, are on their way before the wait for it.
    const uint32_t a_bytes = g.conv_tma ? (uint32_t)(g.Wbox * g.Hbox * g.Bbox) * 128u : GB_A_BYTES;
    int npre = 0;
    if (wres) {
      if (tc::elect_one()) {
        tc::mbar_expect_tx(wfull, wres_bytes);
        for (int kb = 0; kb < kblocks; ++kb) tc::tma_load_2d(smem + (uint32_t)kb * BN * 128u, &bmap, kb * GB_BK, 0, wfull);
      }
      __syncwarp();
    } else if (!IM2COL && blockIdx.x < num_tiles) {
      const int n0 = (blockIdx.x % n_tiles) * g.BN;
      npre = NS < kblocks ? NS : kblocks;
      if (tc::elect_one())
        for (int i = 0; i < npre; ++i) {
          tc::mbar_expect_tx(&full[i], a_bytes + BN * 128u);
          tc::tma_load_2d(ring + (uint32_t)i * stage_bytes + GB_A_BYTES, &bmap, i * GB_BK, n0, &full[i]);
        }
      __syncwarp();
    }
    pdl_sync();
    int s = 0;
    uint32_t sph = 0;
    for (int tile = blockIdx.x; tile < num_tiles && !bad; tile += gridDim.x) {
      const int mt = tile / n_tiles;
      const int m0 = mt * GB_BM, n0 = (tile - mt * n_tiles) * g.BN;
      // conv through TMA: the tile's patch origin (input coordinates of window position (0,0))
      int cw0 = 0, ch0 = 0, cb0 = 0, pr = 0, pc = 0, cb = 0;
      if (g.conv_tma) {
        const int r = mt / g.tiles_w, tw = mt - r * g.tiles_w, b = r / g.tiles_h, th = r - b * g.tiles_h;
        cb0 = b * g.Bbox;
        cw0 = tw * g.Wbox * (g.conv_tma == 2 ? 1 : g.stride) - (g.conv_tma == 2 ? 0 : g.pad_w);
        ch0 = th * g.Hbox * g.stride - g.pad_h;
      }
      for (int kb = 0; kb < kblocks; ++kb) {
        if (__any_sync(0xffffffffu, !tc::mbar_wait(&empty[s], sph ^ 1))) { atomicExch(&g_bf16_error, 5); bad = true; break; }
        unsigned char* a_s = ring + (uint32_t)s * stage_bytes;
        const bool pre = npre > 0;                        // its weight tile is already on the way
        if (tc::elect_one()) {
          if (!pre) tc::mbar_expect_tx(&full[s], (IM2COL ? 0u : a_bytes) + (wres ? 0u : BN * 128u));
          if (g.conv_tma) tc::tma_load_4d(a_s, &amap, cb * GB_BK, cw0 + pc, ch0 + pr, cb0, &full[s]);
          else if (!IM2COL) tc::tma_load_2d(a_s, &amap, kb * GB_BK, m0, &full[s]);
          if (!wres && !pre) tc::tma_load_2d(a_s + GB_A_BYTES, &bmap, kb * GB_BK, n0, &full[s]);
        }
        __syncwarp();
        if (pre) --npre;
        if (g.conv_tma && ++cb == g.kb_per_tap) {
          cb = 0;
          if (++pc == g.pos_w) { pc = 0; ++pr; }
        }
        if (++s == NS) { s = 0; sph ^= 1; }
      }
    }
  } else if (warp == 1) {
    // ================================ MMA issuer ================================
    // The limit of the waits below is for this kernel's own loads: they begin once the producer's wait is over.
    // The whole warp walks the loop, one lane issues (elect_one).
    pdl_wait();
    const uint32_t idesc = make_idesc_bf16(GB_BM, BN);
    if (wres && !tc::mbar_wait(wfull, 0)) { atomicExch(&g_bf16_error, 6); bad = true; }
    bad = __any_sync(0xffffffffu, bad);
    int s = 0, sph = 0, ac = 0, aph = 1;
    for (int tile = blockIdx.x; tile < num_tiles && !bad; tile += gridDim.x) {
      if (__any_sync(0xffffffffu, !tc::mbar_wait(&accempty[ac], aph))) { atomicExch(&g_bf16_error, 6); bad = true; break; }
      tc::fence_after_sync();
      const uint32_t d = tmem_base + (uint32_t)ac * BN;
      for (int kb = 0; kb < kblocks; ++kb) {
        if (__any_sync(0xffffffffu, !tc::mbar_wait(&full[s], sph))) { atomicExch(&g_bf16_error, 6); bad = true; break; }
        tc::fence_after_sync();
        const uint32_t a_s = sbase + wres_bytes + (uint32_t)s * stage_bytes;
        const uint64_t ad = tc::make_desc_sw128(a_s), bd = tc::make_desc_sw128(wres ? sbase + (uint32_t)kb * BN * 128u : a_s + GB_A_BYTES);
        if (tc::elect_one()) {
#pragma unroll
          for (int ks = 0; ks < 4; ++ks) mma_bf16(d, ad + ks * 2, bd + ks * 2, idesc, (kb | ks) ? 1u : 0u);
          tc::commit(&empty[s]);
        }
        __syncwarp();
        if (++s == NS) { s = 0; sph ^= 1; }
      }
      if (bad) break;
      if (tc::elect_one()) tc::commit(&accfull[ac]);
      __syncwarp();
      if (++ac == NACC) { ac = 0; aph ^= 1; }
    }
    // nothing of this warp's tensor work may be in flight when TMEM is freed
    if (tc::elect_one()) tc::commit(done);
    __syncwarp();
    if (!tc::mbar_wait(done, 0) && !bad) atomicExch(&g_bf16_error, 7);
    __syncwarp();
  } else if (warp < 2 + EW) {
    // ================================ epilogue ================================
    // Two halves of eight warps, two per TMEM lane quadrant (im2col: of four).  Half h owns the tiles of its CTA with
    // tile count parity h; accumulator = tile count mod NACC, so a half drains one accumulator while
    // the MMA warp fills its other one.
    const int q = warp & 3;                       // TMEM lane quadrant this warp may read
    const int half = (warp - 2) / (EW / 2);
    const int sub = CW == 1 ? 0 : ((warp - 2) >> 2) & 1;      // CW = 2: which 32 columns of every 64 are this warp's
    const int row = q * 32 + lane;
    const uint32_t tlane = tmem_base + ((uint32_t)(q * 32) << 16);
    pdl_wait();
    // bias, activation on 32 accumulator columns starting at tile column c0
    auto act32 = [&](const uint32_t (&r)[32], int n, float (&v)[32]) {
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
      if (g.bias_n != 0) {
        const float4* bp = reinterpret_cast<const float4*>(bias_s + n);
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
          const float4 b4 = bp[j >> 2];
          v[j] += b4.x; v[j + 1] += b4.y; v[j + 2] += b4.z; v[j + 3] += b4.w;
        }
      } else if (g.bias != nullptr) {
        const float4* bp = reinterpret_cast<const float4*>(g.bias + n);
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
          const float4 b4 = __ldg(bp + (j >> 2));
          v[j] += b4.x; v[j + 1] += b4.y; v[j + 2] += b4.z; v[j + 3] += b4.w;
        }
      }
      if (g.act == 1) {
#pragma unroll
        for (int j = 0; j < 32; j += 2) gelu_tanh_x2(v[j], v[j + 1]);
      } else if (g.act == 2) {
#pragma unroll
        for (int j = 0; j < 32; j += 2) silu_tanh_x2(v[j], v[j + 1]);
      }
    };
    if constexpr (ROWS) {
      // A warp has 32 rows of every other box of 64 columns: it stages them in a 4 KB slot of its own and writes them with a
      // TMA store of its own, so it waits for nobody but the accumulator.
      unsigned char* stg = out_s + (uint32_t)(warp - 2) * 4096u;
      const int nb = g.BN / 64;
      for (int tcnt = half;; tcnt += 2) {
        const int tile = blockIdx.x + tcnt * (int)gridDim.x;
        if (tile >= num_tiles) break;
        const int m0 = (tile / n_tiles) * GB_BM, n0 = (tile % n_tiles) * g.BN;
        const int ac = tcnt % NACC, aph = (tcnt / NACC) & 1;
        const bool has_res = g.res != nullptr && m0 + row < g.M;
        const uint4* rrow = reinterpret_cast<const uint4*>(g.res + (has_res ? (size_t)(m0 + row) * g.ldr + n0 : 0));
        uint4 rs[4];                              // residual of the warp's next 32 columns
        auto fetch_res = [&](int c) {
#pragma unroll
          for (int j = 0; j < 4; ++j) rs[j] = has_res && c < 2 * nb ? __ldg(rrow + c * 4 + j) : make_uint4(0u, 0u, 0u, 0u);
        };
        const int s0 = (sub + (tcnt >> 1)) & (CW - 1);      // (an odd number of boxes: the two warps take the extra one in turn)
        if (g.res != nullptr) fetch_res(2 * s0);
        if (__any_sync(0xffffffffu, !tc::mbar_wait(&accfull[ac], aph))) { atomicExch(&g_bf16_error, 8); break; }
        tc::fence_after_sync();
        const uint32_t taddr = tlane + (uint32_t)ac * BN;
        for (int box = s0; box < nb; box += CW) {
#pragma unroll
          for (int hh = 0; hh < 2; ++hh) {
            uint32_t ra[32];
            float v[32];
            tc::ld_32x32b_x32(taddr + box * 64 + hh * 32, ra);
            tc::wait_ld();
            act32(ra, n0 + box * 64 + hh * 32, v);
            if (g.res != nullptr) {
#pragma unroll
              for (int j4 = 0; j4 < 4; ++j4) {
                float f[8];
                unpack8(rs[j4], f);
#pragma unroll
                for (int e = 0; e < 8; ++e) v[j4 * 8 + e] += f[e];
              }
              fetch_res(hh == 0 ? 2 * box + 1 : 2 * (box + CW));
            }
            if (hh == 0) {
              // the store before has read the slot
              if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
              __syncwarp();
            }
#pragma unroll
            for (int j4 = 0; j4 < 4; ++j4) {
              const float f[8] = {v[j4 * 8], v[j4 * 8 + 1], v[j4 * 8 + 2], v[j4 * 8 + 3],
                                  v[j4 * 8 + 4], v[j4 * 8 + 5], v[j4 * 8 + 6], v[j4 * 8 + 7]};
              *reinterpret_cast<uint4*>(stg + tc::sw128_offset(lane, hh * 4 + j4)) = pack8(f);
            }
          }
          tc::fence_proxy_async();
          __syncwarp();
          if (lane == 0) {
            tc::tma_store_2d(&omap, stg, n0 + box * 64, m0 + q * 32);
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          }
        }
        tc::fence_before_sync();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&accempty[ac]);
      }
      // the slot must outlive the last TMA store that reads it
      if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    } else if constexpr (TMA_OUT) {
      // Output boxes of 128 rows x 64 bf16 columns are staged in the 128-byte swizzle in a ring of D
      // slots per half and written by TMA tensor stores.  A residual is fetched by TMA into the
      // very slot its box will be staged in, D - 2 boxes ahead (the wait before a slot is reused
      // leaves only the most recent store pending), and is added in place.
      // (Both halves draining every tile of a two-accumulator configuration, each every other box,
      // measured slower than whole tiles in turn: 232 against 197 us for M = 1.6 M, K = 64, N = 256.)
      const bool issuer = q == 0 && sub == 0 && lane == 0;    // issues this half's TMA loads and stores
      const int D = g.ostg, nb = g.BN / 64;
      constexpr int b0 = 0, bstep = 1, tstep = 2;
      const int t0 = half;
      unsigned char* stgh = out_s + (uint32_t)(half * D) * 16384u;
      uint64_t* resf = resfull + half * 4;
      constexpr bool rtma = RTMA;
      const bool rreg = !RTMA && g.res != nullptr;      // residual rows by plain loads
      int pf_t = t0, pf_box = b0, pf_q = 0;       // issuer: the next box whose residual is to be fetched
      auto pf_issue = [&]() {
        const int tile = blockIdx.x + pf_t * (int)gridDim.x;
        if (tile >= num_tiles) return;
        const int slot = pf_q % D;
        tc::mbar_expect_tx(&resf[slot], 16384u);
        tc::tma_load_2d(stgh + (uint32_t)slot * 16384u, &rmap, (tile % n_tiles) * g.BN + pf_box * 64,
                        (tile / n_tiles) * GB_BM, &resf[slot]);
        ++pf_q;
        pf_box += bstep;
        if (pf_box >= nb) { pf_box = b0; pf_t += tstep; }
      };
      if (rtma && issuer)
        for (int k = 0; k < D - 2; ++k) pf_issue();
      // all threads of the half agree on `ok` (and meet, as a barrier)
      auto all_ok = [&](bool ok) {
        uint32_t r;
        asm volatile(
            "{\n\t.reg .pred p, q;\n\t"
            "setp.ne.u32 p, %1, 0;\n\t"
            "bar.red.and.pred q, %2, %3, p;\n\t"
            "selp.u32 %0, 1, 0, q;\n\t}"
            : "=r"(r) : "r"((uint32_t)ok), "r"(1 + half), "n"(HALF_THREADS) : "memory");
        return r != 0;
      };
      int bq = 0;                                 // boxes staged by this half so far
      bool live = true;
      for (int tcnt = t0; live; tcnt += tstep) {
        const int tile = blockIdx.x + tcnt * (int)gridDim.x;
        if (tile >= num_tiles) break;
        const int m0 = (tile / n_tiles) * GB_BM, n0 = (tile % n_tiles) * g.BN;
        const int ac = tcnt % NACC, aph = (tcnt / NACC) & 1;
        const bool has_res = rreg && m0 + row < g.M;
        const uint4* rrow = reinterpret_cast<const uint4*>(g.res + (has_res ? (size_t)(m0 + row) * g.ldr + n0 : 0));
        uint4 rs[8 / CW];                         // rreg: residual of this warp's part of the next 64 columns
        auto fetch_res = [&](int c0) {
#pragma unroll
          for (int j = 0; j < 8 / CW; ++j) rs[j] = has_res ? __ldg(rrow + (c0 >> 3) + sub * 4 + j) : make_uint4(0u, 0u, 0u, 0u);
        };
        if (rreg) fetch_res(0);
        if (!all_ok(tc::mbar_wait(&accfull[ac], aph))) { atomicExch(&g_bf16_error, 8); break; }
        tc::fence_after_sync();
        const uint32_t taddr = tlane + (uint32_t)ac * BN;
        uint32_t ra[32];
        for (int box = b0; box < nb; box += bstep, ++bq) {
          const int slot = bq % D;
          unsigned char* stg = stgh + (uint32_t)slot * 16384u;
          // residual by TMA: its box landed in this slot two boxes ago (a wait that expires is
          // recorded and the data is wrong, but every thread still meets the barriers below)
          if (rtma && !tc::mbar_wait(&resf[slot], (bq / D) & 1)) atomicExch(&g_bf16_error, 8);
          // accumulator -> bias, activation, residual -> eight packed 16-byte chunks.  Nothing here
          // writes the slot, so it runs while the earlier stores drain.  (Keeping the TMEM load of the
          // next 32 columns in flight during the arithmetic measured slower.)
          uint4 pk[8 / CW];
#pragma unroll
          for (int i = 0; i < 2 / CW; ++i) {
            const int hh = CW == 1 ? i : sub;
            float v[32];
            tc::ld_32x32b_x32(taddr + box * 64 + hh * 32, ra);
            tc::wait_ld();
            act32(ra, n0 + box * 64 + hh * 32, v);
            if (rtma || rreg) {
#pragma unroll
              for (int j4 = 0; j4 < 4; ++j4) {
                float f[8];
                unpack8(rtma ? *reinterpret_cast<const uint4*>(stg + tc::sw128_offset(row, hh * 4 + j4))
                             : rs[i * 4 + j4], f);
#pragma unroll
                for (int e = 0; e < 8; ++e) v[j4 * 8 + e] += f[e];
              }
            }
#pragma unroll
            for (int j4 = 0; j4 < 4; ++j4) {
              const float f[8] = {v[j4 * 8], v[j4 * 8 + 1], v[j4 * 8 + 2], v[j4 * 8 + 3],
                                  v[j4 * 8 + 4], v[j4 * 8 + 5], v[j4 * 8 + 6], v[j4 * 8 + 7]};
              pk[i * 4 + j4] = pack8(f);
            }
          }
          if (issuer) {
            // the store that last read the slot about to be refilled has drained: with a residual
            // that slot is the one of two boxes back, else this box's own (D boxes back)
            if (rtma || D < 3) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
            else if (D == 3) asm volatile("cp.async.bulk.wait_group.read 2;" ::: "memory");
            else asm volatile("cp.async.bulk.wait_group.read 3;" ::: "memory");
            if (rtma) pf_issue();
          }
          // without the TMA residual the slot's last reader is only known to the issuer; with it
          // every thread rewrites just its own row of the box it has read
          if (!rtma) asm volatile("bar.sync %0, %1;" ::"r"(1 + half), "n"(HALF_THREADS) : "memory");
          if (rreg && box + 1 < nb) fetch_res((box + 1) * 64);
#pragma unroll
          for (int c = 0; c < 8 / CW; ++c)
            *reinterpret_cast<uint4*>(stg + tc::sw128_offset(row, sub * 4 + c)) = pk[c];
          tc::fence_proxy_async();
          asm volatile("bar.sync %0, %1;" ::"r"(1 + half), "n"(HALF_THREADS) : "memory");
          if (issuer) {
            if (g.conv_tma) {
              const int mt = tile / n_tiles;
              const int tw = mt % g.tiles_w, th = (mt / g.tiles_w) % g.tiles_h;
              tc::tma_store_4d(&omap, stg, n0 + box * 64, tw * g.Wbox, th * g.Hbox,
                               (mt / (g.tiles_w * g.tiles_h)) * g.Bbox);
            } else {
              tc::tma_store_2d(&omap, stg, n0 + box * 64, m0);
            }
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          }
        }
        if (!live) break;
        tc::fence_before_sync();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&accempty[ac]);
      }
      // the staging slots must outlive the last TMA stores that read them
      if (issuer) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    } else {
      // direct 16-byte stores (N not a multiple of 64, or no tensor map): residual rows by plain loads
      for (int i = 0;; ++i) {
        const int tcnt = 2 * i + half;
        const int tile = blockIdx.x + tcnt * (int)gridDim.x;
        if (tile >= num_tiles) break;
        const int m0 = (tile / n_tiles) * GB_BM, n0 = (tile % n_tiles) * g.BN;
        const int ac = tcnt % NACC, aph = (tcnt / NACC) & 1;
        const int m = m0 + row;
        const bool has_res = g.res != nullptr && m < g.M;
        const uint4* rrow = reinterpret_cast<const uint4*>(g.res + (has_res ? (size_t)m * g.ldr + n0 : 0));
        uint4 rs[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) rs[j] = has_res && sub * 32 < g.BN ? __ldg(rrow + sub * 4 + j) : make_uint4(0u, 0u, 0u, 0u);
        if (__any_sync(0xffffffffu, !tc::mbar_wait(&accfull[ac], aph))) { atomicExch(&g_bf16_error, 8); break; }
        tc::fence_after_sync();
        const uint32_t taddr = tlane + (uint32_t)ac * BN;
        uint32_t ra[32];
        for (int c0 = sub * 32; c0 < g.BN; c0 += 32 * CW) {
          float v[32];
          tc::ld_32x32b_x32(taddr + c0, ra);
          tc::wait_ld();
          act32(ra, n0 + c0, v);
#pragma unroll
          for (int j4 = 0; j4 < 4; ++j4) {
            float f[8];
            unpack8(rs[j4], f);
#pragma unroll
            for (int e = 0; e < 8; ++e) v[j4 * 8 + e] += f[e];
          }
          if (c0 + 32 * CW < g.BN) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
              rs[j] = has_res ? __ldg(rrow + ((c0 + 32 * CW) >> 3) + j) : make_uint4(0u, 0u, 0u, 0u);
          }
          if (m < g.M) {
            uint4* op = reinterpret_cast<uint4*>(g.out + (size_t)m * g.ldo + n0 + c0);
#pragma unroll
            for (int j4 = 0; j4 < 4; ++j4) {
              const float f[8] = {v[j4 * 8], v[j4 * 8 + 1], v[j4 * 8 + 2], v[j4 * 8 + 3],
                                  v[j4 * 8 + 4], v[j4 * 8 + 5], v[j4 * 8 + 6], v[j4 * 8 + 7]};
              op[j4] = pack8(f);
            }
          }
        }
        tc::fence_before_sync();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&accempty[ac]);
      }
    }
  } else if (IM2COL) {
    // ================================ im2col producers ================================
    pdl_wait();
    // lane = (row group rg, chunk c): the eight lanes of a group read the eight 16-byte chunks of one
    // output pixel's K block (contiguous channels of one or two taps); thread handles rows rg + 16 i.
    const int pt = tid - (2 + EW) * 32;           // 0..127
    const int c = pt & 7, rg = pt >> 3;
    const int HWo = g.Ho * g.Wo;
    int it = 0;
    for (int tile = blockIdx.x; tile < num_tiles && !bad; tile += gridDim.x) {
      const int mt = (tile / n_tiles) * GB_BM;
      int hi0[8], wi0[8], pb[8];                    // window origin and first pixel of the image
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int m = mt + rg + 16 * i;
        const bool live = m < g.M;
        const int b = live ? m / HWo : 0;
        const int px = live ? m - b * HWo : 0;
        const int ho = px / g.Wo, wo = px - ho * g.Wo;
        hi0[i] = live ? ho * g.stride - g.pad_h : -100000;     // dead rows fail the bounds test
        wi0[i] = wo * g.stride - g.pad_w;
        pb[i] = b * g.Hi * g.Wi;
      }
      auto gather = [&](int kb, uint4 (&v)[8]) {
        const int k0 = kb * GB_BK + c * 8;
        const int tap = k0 / g.Cin, c0 = k0 - tap * g.Cin;
        const int ti = tap / g.ksz, tj = tap - ti * g.ksz;
        const bool kin = kb < kblocks && k0 < g.K;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int hi = hi0[i] + ti, wi = wi0[i] + tj;
          const bool in = kin && hi >= 0 && hi < g.Hi && wi >= 0 && wi < g.Wi;
          v[i] = in ? __ldg(reinterpret_cast<const uint4*>(g.A + (size_t)(pb[i] + hi * g.Wi + wi) * g.Cin + c0))
                    : make_uint4(0u, 0u, 0u, 0u);
        }
      };
      // register ring two K blocks deep
      uint4 r0[8], r1[8], r2[8];
      gather(0, r0);
      gather(1, r1);
      for (int kb = 0; kb < kblocks && !bad; kb += 3) {
        // three blocks per trip so that the ring slots keep compile-time names
#pragma unroll
        for (int u = 0; u < 3; ++u) {
          if (kb + u >= kblocks) break;
          uint4 (&cur)[8] = u == 0 ? r0 : (u == 1 ? r1 : r2);
          uint4 (&nxt)[8] = u == 0 ? r2 : (u == 1 ? r0 : r1);
          gather(kb + u + 2, nxt);
          const int s = it % NS;
          if (__any_sync(0xffffffffu, !tc::mbar_wait(&empty[s], ((it / NS) & 1) ^ 1))) { atomicExch(&g_bf16_error, 9); bad = true; break; }
          unsigned char* a_s = ring + (uint32_t)s * stage_bytes;
#pragma unroll
          for (int i = 0; i < 8; ++i)
            *reinterpret_cast<uint4*>(a_s + tc::sw128_offset(rg + 16 * i, c)) = cur[i];
          tc::fence_proxy_async();
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(&full[s]);
          ++it;
        }
      }
    }
  }
  // error path only: give copies that may still be in flight a bounded time to land
  if (bad)
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem_base, tmem_cols);
  }
}

// K-major bf16 matrix [rows][kcols] (row stride ld elements) -> boxes of 64 k x box_rows rows
static bool make_kmajor_map(CUtensorMap* map, const void* base, uint64_t rows, uint64_t kcols,
                            uint64_t ld, uint32_t box_rows) {
  const tc::EncodeTiledFn enc = tc::encode_fn();
  if (!enc) return false;
  const cuuint64_t dims[2] = {kcols, rows};
  const cuuint64_t strides[1] = {ld * 2};
  const cuuint32_t box[2] = {64, box_rows}, es[2] = {1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, es,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
             CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int read_bf16_error(int* out, int clear) {
  cudaError_t e = cudaMemcpyFromSymbol(out, g_bf16_error, sizeof(int));
  if (e == cudaSuccess && clear && *out != 0) {
    const int zero = 0;
    e = cudaMemcpyToSymbol(g_bf16_error, &zero, sizeof(int));
  }
  if (e != cudaSuccess) { set_cuda_error(e); return CSSM_ERR_CUDA; }
  return CSSM_OK;
}

// (rows x cols) bf16 output with row stride ld -> boxes of 64 columns x 128 rows for the TMA stores
static bool make_out_map(CUtensorMap* map, void* base, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows = 128) {
  const tc::EncodeTiledFn enc = tc::encode_fn();
  if (!enc) return false;
  const cuuint64_t dims[2] = {cols, rows};
  const cuuint64_t strides[1] = {ld * 2};
  const cuuint32_t box[2] = {64, box_rows}, es[2] = {1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, base, dims, strides, box, es,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
             CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// 4-D bf16 tensor (d0 innermost) with byte strides st[0..2] of dims 1..3, boxes and traversal strides
static bool make_map_4d(CUtensorMap* map, const void* base, const uint64_t (&dims)[4], const uint64_t (&st)[3],
                        const uint32_t (&box)[4], const uint32_t (&es)[4]) {
  const tc::EncodeTiledFn enc = tc::encode_fn();
  if (!enc) return false;
  const cuuint64_t d[4] = {dims[0], dims[1], dims[2], dims[3]};
  const cuuint64_t s[3] = {st[0], st[1], st[2]};
  const cuuint32_t b[4] = {box[0], box[1], box[2], box[3]};
  const cuuint32_t e[4] = {es[0], es[1], es[2], es[3]};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), d, s, b, e,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
             CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int conv3x3s2_weight_layout(int Cin, int Wi, int Cout) { return (Cin == 32 && Wi % 2 == 0 && Cout % 64 == 0) ? 1 : 0; }
int conv3x3s2_packed_k(int Cin, int Wi, int Cout) { return conv3x3s2_weight_layout(Cin, Wi, Cout) ? 384 : 9 * Cin; }

int launch_gemm_bf16(Bf16GemmArgs g, cudaStream_t st) {
  if (g.M <= 0 || g.N <= 0 || g.K <= 0) return CSSM_ERR_DIMS;
  const bool conv = g.ksz > 0;
  const int wide = conv ? conv3x3s2_weight_layout(g.Cin, g.Wi, g.N) : 0;
  // 3x3 stride-2 convs with 64-channel K blocks go through strided TMA boxes (no gather warps)
  g.conv_tma = 0;
  if (conv && g.ksz == 3 && g.stride == 2 && g.N % 64 == 0 && g.res == nullptr && (wide || g.Cin % 64 == 0))
    g.conv_tma = wide ? 2 : 1;
  const int Kw = conv ? conv3x3s2_packed_k(g.Cin, g.Wi, g.N) : g.K;      // K as the packed weights lay it out
  g.Kpad = (Kw + GB_BK - 1) / GB_BK * GB_BK;
  g.BN = gb_columns(g.N, g.K, g.res != nullptr);
  if (g.BN == 0 || g.ldw < g.Kpad || (g.ldw % 8) != 0) return CSSM_ERR_UNSUPPORTED;
  if (g.ldo % 8 != 0 || (g.res != nullptr && g.ldr % 8 != 0)) return CSSM_ERR_UNSUPPORTED;
  if (!aligned16(g.A) || !aligned16(g.Wt) || (g.out && !aligned16(g.out)) ||
      (g.out_f32 && !aligned16(g.out_f32)) || (g.res && !aligned16(g.res)))
    return CSSM_ERR_ALIGN;
  if (g.out_f32 != nullptr || g.out == nullptr) return CSSM_ERR_UNSUPPORTED;
  const bool im2col = conv && !g.conv_tma;
  if (conv) {
    if (g.Cin % 8 != 0 || g.K != g.ksz * g.ksz * g.Cin) return CSSM_ERR_UNSUPPORTED;
    if (wide && !g.conv_tma) return CSSM_ERR_UNSUPPORTED;          // the wide weight layout has no gather path
  } else if (g.K % 8 != 0 || g.lda % 8 != 0 || g.lda < g.K) {
    return CSSM_ERR_UNSUPPORTED;
  }
  if (gemm_small_supported(g)) return launch_gemm_small(g, nullptr, nullptr, st);
  CUtensorMap amap, bmap, omap, rmap;
  memset(&amap, 0, sizeof(amap));
  memset(&bmap, 0, sizeof(bmap));
  memset(&omap, 0, sizeof(omap));
  memset(&rmap, 0, sizeof(rmap));
  bool tma_out = g.BN % 64 == 0;
  int m_tiles = (g.M + GB_BM - 1) / GB_BM;
  const int sms = sm_count();
  if (g.conv_tma) {
    // M tile = Bbox images x Hbox output rows x Wbox output columns, at most 128 pixels
    g.Bimg = g.M / (g.Ho * g.Wo);
    g.tiles_w = (g.Wo + 127) / 128;
    g.Wbox = (g.Wo + g.tiles_w - 1) / g.tiles_w;
    const int hmax = 128 / g.Wbox > 0 ? 128 / g.Wbox : 1;
    g.tiles_h = (g.Ho + hmax - 1) / hmax;
    g.Hbox = (g.Ho + g.tiles_h - 1) / g.tiles_h;
    g.Bbox = (g.tiles_w == 1 && g.tiles_h == 1) ? 128 / (g.Wbox * g.Hbox) : 1;
    if (g.Bbox > g.Bimg) g.Bbox = g.Bimg;
    if (g.Bbox < 1) g.Bbox = 1;
    m_tiles = g.tiles_w * g.tiles_h * ((g.Bimg + g.Bbox - 1) / g.Bbox);
    g.BN = gb_narrow(g.BN, g.N, m_tiles, sms);
    const uint64_t C = (uint64_t)g.Cin;
    bool ok;
    if (g.conv_tma == 2) {
      // pairs of adjacent input pixels as 64-channel "wide pixels": window columns {0,1} and {2,(3)}
      const uint64_t W2 = (uint64_t)g.Wi / 2;
      const uint64_t dims[4] = {64, W2, (uint64_t)g.Hi, (uint64_t)g.Bimg};
      const uint64_t stb[3] = {128, W2 * 128, (uint64_t)g.Hi * W2 * 128};
      const uint32_t box[4] = {64, (uint32_t)g.Wbox, (uint32_t)g.Hbox * 2, (uint32_t)g.Bbox};
      const uint32_t es[4] = {1, 1, 2, 1};
      ok = make_map_4d(&amap, g.A, dims, stb, box, es);
      g.kb_per_tap = 1; g.pos_w = 2;
    } else {
      const uint64_t dims[4] = {C, (uint64_t)g.Wi, (uint64_t)g.Hi, (uint64_t)g.Bimg};
      const uint64_t stb[3] = {C * 2, (uint64_t)g.Wi * C * 2, (uint64_t)g.Hi * g.Wi * C * 2};
      const uint32_t box[4] = {64, (uint32_t)g.Wbox * 2, (uint32_t)g.Hbox * 2, (uint32_t)g.Bbox};
      const uint32_t es[4] = {1, 2, 2, 1};
      ok = make_map_4d(&amap, g.A, dims, stb, box, es);
      g.kb_per_tap = g.Cin / 64; g.pos_w = 3;
    }
    const uint64_t N = (uint64_t)g.N;
    const uint64_t odims[4] = {N, (uint64_t)g.Wo, (uint64_t)g.Ho, (uint64_t)g.Bimg};
    const uint64_t ost[3] = {(uint64_t)g.ldo * 2, (uint64_t)g.Wo * g.ldo * 2, (uint64_t)g.Ho * g.Wo * g.ldo * 2};
    const uint32_t obox[4] = {64, (uint32_t)g.Wbox, (uint32_t)g.Hbox, (uint32_t)g.Bbox};
    const uint32_t oes[4] = {1, 1, 1, 1};
    ok = ok && make_map_4d(&omap, g.out, odims, ost, obox, oes);
    if (!ok) return CSSM_ERR_CUDA;
  } else {
    g.BN = gb_narrow(g.BN, g.N, m_tiles, sms);
    // A: out-of-range k columns (K < Kpad) and rows (M not a multiple of 128) arrive as zeros
    if (!im2col && !make_kmajor_map(&amap, g.A, (uint64_t)g.M, (uint64_t)g.K, (uint64_t)g.lda, GB_BM))
      return CSSM_ERR_CUDA;
    // (boxes of 32 rows: see ROWS)
    const bool boxes128 = im2col || (g.res != nullptr && g.BN <= 128);
    tma_out = tma_out && make_out_map(&omap, g.out, (uint64_t)g.M, (uint64_t)g.N, (uint64_t)g.ldo, boxes128 ? 128 : 32);
    if (tma_out && g.res != nullptr && g.BN <= 128)
      tma_out = make_out_map(&rmap, const_cast<__nv_bfloat16*>(g.res), (uint64_t)g.M, (uint64_t)g.N, (uint64_t)g.ldr);
  }
  if (!make_kmajor_map(&bmap, g.Wt, (uint64_t)g.N, (uint64_t)g.Kpad, (uint64_t)g.ldw, (uint32_t)g.BN))
    return CSSM_ERR_CUDA;
  cudaError_t e;
  const int tiles = m_tiles * (g.N / g.BN);
  const int grid = tiles < sms ? tiles : sms;
  const bool rtma = tma_out && g.res != nullptr && !conv && g.BN <= 128;
  const Bf16Room room = gb_room({g.N, g.BN, g.Kpad, tiles / grid, im2col, tma_out, g.res != nullptr, rtma, g.act != 0, g.bias != nullptr,
                                 aligned16(g.bias)});
  if (room.bytes == 0) return CSSM_ERR_UNSUPPORTED;
  if (g.bias != nullptr && room.bias_n == 0 && !aligned16(g.bias)) return CSSM_ERR_ALIGN;
  g.wres = room.wres; g.stages = room.stages; g.ostg = room.ostg; g.bias_n = room.bias_n;
  // Residual by TMA (plain GEMMs with tiles of at most 128 columns): four accumulators.  Everything else: two, residual rows (if any)
  // by plain loads -- the configuration that measured best without a residual.
  g.nacc = rtma ? 4 : 2;
  const size_t smem = room.bytes;
  auto kern = im2col ? (tma_out ? gemm_bf16_kernel<true, true, false> : gemm_bf16_kernel<true, false, false>)
                     : (tma_out ? (rtma ? gemm_bf16_kernel<false, true, true> : conv ? gemm_bf16_kernel<false, true, false> : gemm_bf16_kernel<false, true, false, true>)
                                : gemm_bf16_kernel<false, false, false>);
  e = func_smem(kern, smem);
  if (e != cudaSuccess) { set_cuda_error(e); return CSSM_ERR_CUDA; }
  launch_k(kern, grid, im2col ? gb_threads<true> : gb_threads<false>, smem, st, g, amap, bmap, omap, rmap);
  return check_launch();
}

}  // namespace cssm
