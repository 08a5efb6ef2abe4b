// GDN fused spectral kernel for 32x32 planes, d_k = d_v = 4: persistent CTAs of 16 warps, one per SM, that stream the steps of one
// (batch, head) after another through two kinds of warps, which hand over by mbarriers:
//   warps 9-15  transforms, dealt out in turn, eight tasks a step: forward of two of the twelve planes q, k, v (TMA a step ahead,
//               rows, columns; csrc/fft32.cuh: whole FFTs in a lane's registers) into one of two sets of spectra, and inverse of
//               two of the step before's output planes (columns, rows, TMA store over the v planes);
//   warps 0-8   bins: a lane owns two frequency bins with their 4x4 states (64 registers), normalises k and q as it reads
//               them, updates all four rows of both bins (packed f32x2 over pairs of rows), writes the readout's spectrum.
// (16 warps at 128 registers a thread; a seventeenth would leave 96.)
// So a plane crosses shared memory six times (in, rows out, columns in and out, bins, and no exchange inside an FFT), the states
// never leave the registers, and while the bins of a step are updated the next step is transformed.
// Bound: issue and instruction fetch with four warps a scheduler (20 K warp instructions a step, issue slots 55 % busy, no warp waits
// for another for more than a tenth of its time).  The kernel before shared every FFT among four lanes, kept the states in L2 and
// was bound by the shared-memory pipe and its barriers: 128 x 32 x 32 x 32 x 64 3853 -> 2346 us.  Taken back: an inverse warp
// beside six forward ones (2544: it sets the pace), one copy of the FFT per pass (2494), the inverse a step later (2449).
// It is ahead of that kernel at every number of heads and steps (a block's pass, us): one head, T = 1 52 -> 48, T = 32 380 -> 222; 64 heads
// 62 -> 58 and 519 -> 337; 148 heads 66 -> 64 and 1035 -> 851; 160 heads 72 -> 68 and 882 -> 640.
// Every wait is bounded; on expiry the kernel records an error code (cssm_device_error) and winds down.
//
// The same stream serves the scalar delta rule of the DeltaNet block with per-channel gates (DN): a "head" is four channels, whose q,
// k and v planes and outputs take the places of the four rows, and a bin's state is one number a channel.  24 x 12 x 32 x 32 x 64:
// 337 -> 194 us.  (Gate maps over the bins scale k before its norm is taken, which the row pass here cannot see:
// csrc/deltanet_spectral_r32.cu.)

// Complex adds as scalar pairs: a lane's FFT is all register renaming then, where packed adds want their operands in aligned
// register pairs and the moves for that cost more than the issue slots they save (2368 -> 2346 us).
#define CSSM_F32X2 0
#include <cuda.h>
#include <string.h>
#include "fft32.cuh"
#include "kernels.cuh"
#include "bf16_ops.cuh"
#include "tc05.cuh"

namespace cssm {

__device__ int g_p32_error = 0;

constexpr int GP_THREADS = 16 * 32, GP_FFT = 9, GP_NFFT = 7;
constexpr uint32_t GP_RAW_OFF = 0;                                         // [6] pairs of planes
constexpr uint32_t GP_OUT_OFF = GP_RAW_OFF + 6u * P32_RAW;                 // [2][2] pairs of output spectra, then their staged planes
constexpr uint32_t GP_OUT_BYTES = 9216;                                    // >= 2 P32_PLANE_CF * 8 and P32_RAW, a multiple of 1024
constexpr uint32_t GP_SPEC_OFF = GP_OUT_OFF + 4u * GP_OUT_BYTES;           // [2][12 planes]
constexpr uint32_t GP_BAR_OFF = GP_SPEC_OFF + 24u * P32_PLANE_CF * 8u;
constexpr uint32_t GP_SMEM = GP_BAR_OFF + 256u;
static_assert(GP_OUT_BYTES >= 2 * P32_PLANE_CF * 8 && GP_SMEM + 1024 <= 227 * 1024, "one CTA per SM");

struct P32Args {
  float* qkv; const cf* what;
  const float2* ab; int ab_heads;              // GDN: gate maps
  const float2* chan; float rho, floor_mag;    // DeltaNet: (BT, C) {alpha, beta}
  int B, T, C, use_l2;
};

// LAST: only the last step's output planes are produced: the q planes, the readout and the inverse of earlier steps are skipped.
template <bool LAST, bool DN>
__global__ void __launch_bounds__(GP_THREADS, 1) gdn_spectral_p32(const P32Args a, const __grid_constant__ CUtensorMap map) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned char* smem = smem_raw + ((1024u - (tc::smem_u32(smem_raw) & 1023u)) & 1023u);
  uint64_t* raw_full = reinterpret_cast<uint64_t*>(smem + GP_BAR_OFF);     // [6]
  uint64_t* spec_full = raw_full + 6;                                      // [2] the step's spectra are complete (6 tasks)
  uint64_t* spec_empty = spec_full + 2;                                    // [2] and have been read (9 warps)
  uint64_t* out_full = spec_empty + 2;                                     // [2][2] a pair of output spectra is complete (9 warps)
  uint64_t* out_empty = out_full + 4;                                      // [2][2] and stored
  __shared__ __align__(16) float nrm[2][8];                                // scales of the q and k planes
  __shared__ volatile int armed[6];                                        // copies issued for each pair of planes
  __shared__ int s_bad;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr int DK = 4, NB = 32 * 17;
  const int nh = a.C / DK, heads = a.B * nh, T = a.T;
  if (tid == 0) {
    for (int i = 0; i < 6; ++i) tc::mbar_init(&raw_full[i], 1);
    for (int i = 0; i < 2; ++i) { tc::mbar_init(&spec_full[i], 6); tc::mbar_init(&spec_empty[i], 9); }
    for (int i = 0; i < 4; ++i) { tc::mbar_init(&out_full[i], 9); tc::mbar_init(&out_empty[i], 1); }
    for (int i = 0; i < 6; ++i) armed[i] = 0;
    tc::fence_mbar_init();
    s_bad = 0;
  }
  __syncthreads();
  pdl_sync();
  const int mine = (heads - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;      // heads of this CTA
  // all lanes of a warp agree
  auto wait = [&](uint64_t* bar, uint32_t phase, int code) {
    const bool ok = !__any_sync(0xffffffffu, !tc::mbar_wait_spin(bar, phase));
    if (!ok) { if (lane == 0) atomicExch(&g_p32_error, code); s_bad = 1; }
    return ok;
  };

  if (warp >= GP_FFT) {
    // ================================ transforms ================================
    const int pl = lane >> 4, j = lane & 15, steps = mine * T;
    // planes of pair p (q 0 1, k 2 3, v 4 5) of step s -> raw buffer p
    auto load = [&](int p, int s) {
      const int hi = s / T, t = s - hi * T, head = blockIdx.x + hi * gridDim.x, b = head / nh, hd = head - b * nh;
      tc::mbar_expect_tx(&raw_full[p], P32_RAW);
      tc::tma_load_2d(smem + GP_RAW_OFF + p * P32_RAW, &map, 0, ((b * T + t) * 3 * a.C + (p >> 1) * a.C + hd * DK + (p & 1) * 2) * 32, &raw_full[p]);
      __threadfence_block();
      armed[p] = (LAST && p < 2 ? hi : s) + 1;
    };
    if (warp == GP_FFT && lane == 0 && steps > 0)
      for (int p = 0; p < 6; ++p) load(p, LAST && p < 2 ? T - 1 : 0);
    int pend = -1;                                                        // output buffer whose store is still being read
    auto flush = [&]() {
      if (pend >= 0 && lane == 0) {
        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        tc::mbar_arrive(&out_empty[pend]);
      }
      pend = -1;
    };
    for (int n = warp - GP_FFT; n < 8 * (steps + 1); n += GP_NFFT) {
      // Two passes a task, through one copy of the FFT's code (four are more than the instruction caches like): forward rows and
      // columns, or inverse columns and rows with real and imaginary parts exchanged before and after.
      const int p = n & 7;
      const bool fwd = p < 6;
      const int s = (n >> 3) - (fwd ? 0 : 1), hi = s / T, t = s - hi * T, slot = s & 1;
      if (fwd && s >= steps) {
        // No work, but the wait of every forward task: it keeps a warp from running a phase of out_full ahead, whose
        // parity would pass (an inverse of output e then begins after the bins have read step e).
        flush();
        if (!wait(&spec_empty[slot], ((s >> 1) & 1) ^ 1, 2)) break;
        continue;
      }
      const bool want = fwd ? !LAST || p >= 2 || t == T - 1 : s >= 0 && (!LAST || t == T - 1);
      if (!want) {
        if (!fwd) continue;
        flush();
        if (!wait(&spec_empty[slot], ((s >> 1) & 1) ^ 1, 2)) break;
        if (lane == 0) tc::mbar_arrive(&spec_full[slot]);
        continue;
      }
      const int em = LAST ? hi : s, buf = fwd ? 0 : (em & 1) * 2 + p - 6;
      unsigned char* out = smem + GP_OUT_OFF + buf * GP_OUT_BYTES;
      cf* sp = fwd ? reinterpret_cast<cf*>(smem + GP_SPEC_OFF) + (slot * 12 + 2 * p + pl) * P32_PLANE_CF
                   : reinterpret_cast<cf*>(out) + pl * P32_PLANE_CF;
      cf z[32];
      float xx = 0.f;
      bool ok = true;
      if (fwd) {
        // Copy number `idx` into this buffer: another warp issues it when it has read the one before.  Its barrier may only
        // be waited on from then on: a phase further on has the parity of the one before the current.
        const int idx = LAST && p < 2 ? hi : s;
        if (armed[p] <= idx) {
          flush();                                                        // nobody may wait for this warp meanwhile
          uint32_t polls = 0;
          while (armed[p] <= idx && ++polls < (1u << 24)) __nanosleep(20);
        }
        __syncwarp();
        const bool issued = !__any_sync(0xffffffffu, armed[p] <= idx);
        __threadfence_block();
        if (!issued) { if (lane == 0) atomicExch(&g_p32_error, 6); s_bad = 1; break; }
        if (!wait(&raw_full[p], idx & 1, 1)) break;
        p32_load_rows(smem + GP_RAW_OFF + p * P32_RAW, pl, j, z);
        tc::fence_proxy_async();                                          // these reads come before the copy that reuses the buffer
        __syncwarp();
        const int next = s + (LAST && p < 2 ? T : 1);
        if (lane == 0 && next < steps) load(p, next);
        if (p < 4) {
          float yy = 0.f;
#pragma unroll
          for (int i = 0; i < 32; ++i) { xx = fmaf(z[i].x, z[i].x, xx); yy = fmaf(z[i].y, z[i].y, yy); }
          xx += yy;
        }
      } else {
        flush();
        if (!wait(&out_full[buf], (em >> 1) & 1, 5)) break;
#pragma unroll
        for (int r = 0; r < 32; ++r) { const cf v = sp[r * P32_PITCH + j]; z[r] = mk(v.y, v.x); }
      }
#pragma unroll 1
      for (int pass = 0; pass < 2; ++pass) {
        fft32_lane<false>(z);
        if (pass == 0) {
          if (fwd) {
            if (p < 4) xx = p32_energy(xx, z);
            flush();
            if (!(ok = wait(&spec_empty[slot], ((s >> 1) & 1) ^ 1, 2))) break;
            p32_put_rows(sp, j, z);
            __syncwarp();
#pragma unroll
            for (int r = 0; r < 32; ++r) z[r] = sp[r * P32_PITCH + j];
          } else {
#pragma unroll
            for (int r = 0; r < 32; ++r) sp[r * P32_PITCH + j] = mk(z[r].y, z[r].x);
            __syncwarp();
            p32_get_rows_swapped(sp, j, z);
            __syncwarp();
          }
        } else if (fwd) {
#pragma unroll
          for (int r = 0; r < 32; ++r) sp[r * P32_PITCH + j] = z[r];
          if (p < 4 && j == 0) nrm[slot][2 * p + pl] = a.use_l2 ? rsqrtf(xx + 1e-6f) : 1.f;
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(&spec_full[slot]);
        } else {
          p32_store_rows_swapped(out, pl, j, z);                          // over the spectra, which every lane has read
          tc::fence_proxy_async();
          __syncwarp();
          if (lane == 0) {
            const int head = blockIdx.x + hi * gridDim.x, b = head / nh, hd = head - b * nh;
            if (!s_bad) tc::tma_store_2d(&map, out, 0, ((b * T + t) * 3 * a.C + 2 * a.C + hd * DK + (p - 6) * 2) * 32);
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          }
          pend = buf;
        }
      }
      if (!ok) break;
    }
    flush();
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  } else {
    // ================================ bins ================================
    const bool on = tid < 272, real = warp == 0;
    int kw, kh[2];
    p32_bins(on ? tid : 271, kw, kh);
    const int g0 = (((((kh[0] >> 2) & 1) << 2) | (kh[0] >> 3)) * 17 + kw) * 4 + (kh[0] & 3);      // bin_index, PATH_R32
    const int g1 = (((((kh[1] >> 2) & 1) << 2) | (kh[1] >> 3)) * 17 + kw) * 4 + (kh[1] & 3);
    typedef unsigned long long u64;
    u64 Sx[2][2][4], Sy[2][2][4];                                         // [bin][row pair][column of the state]
    float2 gn[2], wn[2];                                                  // gates and W_hat of the step to come
    cf hs[2][4], wd[2][4];                                                // DN: states and W_hat of the head's channels
    float2 cn = make_float2(0.f, 0.f);                                    // DN: gates of channel lane & 3 in the step to come
    auto fetch = [&](int head, int t) {
      const int b = head / nh, hd = head - b * nh;
      if constexpr (DN) {
        cn = __ldg(a.chan + (size_t)(b * T + t) * a.C + hd * DK + (lane & 3));
      } else {
        const float2* ab = a.ab + ((size_t)(b * T + t) * a.ab_heads + (a.ab_heads > 1 ? hd : 0)) * NB;
        const float2* wh = reinterpret_cast<const float2*>(a.what) + (size_t)hd * NB;
        gn[0] = __ldg(ab + g0); gn[1] = __ldg(ab + g1);
        wn[0] = __ldg(wh + g0); wn[1] = __ldg(wh + g1);
      }
    };
    if (mine > 0) fetch(blockIdx.x, 0);
    int step = 0, emitted = 0;
    bool ok = true;
    for (int h = 0; h < mine && ok; ++h) {
      const int head = blockIdx.x + h * gridDim.x;
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          if constexpr (DN) {
            const float2 u = __ldg(reinterpret_cast<const float2*>(a.what) + (size_t)((head % nh) * DK + c) * NB + (i ? g1 : g0));
            wd[i][c] = mk(u.x, u.y);
            hs[i][c] = mk(0.f, 0.f);
          } else {
#pragma unroll
            for (int r = 0; r < 2; ++r) Sx[i][r][c] = Sy[i][r][c] = 0ull;
          }
        }
      for (int t = 0; t < T; ++t, ++step) {
        const int slot = step & 1;
        const bool emit = !LAST || t == T - 1;
        const float2 gc[2] = {gn[0], gn[1]}, wc[2] = {wn[0], wn[1]}, cc = cn;
        if (t + 1 < T) fetch(head, t + 1);
        else if (h + 1 < mine) fetch(head + gridDim.x, 0);
        if (!(ok = wait(&spec_full[slot], (step >> 1) & 1, 3))) break;
        const cf* sp = reinterpret_cast<const cf*>(smem + GP_SPEC_OFF) + slot * 12 * P32_PLANE_CF;
        float nv[8];
        {
          const float4 n0 = *reinterpret_cast<const float4*>(&nrm[slot][0]), n1 = *reinterpret_cast<const float4*>(&nrm[slot][4]);
          nv[0] = n0.x; nv[1] = n0.y; nv[2] = n0.z; nv[3] = n0.w; nv[4] = n1.x; nv[5] = n1.y; nv[6] = n1.z; nv[7] = n1.w;
        }
        cf oo[2][4];
        if constexpr (DN) {
          // per channel: A = squash(alpha W_hat (1 - beta |k|^2)), h = A h + beta v conj(k), o = h q
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const float alpha = __shfl_sync(0xffffffffu, cc.x, c), beta = __shfl_sync(0xffffffffu, cc.y, c);
            const float nq = nv[c] * (1.0f / 1024.0f), nk = nv[4 + c];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              const cf ks = p32_read1(sp + (4 + c) * P32_PLANE_CF, real, kw, kh, q), v = p32_read1(sp + (8 + c) * P32_PLANE_CF, real, kw, kh, q);
              const cf k = mk(ks.x * nk, ks.y * nk);
              const float sc = alpha * (1.0f - beta * (k.x * k.x + k.y * k.y));
              cf A = mk(wd[q][c].x * sc, wd[q][c].y * sc);
              const float am = sqrtf(A.x * A.x + A.y * A.y), sq = a.rho / (1.0f + am);
              A = mk(A.x * sq, A.y * sq);
              if (am * sq < a.floor_mag) A = mk(a.floor_mag, 0.f);
              cf U = cmulc(v, k);
              U = mk(U.x * beta, U.y * beta);
              if (U.x * U.x + U.y * U.y < a.floor_mag * a.floor_mag) U = mk(a.floor_mag, 0.f);
              cf hn = cmul(A, hs[q][c]);
              hn.x += U.x; hn.y += U.y;
              hs[q][c] = hn;
              if (emit) {
                const cf qs = p32_read1(sp + c * P32_PLANE_CF, real, kw, kh, q);
                oo[q][c] = cmul(hn, mk(qs.x * nq, qs.y * nq));
              }
            }
          }
        } else {
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const float beta = gc[q].y;
            u64 kx[4], ky[4], kyn[4];
            {
              cf kk[4];
              float ks = 0.f;
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const cf k = p32_read1(sp + (4 + i) * P32_PLANE_CF, real, kw, kh, q);
                kk[i] = mk(k.x * nv[4 + i], k.y * nv[4 + i]);
                ks += kk[i].x * kk[i].x + kk[i].y * kk[i].y;
              }
              const float kn = rsqrtf(ks + 1e-6f);
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const float x = kk[i].x * kn, y = kk[i].y * kn;
                kx[i] = pk2(x, x); ky[i] = pk2(y, y); kyn[i] = pk2(-y, -y);
              }
            }
            const float awx = gc[q].x * wc[q].x, awy = gc[q].x * wc[q].y;
            const u64 ax = pk2(awx, awx), ay = pk2(awy, awy), ayn = pk2(-awy, -awy), bn = pk2(-beta, -beta);
#pragma unroll
            for (int r = 0; r < 2; ++r) {
              const cf v0 = p32_read1(sp + (8 + 2 * r) * P32_PLANE_CF, real, kw, kh, q), v1 = p32_read1(sp + (9 + 2 * r) * P32_PLANE_CF, real, kw, kh, q);
              // d = sum_j conj(k_j) S_j;  S_i <- aw (S_i - beta k_i d) + beta v conj(k_i)
              u64 dr = 0ull, di = 0ull;
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                dr = fma2(Sx[q][r][i], kx[i], dr); dr = fma2(Sy[q][r][i], ky[i], dr);
                di = fma2(Sy[q][r][i], kx[i], di); di = fma2(Sx[q][r][i], kyn[i], di);
              }
              const u64 er = mul2(dr, bn), ei = mul2(di, bn);
              const u64 bvx = pk2(beta * v0.x, beta * v1.x), bvy = pk2(beta * v0.y, beta * v1.y), bvxn = pk2(-beta * v0.x, -beta * v1.x);
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const u64 ir = fma2(kyn[i], ei, fma2(kx[i], er, Sx[q][r][i])), ii = fma2(ky[i], er, fma2(kx[i], ei, Sy[q][r][i]));
                Sx[q][r][i] = fma2(bvy, ky[i], fma2(bvx, kx[i], fma2(ayn, ii, mul2(ax, ir))));
                Sy[q][r][i] = fma2(bvxn, ky[i], fma2(bvy, kx[i], fma2(ay, ir, mul2(ax, ii))));
              }
            }
            if (emit) {
              // o = sum_i S_i q_i
              u64 orr[2] = {0ull, 0ull}, oi[2] = {0ull, 0ull};
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const cf qv = p32_read1(sp + i * P32_PLANE_CF, real, kw, kh, q);
                const float sc = nv[i] * (1.0f / 1024.0f), x = qv.x * sc, y = qv.y * sc;
                const u64 qx = pk2(x, x), qy = pk2(y, y), qyn = pk2(-y, -y);
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                  orr[r] = fma2(Sx[q][r][i], qx, orr[r]); orr[r] = fma2(Sy[q][r][i], qyn, orr[r]);
                  oi[r] = fma2(Sx[q][r][i], qy, oi[r]); oi[r] = fma2(Sy[q][r][i], qx, oi[r]);
                }
              }
#pragma unroll
              for (int r = 0; r < 2; ++r) {
                upk2(orr[r], oo[q][2 * r].x, oo[q][2 * r + 1].x);
                upk2(oi[r], oo[q][2 * r].y, oo[q][2 * r + 1].y);
              }
            }
          }
        }
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&spec_empty[slot]);
        if (emit) {
#pragma unroll
          for (int w = 0; w < 2; ++w) {
            const int buf = (emitted & 1) * 2 + w;
            if (!(ok = wait(&out_empty[buf], ((emitted >> 1) & 1) ^ 1, 4))) break;
            cf* op = reinterpret_cast<cf*>(smem + GP_OUT_OFF + buf * GP_OUT_BYTES);
            if (on) {
              p32_write(op, real, kw, kh, oo[0][2 * w], oo[1][2 * w]);
              p32_write(op + P32_PLANE_CF, real, kw, kh, oo[0][2 * w + 1], oo[1][2 * w + 1]);
            }
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&out_full[buf]);
          }
          if (!ok) break;
          ++emitted;
        }
      }
    }
  }
  __syncthreads();
  // error path only: copies that may still be in flight get a bounded time (~1 ms) to land
  if (s_bad)
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
}

// rows of 32 floats, boxes of two planes
static bool plane_map(CUtensorMap* map, float* base, uint64_t rows) {
  const tc::EncodeTiledFn enc = tc::encode_fn();
  if (!enc) return false;
  const cuuint64_t dims[2] = {32, rows}, strides[1] = {128};
  const cuuint32_t box[2] = {32, 64}, es[2] = {1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, base, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

static int launch_p32(const P32Args& a, bool last_only, bool dn, cudaStream_t st) {
  const long long rows = (long long)a.B * a.T * 3 * a.C * 32;
  if (rows >= (1LL << 31)) return CSSM_ERR_UNSUPPORTED;
  CUtensorMap map;
  memset(&map, 0, sizeof(map));
  if (!plane_map(&map, a.qkv, (uint64_t)rows)) return CSSM_ERR_CUDA;
  auto kern = dn ? gdn_spectral_p32<false, true> : last_only ? gdn_spectral_p32<true, false> : gdn_spectral_p32<false, false>;
  const size_t smem = GP_SMEM + 1024;
  const cudaError_t e = func_smem(kern, smem);
  if (e != cudaSuccess) { set_cuda_error(e); return CSSM_ERR_CUDA; }
  const int heads = a.B * (a.C / 4), sms = sm_count();
  launch_k(kern, heads < sms ? heads : sms, GP_THREADS, smem, st, a, map);
  return check_launch();
}

int launch_gdn_spectral_p32(const GdnSpectralArgs& g, cudaStream_t st) {
  if (g.static_image || g.dk != 4 || g.H != 32 || g.W != 32) return CSSM_ERR_UNSUPPORTED;
  P32Args a;
  memset(&a, 0, sizeof(a));
  a.qkv = g.qkv; a.what = g.what; a.ab = g.ab; a.ab_heads = g.ab_heads;
  a.B = g.B; a.T = g.T; a.C = g.C; a.use_l2 = g.use_l2;
  return launch_p32(a, g.last_only != 0, false, st);
}

int launch_deltanet_spectral_p32(const DnSpectralArgs& g, cudaStream_t st) {
  if (g.chan == nullptr || g.H != 32 || g.W != 32 || g.C % 4 != 0) return CSSM_ERR_UNSUPPORTED;
  P32Args a;
  memset(&a, 0, sizeof(a));
  a.qkv = g.qkv; a.what = g.what; a.chan = g.chan; a.rho = g.rho; a.floor_mag = g.goom_floor ? 1e-7f : 0.f;
  a.B = g.B; a.T = g.T; a.C = g.C; a.use_l2 = 1;
  return launch_p32(a, false, true, st);
}

int read_p32_error(int* out, int clear) {
  cudaError_t e = cudaMemcpyFromSymbol(out, g_p32_error, sizeof(int));
  if (e == cudaSuccess && clear && *out != 0) {
    const int zero = 0;
    e = cudaMemcpyToSymbol(g_p32_error, &zero, sizeof(int));
  }
  if (e != cudaSuccess) { set_cuda_error(e); return CSSM_ERR_CUDA; }
  return CSSM_OK;
}

}  // namespace cssm
