// Fused spectral kernel of the gated block for planes of any size (64x64, 32x32 and most square ones have their own):
// rfft2 -> gated recurrence over T -> irfft2 -> * silu(z), on the folded-DFT products of dft_plane.cuh.
//
// A CTA takes P consecutive channels of one batch element and walks t = 0 .. T-1 with their state in
// shared memory; CTAs are persistent and loop over the channel groups, so the DFT tables are made once.
// A thread always owns the same (column, row frequency pair) cells, so the state needs no barrier.
// P, the register tile and the number of threads (128 or 256) are chosen by the launcher (dp_choose).
//
// Bound: the packed FMAs of the four products and the shared-memory reads that feed them
// (4 P Hp Wp (Hp + Wp) / 2 packed multiply-adds a step); below 20 x 20 pixels the loads and barriers.
// 16 x 8 x 56 x 56 x 32: 1074 (direct DFTs, one thread per output) -> 223 -> 197 us (1 x 8 cells a lane in three passes instead
// of 2 x 4); 12 x 8 x 28 x 28 x 64 82 -> 74, 2 x 4 x 72 x 72 x 32 92 -> 72, 512 x 1 x 7 x 7 x 384 84 -> 72; 48 x 8 x 14 x 14 x 256 and
// 7 x 7 x 384, last frame only: 676 -> 283 us for the three launches of a forward.
#include <math.h>
#include <string.h>
#include "kernels.cuh"
#include "dft_plane.cuh"

namespace cssm {

struct GatedDftArgs {
  float* xz; const cf* khat; const float4* gates; const float* dchan;
  int B, T, C, P, groups, last_only, mode;        // mode: see launch_spectral
  size_t region; int ldx, ldc;
  DpGeom g;
  int reps;                                       // EQUAL: recurrence steps of frame T - 1
};

// EQUAL: clips of equal frames, of which the T first are there (launch_gated_spectral_dft).  A variant of its own: the tests and the
// loop of steps took 0.5 to 5 % of the other blocks' passes (NoGate 367 x 5 x 8 x 8 x 32 88.2 us with, 84.5 without; 22 x 8 x 37 x 16 x 64
// 121.7, 119.4; gated 16 x 8 x 14 x 14 x 64 86.7, 84.9).
template <class TL, int NT, bool EQUAL>
__global__ void __launch_bounds__(NT, 512 / NT) gated_spectral_dft(const GatedDftArgs a) {
  constexpr int RT = TL::RT, YT = TL::YT, RL = TL::RL, YL = TL::YL;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const DpGeom& g = a.g;
  float2* TW = reinterpret_cast<float2*>(smem_raw);
  float2* TH = TW + g.Wp * g.ldw;
  unsigned char* base = reinterpret_cast<unsigned char*>(TW + dp_table_pairs(g));
  float4* RA = reinterpret_cast<float4*>(base);
  float4* RB = reinterpret_cast<float4*>(base + a.region);
  float4* ST = reinterpret_cast<float4*>(base + 2 * a.region);       // [k][col] {h_k, h_{H-k}}
  const int HW = g.H * g.W, NB = g.H * g.Wp, ldx = a.ldx, ldc = a.ldc;
  dp_fill_table<NT>(TW, g.W, g.ldw);
  dp_fill_table<NT>(TH, g.H, g.ldh);
  pdl_sync();
  const int cgroups = (a.C + a.P - 1) / a.P;
  const float invHW = 1.0f / (float)HW;
  const bool keep = a.T > 1;

  for (int grp = blockIdx.x; grp < a.groups; grp += gridDim.x) {
    const int b = grp / cgroups, c0 = (grp - b * cgroups) * a.P, P = min(a.P, a.C - c0);
    for (int t = 0; t < a.T; ++t) {
      const size_t frame = (size_t)(b * a.T + t);
      float* xp = a.xz + (frame * 2 * a.C + c0) * HW;
      const bool emit = !a.last_only || t == a.T - 1;                // same for the whole CTA
      __syncthreads();                                               // tables written; RA free again
      dp_load_fold<NT>(g, xp, RA, ldx, P);
      __syncthreads();
      dp_rows<RL, YL, NT>(g, RA, ldx, TW, RB, ldc, P);
      __syncthreads();
      const float4* gp = a.gates + frame * NB;
      dp_cols<RT, YT, NT>(g, RB, ldc, TH, P, [&](int x, int kr, int m, const cf* f0, const cf* f1) {
        const int pl = g.dWp.div(x), kw = x - pl * g.Wp;
        const float4* gx = gp + kw;
        const cf* kx = a.khat + (size_t)(c0 + pl) * NB + kw;
        float4 g0[YT], g1[YT];
        cf k0[YT], k1[YT];
        const int reps = EQUAL && t == a.T - 1 ? a.reps : 1;
        const bool need_k = t > 0 || (EQUAL && reps > 1);
#pragma unroll
        for (int e = 0; e < YT; ++e) {
          const int k = min(kr + e, g.Hp - 1), o0 = k * g.Wp, o1 = k == 0 ? 0 : (g.H - k) * g.Wp;
          g0[e] = g1[e] = make_float4(1.f, 1.f, invHW, 0.f);         // ungated: A = K_hat, U = X_hat
          if (a.mode != 1) { g0[e] = __ldg(gx + o0); g1[e] = __ldg(gx + o1); }
          k0[e] = k1[e] = mk(0.f, 0.f);
          if (need_k) {
            const float2 u0 = __ldg(reinterpret_cast<const float2*>(kx + o0)), u1 = __ldg(reinterpret_cast<const float2*>(kx + o1));
            k0[e] = mk(u0.x, u0.y); k1[e] = mk(u1.x, u1.y);
          }
        }
        const float dc = (a.mode == 3 && need_k) ? __ldg(a.dchan + frame * a.C + c0 + pl) : 1.f;
        auto step = [](float4 gt, cf kh, cf f, cf h) {
          cf U = mk(gt.y * f.x, gt.y * f.y);
          if (U.x * U.x + U.y * U.y < gt.w * gt.w) U = mk(gt.w, 0.f);
          const cf A = mk(kh.x * gt.x, kh.y * gt.x);
          const cf n = cmul(A, h);
          return mk(n.x + U.x, n.y + U.y);
        };
#pragma unroll
        for (int e = 0; e < YT; ++e) {
          if (e >= m) continue;
          const int k = kr + e;
          float4 st = make_float4(0.f, 0.f, 0.f, 0.f);
          if (t > 0) st = ST[k * ldc + x];
          g0[e].x *= dc; g1[e].x *= dc;
          cf h0 = step(g0[e], k0[e], f0[e], mk(st.x, st.y)), h1 = step(g1[e], k1[e], f1[e], mk(st.z, st.w));
          if (EQUAL) for (int r = 1; r < reps; ++r) { h0 = step(g0[e], k0[e], f0[e], h0); h1 = step(g1[e], k1[e], f1[e], h1); }
          if (keep) ST[k * ldc + x] = make_float4(h0.x, h0.y, h1.x, h1.y);
          if (emit)
            RA[k * ldc + x] = dp_fold_spec(k == 0 || 2 * k == g.H, mk(g0[e].z * h0.x, g0[e].z * h0.y),
                                           mk(g1[e].z * h1.x, g1[e].z * h1.y));
        }
      });
      if (!emit) continue;
      __syncthreads();
      dp_inv_cols<RL, YL, NT>(g, RA, ldc, TH, RB, ldx, P);
      __syncthreads();
      float* out = reinterpret_cast<float*>(RA);
      dp_inv_rows<RL, YL, NT>(g, RB, ldx, TW, out, P);
      __syncthreads();
      if constexpr (EQUAL) dp_store<NT>(g, out, xp, a.xz + (((size_t)b * a.T * 2 + 1) * a.C + c0) * HW, P);      // (mode 0)
      else dp_store<NT>(g, out, xp, a.mode == 0 ? xp + (size_t)a.C * HW : nullptr, P);
    }
  }
}

// Planes per CTA, register tiles and threads: the estimate adds up, for a wave of CTAs, the time of the four passes of a step (from the
// throughput of the SM and the latency of a pass when its tiles do not fill the threads) and a fixed part for the loads and barriers.
// The constants were fitted to measured times of all choices (on 148 SMs; another device's count takes the place of that number): 40
// shapes of the gated kernel and 19 of the gated DeltaNet's for DP_FEW; 750 of the delta rules for DP_MANY, which has the groups of nine
// planes and more (key dimension 3 and 4).  Those often leave one CTA of eight warps an SM, where throughput and latency both count
// (the root of their squares); with the larger of the two 1 x 4 cells were taken there, 3 % behind 2 x 4 or 1 x 8 (31 x 8 x 39 x 39 x 32,
// dk = 4: 466 us, now 450).  307 other shapes of dk 3 and 4: 0.991 of the times with DP_FEW; of key dimension 1 and 2 as many lose as gain.
struct DpTileCost { int r, y; double per, lat, epi; };      // cells; clocks: SM time of a tile and step, latency of a step, of an epilogue
struct DpModel { DpTileCost heavy[2], light[4]; double border, cell, step, plane, wide; bool both; };
static constexpr DpModel DP_FEW = {{{1, 2, 0.11, 34.7, 198}, {2, 4, 0.0501, 39, 954}},
                                   {{1, 2, 0.082, 36, 216}, {1, 4, 0.123, 37.9, 304}, {2, 4, 0.272, 78.5, 478}, {1, 8, 0.224, 77.2, 427}},
                                   0.185, 0.0108, 455, 0.252, 1.03, false};
static constexpr DpModel DP_MANY = {{{1, 2, 0.0235, 29.8, 219}, {2, 4, 0.00509, 18.6, 171}},
                                    {{1, 2, 0.0474, 38.9, 130}, {1, 4, 0.0791, 48.7, 352}, {2, 4, 0.268, 44.6, 955}, {1, 8, 0.295, 60.5, 518}},
                                    0.65, 0.0104, 1890, 0.181, 1.038, true};
// The search is a few microseconds of host time, so each thread remembers its last few answers: a pure function of the key.
DpChoice dp_choose(int H, int W, int C, int B, int unit, int back, size_t limit, size_t (*bytes)(const DpGeom&, int, int), int arg) {
  struct Memo { int H, W, C, B, unit, back, arg, sms; size_t limit; size_t (*bytes)(const DpGeom&, int, int); DpChoice c; };
  static thread_local Memo memo[8] = {};
  const int sms = sm_count();
  Memo& m = memo[(H * 31 + W * 17 + C + B * 7 + arg + unit) & 7];
  if (m.bytes == bytes && m.H == H && m.W == W && m.C == C && m.B == B && m.unit == unit && m.back == back && m.arg == arg && m.sms == sms &&
      m.limit == limit)
    return m.c;
  const DpGeom g = dp_geom(H, W);
  const DpModel& dm = unit < 9 ? DP_FEW : DP_MANY;
  DpChoice best;
  best.P = 0; best.cost = 1e30; best.tiles = 0; best.ctas = 1; best.smem = 0;
  for (int P = unit; P <= C && P <= 128 * unit; P += unit) {
    const size_t smem = bytes(g, P, arg);
    if (smem > limit) break;
    const double groups = (double)B * ((C + P - 1) / P);
    for (int v = 0; v < 2 * DP_TILES; ++v) {
      const int tiles = v >> 1, nt = v & 1 ? 256 : 128;
      const int fit = (int)((227 * 1024) / (smem + 1024)), most = 512 / nt, occ = fit > most ? most : (fit < 1 ? 1 : fit);
      const DpTileCost &h = dm.heavy[tiles >= 2], &l = dm.light[tiles >= 2 ? tiles - 1 : tiles];
      auto up = [](int a, int b) { return (a + b - 1) / b; };
      auto pass = [&](const DpTileCost& t, int X, int Y, double q) {
        const int nx = up(X, t.r);                 // (a warp on the border of two rows of tiles reads two table entries)
        const double n = (double)nx * up(Y, t.y);
        const double thr = q * n * (Y * t.per * (1 + dm.border * 32 / nx) + dm.cell * t.r * t.y), ltn = ceil(n / nt) * (Y * t.lat + t.epi);
        return dm.both ? sqrt(thr * thr + ltn * ltn) : thr > ltn ? thr : ltn;
      };
      const double resident = groups < (double)sms * occ ? ceil(groups / sms) : occ;
      const int Q = P / back;
      const double step = pass(l, P * g.Hp, g.Wp, resident) + pass(h, P * g.Wp, g.Hp, resident) + pass(l, Q * g.Wp, g.Hp, resident) +
                          pass(l, Q * g.Hp, g.Wp, resident) + dm.step + dm.plane * resident * P * H * W;
      const double cost = ceil(groups / (sms * resident)) * step * (nt > 128 ? dm.wide : 1.0);
      if (cost < best.cost) { best.cost = cost; best.P = P; best.tiles = tiles; best.ctas = occ; best.threads = nt; best.smem = smem; }
    }
  }
  m = Memo{H, W, C, B, unit, back, arg, sms, limit, bytes, best};
  return best;
}

static size_t gated_dft_bytes(const DpGeom& g, int P, int T) {
  return dp_table_bytes(g) + 2 * dp_region_bytes(g, P) + (T > 1 ? (size_t)g.Hp * dp_ld_cols(g, P) * 16 : 0);
}

bool gated_spectral_dft_fits(int H, int W, int T) { return gated_dft_bytes(dp_geom(H, W), 1, T) <= DP_SMEM_LIMIT; }

template <bool EQUAL>
static auto pick_kernel(const DpChoice& ch) {
  return dp_pick(ch.tiles, [&](auto tl) {
    using TL = decltype(tl);
    return ch.threads == 256 ? gated_spectral_dft<TL, 256, EQUAL> : gated_spectral_dft<TL, 128, EQUAL>;
  });
}

int launch_gated_spectral_dft(int B, int T, int H, int W, int C, const cf* khat, const float* gates, float* xz,
                              int last_only, int mode, cudaStream_t st, const float* dchan, int equal_steps) {
  if (equal_steps > 0 && mode != 0) return CSSM_ERR_UNSUPPORTED;
  if (gated_spectral_fft_takes(B, T, H, W, C)) return launch_gated_spectral_fft(B, T, H, C, khat, gates, xz, last_only, mode, st, dchan, equal_steps);
  const DpChoice ch = dp_choose(H, W, C, B, 1, 1, DP_SMEM_LIMIT, gated_dft_bytes, T);
  if (ch.P == 0) return CSSM_ERR_UNSUPPORTED;
  GatedDftArgs a;
  memset(&a, 0, sizeof(a));
  a.xz = xz; a.khat = khat; a.gates = reinterpret_cast<const float4*>(gates); a.dchan = dchan;
  a.B = B; a.T = T; a.C = C; a.P = ch.P; a.last_only = last_only; a.mode = mode;
  a.reps = equal_steps;
  a.g = dp_geom(H, W);
  a.groups = B * ((C + ch.P - 1) / ch.P);
  a.region = dp_region_bytes(a.g, ch.P);
  a.ldx = dp_ld_rows(a.g, ch.P); a.ldc = dp_ld_cols(a.g, ch.P);
  auto kern = equal_steps > 0 ? pick_kernel<true>(ch) : pick_kernel<false>(ch);
  const int slots = sm_count() * ch.ctas, grid = a.groups < slots ? a.groups : slots;
  const PdlOff alone(uneven_rounds(a.groups, ch.ctas));
  const size_t smem = spread_smem(ch.smem, grid);
  cudaError_t e = func_smem(kern, smem);
  if (e != cudaSuccess) { set_cuda_error(e); return CSSM_ERR_CUDA; }
  launch_k(kern, grid, ch.threads, smem, st, a);
  return check_launch();
}

}  // namespace cssm
