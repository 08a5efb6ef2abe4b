// Fused spectral kernels of the two delta-rule blocks (GatedDeltaNetCSSM, DeltaNetCSSM) for planes of any
// size and key dimensions 1 .. 4, on the folded-DFT products of dft_plane.cuh (64x64 and 32x32 planes
// with key dimension 4, and DeltaNet's, have kernels of their own, and so have most square planes with key dimensions 2 and 4,
// and DeltaNet's: csrc/delta_spectral_fft.cuh).
//
// A CTA takes `heads` consecutive heads of one batch element (DeltaNet: channels, key dimension 1): the
// k, v and q planes of the heads are transformed side by side, their spectra stay in shared memory as
// {F_k, F_{H-k}} pairs, the plane norms are summed from there in a fixed order, and a thread updates the
// state of the bin pairs it owns and writes what it reads out in the folded form the inverse passes
// take.  The state lies in shared memory where it fits, else in the caller's scratch.
//
// Bound: the packed FMAs of the products, 4 planes' worth per head and key dimension (the direct DFTs that
// ran here before did four to eight times the multiplications).  GDN 12 x 8 x 28 x 28 x 64, key dimension 2:
// 667 -> 146 us; 16 x 8 x 28 x 28 x 64 238 -> 212 with a pair of register tiles (dp_pick) instead of one for all passes.
#include <math.h>
#include <string.h>
#include "kernels.cuh"
#include "dft_plane.cuh"
#include "gdn_common.cuh"

namespace cssm {

struct DeltaDftArgs {
  int B, T, C, heads, hgroups, groups;      // heads per CTA; groups = B * hgroups
  size_t region; int ldx, ldc, smem_state;
  DpGeom g;
};

// planes [k | v | q] of n planes each (q only when the step is read out) -> spectra in RA[k][col]
template <class TL, int NT, class KGate>
__device__ __forceinline__ void delta_spectra(const DeltaDftArgs& d, const float* base, size_t seg, int n, bool emit,
                                              float4* RA, float4* RB, const float2* TW, const float2* TH, KGate&& kgate) {
  const DpGeom& g = d.g;
  dp_load_fold<NT>(g, base + seg, RA, d.ldx, n);                                 // k
  dp_load_fold<NT>(g, base + 2 * seg, RA + n * g.Hp, d.ldx, n);                  // v
  if (emit) dp_load_fold<NT>(g, base, RA + 2 * n * g.Hp, d.ldx, n);              // q
  const int P = emit ? 3 * n : 2 * n;
  __syncthreads();
  dp_rows<TL::RL, TL::YL, NT>(g, RA, d.ldx, TW, RB, d.ldc, P);
  __syncthreads();
  dp_cols<TL::RT, TL::YT, NT>(g, RB, d.ldc, TH, P, [&](int x, int k0, int m, const cf* f0, const cf* f1) {
#pragma unroll
    for (int e = 0; e < TL::YT; ++e) {
      if (e >= m) continue;
      float s0 = 1.f, s1 = 1.f;
      kgate(x, k0 + e, s0, s1);
      RA[(k0 + e) * d.ldc + x] = make_float4(s0 * f0[e].x, s0 * f0[e].y, s1 * f1[e].x, s1 * f1[e].y);
    }
  });
  __syncthreads();
}

// nrm[pl] = 1 / sqrt(sum |F|^2 + 1e-6) of planes [0, nk) and [2n, 2n + nq), one warp per plane
template <int NT>
__device__ __forceinline__ void delta_norms(const DeltaDftArgs& d, const float4* SP, float* nrm, int n, bool emit, bool on) {
  const DpGeom& g = d.g;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = warp; i < (emit ? 2 * n : n); i += NT / 32) {
    const int pl = i < n ? i : i + n;
    float s = 0.f;
    if (on)
      for (int o = lane; o < g.Hp * g.Wp; o += 32) {
        const int k = g.dWp.div(o), kw = o - k * g.Wp;
        const float4 f = SP[k * d.ldc + pl * g.Wp + kw];
        s += f.x * f.x + f.y * f.y;
        if (k != 0 && 2 * k != g.H) s += f.z * f.z + f.w * f.w;
      }
    for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if (lane == 0) nrm[pl] = on ? rsqrtf(s + 1e-6f) : 1.f;
  }
  __syncthreads();
}

// folded output spectra RB[k][col of n planes] -> real planes at dst
template <class TL, int NT>
__device__ __forceinline__ void delta_output(const DeltaDftArgs& d, float4* RA, float4* RB, const float2* TW, const float2* TH,
                                             float* dst, int n) {
  __syncthreads();
  dp_inv_cols<TL::RL, TL::YL, NT>(d.g, RB, d.ldc, TH, RA, d.ldx, n);
  __syncthreads();
  dp_inv_rows<TL::RL, TL::YL, NT>(d.g, RA, d.ldx, TW, reinterpret_cast<float*>(RB), n);
  __syncthreads();
  dp_store<NT>(d.g, reinterpret_cast<const float*>(RB), dst, nullptr, n);
}

template <class TL, int NT, int DK>
__global__ void __launch_bounds__(NT, 512 / NT) gdn_spectral_dft(const GdnSpectralArgs a, const DeltaDftArgs d) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const DpGeom& g = d.g;
  float2* TW = reinterpret_cast<float2*>(smem_raw);
  float2* TH = TW + g.Wp * g.ldw;
  unsigned char* base = reinterpret_cast<unsigned char*>(TW + dp_table_pairs(g));
  float4* RA = reinterpret_cast<float4*>(base);
  float4* RB = reinterpret_cast<float4*>(base + d.region);
  float* nrm = reinterpret_cast<float*>(base + 2 * d.region);
  float4* ST = reinterpret_cast<float4*>(nrm + (3 * d.heads * DK + 3) / 4 * 4);      // [v][i][cell] {bin k, bin H-k}
  const int HW = g.H * g.W, NB = g.H * g.Wp, cells = g.Hp * g.Wp;
  const int nh = a.C / DK;
  const float invHW = 1.0f / (float)HW;
  const int Tdata = a.static_image ? 1 : a.T;           // frames of q, k, v per batch element
  dp_fill_table<NT>(TW, g.W, g.ldw);
  dp_fill_table<NT>(TH, g.H, g.ldh);
  pdl_sync();

  for (int grp = blockIdx.x; grp < d.groups; grp += gridDim.x) {
    const int b = grp / d.hgroups, h0 = (grp - b * d.hgroups) * d.heads, nhd = min(d.heads, nh - h0), n = nhd * DK;
    for (int t = 0; t < Tdata; ++t) {
      const size_t frame = (size_t)(b * Tdata + t);
      float* fp = a.qkv + (frame * 3 * a.C + (size_t)h0 * DK) * HW;
      const size_t seg = (size_t)a.C * HW;
      const bool emit = !a.last_only || t == Tdata - 1;               // same for the whole CTA
      __syncthreads();                                                // tables written; RA, RB free again
      delta_spectra<TL, NT>(d, fp, seg, n, emit, RA, RB, TW, TH, [](int, int, float&, float&) {});
      delta_norms<NT>(d, RA, nrm, n, emit, a.use_l2 != 0);
      const float2* abf = a.ab + (a.static_image ? (size_t)b * a.T : frame) * a.ab_heads * NB;
      for (int i = threadIdx.x; i < nhd * cells; i += NT) {
        const int r = g.dWp.div(i), kw = i - r * g.Wp;
        const int hl = g.dHp.div(r), k = r - hl * g.Hp, hd = h0 + hl;
        const bool self = k == 0 || 2 * k == g.H;
        const int bin[2] = {k * g.Wp + kw, self ? k * g.Wp + kw : (g.H - k) * g.Wp + kw};
        const float2* ab = abf + (a.ab_heads > 1 ? (size_t)hd * NB : 0);
        const float4* sp = RA + k * d.ldc + kw;
        const int p0 = hl * DK;
        // both bins of the pair: normalised keys and queries
        cf kk[2][DK], qq[2][DK];
        float ks[2] = {0.f, 0.f};
#pragma unroll
        for (int j = 0; j < DK; ++j) {
          const float4 kv = sp[(p0 + j) * g.Wp];
          const float s = nrm[p0 + j];
          kk[0][j] = mk(kv.x * s, kv.y * s); kk[1][j] = mk(kv.z * s, kv.w * s);
          ks[0] += kk[0][j].x * kk[0][j].x + kk[0][j].y * kk[0][j].y;
          ks[1] += kk[1][j].x * kk[1][j].x + kk[1][j].y * kk[1][j].y;
          qq[0][j] = qq[1][j] = mk(0.f, 0.f);
          if (emit) {
            const float4 qv = sp[(2 * n + p0 + j) * g.Wp];
            const float u = nrm[2 * n + p0 + j];
            qq[0][j] = mk(qv.x * u, qv.y * u); qq[1][j] = mk(qv.z * u, qv.w * u);
          }
        }
        float2 gab[2];
        cf aw[2];
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          const float kn = rsqrtf(ks[s] + 1e-6f);
#pragma unroll
          for (int j = 0; j < DK; ++j) kk[s][j] = mk(kk[s][j].x * kn, kk[s][j].y * kn);
          gab[s] = __ldg(ab + bin[s]);
          const float2 w = __ldg(reinterpret_cast<const float2*>(a.what) + (size_t)hd * NB + bin[s]);
          aw[s] = a.static_image ? mk(w.x, w.y) : mk(gab[s].x * w.x, gab[s].x * w.y);
        }
#pragma unroll 1
        for (int v = 0; v < DK; ++v) {
          const float4 vv = sp[(n + p0 + v) * g.Wp];
          cf o[2];
          if (a.static_image) {
            o[0] = gdn_bin_static<DK>(kk[0], qq[0], mk(vv.x, vv.y), aw[0], ab + bin[0], (size_t)a.ab_heads * NB, a.T);
            o[1] = gdn_bin_static<DK>(kk[1], qq[1], mk(vv.z, vv.w), aw[1], ab + bin[1], (size_t)a.ab_heads * NB, a.T);
          } else {
            cf s0[DK], s1[DK];
            cf* gs = a.state + (((size_t)(b * nh + hd) * DK + v) * DK) * NB;
            float4* ss = ST + ((size_t)hl * DK + v) * DK * cells + k * g.Wp + kw;
#pragma unroll
            for (int j = 0; j < DK; ++j) {
              if (t == 0) s0[j] = s1[j] = mk(0.f, 0.f);
              else if (d.smem_state) {
                const float4 w = ss[j * cells];
                s0[j] = mk(w.x, w.y); s1[j] = mk(w.z, w.w);
              } else {
                s0[j] = gs[(size_t)j * NB + bin[0]]; s1[j] = gs[(size_t)j * NB + bin[1]];
              }
            }
            o[0] = gdn_bin_update_regs<DK, true>(s0, kk[0], qq[0], mk(vv.x, vv.y), aw[0], gab[0].y);
            o[1] = gdn_bin_update_regs<DK, true>(s1, kk[1], qq[1], mk(vv.z, vv.w), aw[1], gab[1].y);
            if (t + 1 < Tdata) {
#pragma unroll
              for (int j = 0; j < DK; ++j) {
                if (d.smem_state) ss[j * cells] = make_float4(s0[j].x, s0[j].y, s1[j].x, s1[j].y);
                else {
                  gs[(size_t)j * NB + bin[0]] = s0[j];
                  if (!self) gs[(size_t)j * NB + bin[1]] = s1[j];
                }
              }
            }
          }
          if (emit)
            RB[k * d.ldc + (p0 + v) * g.Wp + kw] = dp_fold_spec(self, mk(o[0].x * invHW, o[0].y * invHW),
                                                               mk(o[1].x * invHW, o[1].y * invHW));
        }
      }
      if (emit) delta_output<TL, NT>(d, RA, RB, TW, TH, fp + 2 * seg, n);
    }
  }
}

template <class TL, int NT>
__global__ void __launch_bounds__(NT, 512 / NT) deltanet_spectral_dft(const DnSpectralArgs a, const DeltaDftArgs d) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const DpGeom& g = d.g;
  float2* TW = reinterpret_cast<float2*>(smem_raw);
  float2* TH = TW + g.Wp * g.ldw;
  unsigned char* base = reinterpret_cast<unsigned char*>(TW + dp_table_pairs(g));
  float4* RA = reinterpret_cast<float4*>(base);
  float4* RB = reinterpret_cast<float4*>(base + d.region);
  float* nrm = reinterpret_cast<float*>(base + 2 * d.region);
  float4* ST = reinterpret_cast<float4*>(nrm + (3 * d.heads + 3) / 4 * 4);           // [channel][cell] {bin k, bin H-k}
  const int HW = g.H * g.W, NB = g.H * g.Wp, cells = g.Hp * g.Wp;
  const float invHW = 1.0f / (float)HW, floor_mag = a.goom_floor ? 1e-7f : 0.f;
  const bool chan = a.chan != nullptr;
  dp_fill_table<NT>(TW, g.W, g.ldw);
  dp_fill_table<NT>(TH, g.H, g.ldh);
  pdl_sync();

  for (int grp = blockIdx.x; grp < d.groups; grp += gridDim.x) {
    const int b = grp / d.hgroups, c0 = (grp - b * d.hgroups) * d.heads, n = min(d.heads, a.C - c0);
    for (int t = 0; t < a.T; ++t) {
      const size_t frame = (size_t)(b * a.T + t), seg = (size_t)a.C * HW;
      float* fp = a.qkv + (frame * 3 * a.C + c0) * HW;
      const float4* gm = a.abkv + frame * NB;
      const float* cg = a.cg + frame * NB;
      __syncthreads();                                                // tables written; RA, RB free again
      delta_spectra<TL, NT>(d, fp, seg, n, true, RA, RB, TW, TH, [&](int x, int k, float& s0, float& s1) {
        if (chan || x >= n * g.Wp) return;                            // B_k scales the key spectra
        const int kw = x - g.dWp.div(x) * g.Wp;
        s0 = __ldg(&gm[k * g.Wp + kw].z);
        s1 = __ldg(&gm[(k == 0 ? 0 : g.H - k) * g.Wp + kw].z);
      });
      delta_norms<NT>(d, RA, nrm, n, true, true);
      for (int i = threadIdx.x; i < n * cells; i += NT) {
        const int r = g.dWp.div(i), kw = i - r * g.Wp;
        const int cl = g.dHp.div(r), k = r - cl * g.Hp, ch = c0 + cl;
        const bool self = k == 0 || 2 * k == g.H;
        const int bin[2] = {k * g.Wp + kw, self ? k * g.Wp + kw : (g.H - k) * g.Wp + kw};
        const float4* sp = RA + k * d.ldc + kw;
        const float4 kf = sp[cl * g.Wp], vf = sp[(n + cl) * g.Wp], qf = sp[(2 * n + cl) * g.Wp];
        const float nk = nrm[cl], nq = nrm[2 * n + cl];
        float4* ss = ST + cl * cells + k * g.Wp + kw;
        const float4 st = t > 0 ? *ss : make_float4(0.f, 0.f, 0.f, 0.f);
        const float2 ab = chan ? __ldg(a.chan + frame * a.C + ch) : make_float2(0.f, 0.f);
        cf h[2], o[2];
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          const float4 gt = chan ? make_float4(ab.x, ab.y, 1.f, 1.f) : __ldg(gm + bin[s]);
          const float2 w = __ldg(reinterpret_cast<const float2*>(a.what) + (size_t)ch * NB + bin[s]);
          const cf kv = s ? mk(kf.z * nk, kf.w * nk) : mk(kf.x * nk, kf.y * nk);
          const cf qv = s ? mk(qf.z * nq, qf.w * nq) : mk(qf.x * nq, qf.y * nq);
          const cf vv = s ? mk(vf.z * gt.w, vf.w * gt.w) : mk(vf.x * gt.w, vf.y * gt.w);
          const float kp = kv.x * kv.x + kv.y * kv.y;
          const float sc = gt.x * (1.0f - gt.y * kp);
          cf A = mk(w.x * sc, w.y * sc);
          const float am = sqrtf(A.x * A.x + A.y * A.y);
          const float sq = a.rho / (1.0f + am);
          A = mk(A.x * sq, A.y * sq);
          if (am * sq < floor_mag) A = mk(floor_mag, 0.f);
          cf U = cmulc(vv, kv);                      // v * conj(k)
          U = mk(U.x * gt.y, U.y * gt.y);
          if (U.x * U.x + U.y * U.y < floor_mag * floor_mag) U = mk(floor_mag, 0.f);
          h[s] = cmul(A, s ? mk(st.z, st.w) : mk(st.x, st.y));
          h[s].x += U.x; h[s].y += U.y;
          const cf oq = cmul(h[s], qv);
          const float c = chan ? invHW : __ldg(cg + bin[s]);
          o[s] = mk(oq.x * c, oq.y * c);
        }
        *ss = make_float4(h[0].x, h[0].y, h[1].x, h[1].y);
        RB[k * d.ldc + cl * g.Wp + kw] = dp_fold_spec(self, o[0], o[1]);
      }
      delta_output<TL, NT>(d, RA, RB, TW, TH, fp + 2 * seg, n);
    }
  }
}

// shared memory of P = 3 * heads * dk forward planes; arg = 2 * dk + (state in shared memory)
static size_t delta_dft_bytes(const DpGeom& g, int P, int arg) {
  const int dk = arg >> 1, heads = P / (3 * dk);
  return dp_table_bytes(g) + 2 * dp_region_bytes(g, P) + (size_t)(P + 3) / 4 * 16 +
         ((arg & 1) ? (size_t)heads * dk * dk * g.Hp * g.Wp * 16 : 0);
}

static bool delta_dft_plan(int B, int T, int C, int H, int W, int dk, bool need_smem_state, DeltaDftArgs* d, DpChoice* ch) {
  memset(d, 0, sizeof(*d));
  for (int st = 1; st >= (need_smem_state ? 1 : 0); --st) {
    *ch = dp_choose(H, W, 3 * C, B, 3 * dk, 3, DP_SMEM_LIMIT, delta_dft_bytes, 2 * dk + st);
    if (ch->P == 0) continue;
    d->smem_state = st;
    d->B = B; d->T = T; d->C = C;
    d->heads = ch->P / (3 * dk);
    d->hgroups = (C / dk + d->heads - 1) / d->heads;
    d->groups = B * d->hgroups;
    d->g = dp_geom(H, W);
    d->region = dp_region_bytes(d->g, ch->P);
    d->ldx = dp_ld_rows(d->g, ch->P); d->ldc = dp_ld_cols(d->g, ch->P);
    return true;
  }
  return false;
}

template <class Kern, class Args>
static int delta_dft_launch(Kern kern, const Args& a, const DeltaDftArgs& d, const DpChoice& ch, cudaStream_t st) {
  const int slots = sm_count() * ch.ctas, grid = d.groups < slots ? d.groups : slots;
  const PdlOff alone(uneven_rounds(d.groups, ch.ctas));
  const size_t smem = spread_smem(ch.smem, grid);
  cudaError_t e = func_smem(kern, smem);
  if (e != cudaSuccess) { set_cuda_error(e); return CSSM_ERR_CUDA; }
  launch_k(kern, grid, ch.threads, smem, st, a, d);
  return check_launch();
}

template <int DK>
static int gdn_dft_dk(const GdnSpectralArgs& a, const DeltaDftArgs& d, const DpChoice& ch, cudaStream_t st) {
  return dp_pick(ch.tiles, [&](auto tl) {
    using TL = decltype(tl);
    return ch.threads == 256 ? delta_dft_launch(gdn_spectral_dft<TL, 256, DK>, a, d, ch, st) : delta_dft_launch(gdn_spectral_dft<TL, 128, DK>, a, d, ch, st);
  });
}

int launch_gdn_spectral_dft(const GdnSpectralArgs& a, cudaStream_t st) {
  DeltaDftArgs d;
  DpChoice ch;
  if (a.H == a.W && !a.static_image && (a.dk == 2 || a.dk == 4)) {
    const int rc = a.dk == 2 ? launch_gdn_spectral_fft2(a, st) : launch_gdn_spectral_fft4(a, st);
    if (rc != CSSM_ERR_UNSUPPORTED) return rc;
  }
  if (!delta_dft_plan(a.B, a.T, a.C, a.H, a.W, a.dk, false, &d, &ch)) return CSSM_ERR_UNSUPPORTED;
  switch (a.dk) {
    case 1: return gdn_dft_dk<1>(a, d, ch, st);
    case 2: return gdn_dft_dk<2>(a, d, ch, st);
    case 3: return gdn_dft_dk<3>(a, d, ch, st);
    default: return gdn_dft_dk<4>(a, d, ch, st);
  }
}

int launch_deltanet_spectral_dft(const DnSpectralArgs& a, cudaStream_t st) {
  DeltaDftArgs d;
  DpChoice ch;
  if (a.H == a.W) {
    const int rc = launch_deltanet_spectral_fft(a, st);
    if (rc != CSSM_ERR_UNSUPPORTED) return rc;
  }
  if (!delta_dft_plan(a.B, a.T, a.C, a.H, a.W, 1, true, &d, &ch)) return CSSM_ERR_UNSUPPORTED;
  return dp_pick(ch.tiles, [&](auto tl) {
    using TL = decltype(tl);
    return ch.threads == 256 ? delta_dft_launch(deltanet_spectral_dft<TL, 256>, a, d, ch, st) : delta_dft_launch(deltanet_spectral_dft<TL, 128>, a, d, ch, st);
  });
}

}  // namespace cssm
