// Weight-only precompute (kernel spectrum, RoPE tables), the per-plane short-conv stencil
// with its plane sums, and the gate-map kernels.
#include "kernels.cuh"
#include "gates.cuh"

namespace cssm {

// ------------------------------------------------------------ kernel spectrum ----
// K[c][kh][kw] = rfft2(centre-padded k[c]) squashed to |K| < rho, floored at 1e-7.
// One thread per bin; double precision (runs once per weight set).
__global__ void khat_kernel(const float* __restrict__ k, cf* __restrict__ out, int nch, int ks,
                            int H, int W, float rho, int squash, int floor_eps, int path) {
  const int Wf = W / 2 + 1, NB = H * Wf;
  const int o = blockIdx.x * blockDim.x + threadIdx.x;
  if (o >= nch * NB) return;
  const int c = o / NB, bin = o % NB, kh = bin / Wf, kw = bin % Wf;
  // crop (ks > H or W) or centre-pad, exactly as the reference slices / pads
  int i0 = 0, i1 = ks, j0 = 0, j1 = ks, offh, offw;
  if (ks > H || ks > W) {
    const int sh = (ks - H) / 2, sw = (ks - W) / 2;
    i0 = sh; i1 = sh + H; j0 = sw; j1 = sw + W; offh = -sh; offw = -sw;
    if (i0 < 0) { i0 = 0; }
    if (j0 < 0) { j0 = 0; }
    if (i1 > ks) i1 = ks;
    if (j1 > ks) j1 = ks;
  } else {
    offh = (H - ks) / 2; offw = (W - ks) / 2;
  }
  double re = 0.0, im = 0.0;
  for (int i = i0; i < i1; ++i) {
    const int ph = i + offh;
    if (ph < 0 || ph >= H) continue;
    for (int j = j0; j < j1; ++j) {
      const int pw = j + offw;
      if (pw < 0 || pw >= W) continue;
      const double ang = -2.0 * ((double)((kh * ph) % H) / H + (double)((kw * pw) % W) / W);
      double s, co;
      sincospi(ang, &s, &co);
      const double v = k[((size_t)c * ks + i) * ks + j];
      re += v * co; im += v * s;
    }
  }
  if (squash) {
    const double mag = sqrt(re * re + im * im);
    const double sc = (double)rho / (1.0 + mag);
    re *= sc; im *= sc;
  }
  if (floor_eps && sqrt(re * re + im * im) < 1e-7) { re = 1e-7; im = 0.0; }
  out[(size_t)c * NB + bin_index(path, kh, kw, H, Wf)] = mk((float)re, (float)im);
}

int launch_khat(const float* k, cf* out, int nch, int ks, int H, int W, float rho, int squash,
                int floor_eps, int path, cudaStream_t st) {
  const int n = nch * H * (W / 2 + 1);
  launch_k(khat_kernel, (n + 127) / 128, 128, 0, st, k, out, nch, ks, H, W, rho, squash, floor_eps, path);
  return check_launch();
}

// ---------------------------------------------------------------- RoPE tables ----
// (cos, sin)(pos * f_axis[i]) for the three axes; f_axis comes from the mode exactly as
// apply_rope slices and right-pads inv_freq (cssm.py:125-244).
__device__ double rope_freq(int axis, int i, int n, int mode, double base, int C) {
  auto inv = [&](int q) { return 1.0 / pow(base, (double)(2 * q) / (double)C); };
  if (mode == CSSM_ROPE_TEMPORAL) return axis == 0 ? inv(i) : 0.0;
  if (mode == CSSM_ROPE_SPATIAL_ONLY) {
    if (axis == 1) { const int q = 2 * i; return q < n ? inv(q) : 0.0; }
    if (axis == 2) { const int q = 2 * i + 1; return q < n ? inv(q) : 0.0; }
    return 0.0;
  }
  if (mode == CSSM_ROPE_SPATIOTEMPORAL) {
    const int nt = n / 3;
    if (axis == 0) return i < nt ? inv(i) : 0.0;
    if (axis == 1) { const int q = nt + 2 * i; return q < n ? inv(q) : 0.0; }
    const int q = nt + 1 + 2 * i; return q < n ? inv(q) : 0.0;
  }
  if (mode == CSSM_ROPE_MROPE) {
    const int nt = n / 3;
    if (i < 3 * nt) {
      const int r = i % 3, q = i / 3;
      if (r != axis) return 0.0;
      return inv(axis * nt + q);
    }
    // left-over width frequencies
    return axis == 2 ? inv(2 * nt + nt + (i - 3 * nt)) : 0.0;
  }
  return 0.0;
}

__global__ void rope_table_kernel(float2* tt, float2* th, float2* tw, float* nz, int T, int H,
                                  int W, int C, int mode, float base) {
  const int n = C / 2;
  const int total = (T + H + W) * n;
  const int o = blockIdx.x * blockDim.x + threadIdx.x;
  if (o < n) {
    // 1 where the pair is rotated on some axis, 0 where its angle is identically zero
    const bool any = rope_freq(0, o, n, mode, (double)base, C) != 0.0 ||
                     rope_freq(1, o, n, mode, (double)base, C) != 0.0 ||
                     rope_freq(2, o, n, mode, (double)base, C) != 0.0;
    nz[o] = any ? 1.f : 0.f;
  }
  if (o >= total) return;
  int pos = o / n, i = o % n, axis = 0;
  float2* dst = tt;
  if (pos >= T + H) { axis = 2; pos -= T + H; dst = tw; }
  else if (pos >= T) { axis = 1; pos -= T; dst = th; }
  const double ang = (double)pos * rope_freq(axis, i, n, mode, (double)base, C);
  dst[pos * n + i] = make_float2((float)cos(ang), (float)sin(ang));
}

int launch_rope_tables(float2* tt, float2* th, float2* tw, float* nz, int T, int H, int W, int C,
                       int mode, float base, cudaStream_t st) {
  const int total = (T + H + W) * (C / 2);
  launch_k(rope_table_kernel, (total + 127) / 128, 128, 0, st, tt, th, tw, nz, T, H, W, C, mode, base);
  return check_launch();
}

// interleaved (sin, cos) temporal code added to the GDN gate context (cssm.py:353-383)
__global__ void tcode_kernel(float* out, int T, int C, float base) {
  const int o = blockIdx.x * blockDim.x + threadIdx.x;
  if (o >= T * C) return;
  const int t = o / C, ch = o % C, i = ch >> 1;
  const double f = 1.0 / pow((double)base, (double)(2 * i) / (double)C);
  const double ang = (double)t * f;
  out[o] = (float)((ch & 1) ? cos(ang) : sin(ang));
}

int launch_tcode(float* out, int T, int C, float base, cudaStream_t st) {
  launch_k(tcode_kernel, (T * C + 127) / 128, 128, 0, st, out, T, C, base);
  return check_launch();
}

// ------------------------------------------------------------- plane stencil ----
// One CTA per (b, channel) walks t = 0..T-1 over planes of a planar tensor, in place:
//   s_t  = dwconv_kxk(raw_t) + b_sp                (if ksp > 0, zero 'SAME' padding)
//   o_t  = b_t + sum_j w_t[j] * s_{t-(kt-1)+j}     (if kt > 0; frames before 0 are zero)
//   o_t  = silu(o_t) (if act); o_t *= post[b,t,pixel] (if post)
// and writes sum over the plane of o_t to sums[(b*T+t)*C + c] (if sums).
constexpr int ST_THREADS = 256;


// KSP / KT >= 0 fix the tap counts at compile time (taps stay in registers); -1 = run time.
template <int KSP, int KT>
__global__ void __launch_bounds__(ST_THREADS) plane_stencil_kernel(const StencilArgs s) {
  pdl_sync();
  extern __shared__ __align__(16) float sm[];
  const int HW = s.H * s.W;
  float* raw = sm;                       // [HW]
  float* hist = sm + HW;                 // [(kt-1)][HW] ring of earlier s planes
  __shared__ float red[ST_THREADS / 32];
  const int tid = threadIdx.x;
  const int b = blockIdx.x / s.C, c = blockIdx.x % s.C;
  const int ksp = KSP >= 0 ? KSP : s.ksp;
  const int kt = KT >= 0 ? KT : s.kt;
  const int nh = kt > 0 ? kt - 1 : 0;

  float wsp[KSP >= 0 ? (KSP * KSP > 0 ? KSP * KSP : 1) : 49];
  if (ksp > 0) {
#pragma unroll
    for (int i = 0; i < ksp * ksp; ++i) wsp[i] = s.wsp[(size_t)i * s.C + c];
  }
  const float bsp = ksp > 0 ? s.bsp[c] : 0.f;
  float wt[KT >= 0 ? (KT > 0 ? KT : 1) : 8];
  if (kt > 0) {
#pragma unroll
    for (int j = 0; j < kt; ++j) wt[j] = s.wt[(size_t)j * s.C + c];
  }
  const float btv = kt > 0 ? s.bt[c] : 0.f;
  const int lo = (ksp - 1) / 2;

  for (int t = 0; t < s.T; ++t) {
    const size_t frame = (size_t)(b * s.T + t);
    float* p = s.buf + (frame * s.planes_per_frame + s.plane0 + c) * HW;
    __syncthreads();
    for (int i = tid; i < HW; i += ST_THREADS) raw[i] = p[i];
    __syncthreads();
    float lsum = 0.f;
    for (int i = tid; i < HW; i += ST_THREADS) {
      float v;
      if (ksp > 0) {
        const int h = i / s.W, w = i % s.W;
        v = bsp;
#pragma unroll
        for (int di = 0; di < ksp; ++di) {
          const int hh = h + di - lo;
          if (hh < 0 || hh >= s.H) continue;
#pragma unroll
          for (int dj = 0; dj < ksp; ++dj) {
            const int ww = w + dj - lo;
            if (ww < 0 || ww >= s.W) continue;
            v = fmaf(wsp[di * ksp + dj], raw[hh * s.W + ww], v);
          }
        }
      } else {
        v = raw[i];
      }
      float o = v;
      if (kt > 0) {
        o = btv + wt[kt - 1] * v;
        // tap j reads s_{t-(kt-1)+j}; ring slot of frame f is f % nh
#pragma unroll
        for (int j = 0; j < kt - 1; ++j) {
          const int f = t - (kt - 1) + j;
          if (f >= 0) o = fmaf(wt[j], hist[(f % (nh > 0 ? nh : 1)) * HW + i], o);
        }
      }
      // each thread owns pixel i in every pass, so the ring can be updated in place:
      // slot t % nh holds s_{t-nh}, which tap 0 has just consumed
      if (nh > 0) hist[(t % (nh > 0 ? nh : 1)) * HW + i] = v;
      if (s.act) o = silu_f(o);
      if (s.post) o *= s.post[(frame * HW + i) * s.post_stride + s.post_off];
      p[i] = o;
      lsum += o;
    }
    if (s.sums) {
      for (int off = 16; off > 0; off >>= 1) lsum += __shfl_down_sync(0xffffffffu, lsum, off);
      if ((tid & 31) == 0) red[tid >> 5] = lsum;
      __syncthreads();
      if (tid == 0) {
        float tot = 0.f;
        for (int i = 0; i < ST_THREADS / 32; ++i) tot += red[i];
        s.sums[frame * s.C + c] = tot;
      }
    }
  }
}

// Fast path of the plane stencil for rows of whole float4 groups: float4 loads with the next
// step's plane prefetched into registers, the temporal history in registers, the spatial
// conv from a zero-haloed shared tile, per-step sums reduced once at the end.
// NP = float4 groups per thread = H*W / 1024; ANY: planes of any size with W % 4 == 0, blockDim.x threads and groups past the end of the plane.
template <int KSP, int KT, int NP, bool ANY>
__global__ void __launch_bounds__(ANY ? 512 : ST_THREADS) plane_stencil_fast_kernel(const StencilArgs s) {
  pdl_sync();
  extern __shared__ __align__(16) float sm[];
  const int H = s.H, W = s.W, HW = H * W, nt = ANY ? blockDim.x : ST_THREADS, nw = nt >> 5, groups = HW >> 2;
  const int RS = W + 8;                              // tile row stride (4-float pad each side)
  float* tile = sm;                                  // [(H+2)][RS], used when KSP > 0
  float* red = sm + (KSP > 0 ? (H + 2) * RS : 0);    // [T][warps] per-warp partial sums
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int b = blockIdx.x / s.C, c = blockIdx.x % s.C;
  constexpr int NHIST = KT > 0 ? KT - 1 : 0;

  float wsp[KSP * KSP > 0 ? KSP * KSP : 1];
  if (KSP > 0) {
#pragma unroll
    for (int i = 0; i < KSP * KSP; ++i) wsp[i] = s.wsp[(size_t)i * s.C + c];
  }
  const float bsp = KSP > 0 ? s.bsp[c] : 0.f;
  float wt[KT > 0 ? KT : 1];
  if (KT > 0) {
#pragma unroll
    for (int j = 0; j < KT; ++j) wt[j] = s.wt[(size_t)j * s.C + c];
  }
  const float btv = KT > 0 ? s.bt[c] : 0.f;
  if (KSP > 0) {
    for (int i = tid; i < (H + 2) * RS; i += nt) tile[i] = 0.f;
  }
  float4 hist[NP][NHIST > 0 ? NHIST : 1];
#pragma unroll
  for (int j = 0; j < NP; ++j)
#pragma unroll
    for (int k = 0; k < NHIST; ++k) hist[j][k] = make_float4(0.f, 0.f, 0.f, 0.f);

  const size_t pstride = (size_t)s.planes_per_frame * HW;       // plane of the next frame
  float* p0 = s.buf + ((size_t)(b * s.T) * s.planes_per_frame + s.plane0 + c) * HW;
  float4 cur[NP], nxt[NP];
  int toff[NP];                    // tile offset of the thread's group j (interior origin)
  const int gpr = W >> 2;          // float4 groups per image row; lanes are consecutive groups
  bool left_edge[NP], right_edge[NP];
#pragma unroll
  for (int j = 0; j < NP; ++j) {
    const int g4 = ANY ? min(tid + j * nt, groups - 1) : tid + j * nt;
    cur[j] = reinterpret_cast<const float4*>(p0)[g4];
    const int h = g4 / gpr, gc = g4 - h * gpr;
    toff[j] = (h + 1) * RS + 4 + gc * 4;
    left_edge[j] = gc == 0 || lane == 0;
    right_edge[j] = gc == gpr - 1 || lane == 31;
  }
  __syncthreads();

  for (int t = 0; t < s.T; ++t) {
    float* p = p0 + (size_t)t * pstride;
    if (t + 1 < s.T) {
#pragma unroll
      for (int j = 0; j < NP; ++j)
        nxt[j] = reinterpret_cast<const float4*>(p + pstride)[ANY ? min(tid + j * nt, groups - 1) : tid + j * nt];
    }
    if (KSP > 0) {
#pragma unroll
      for (int j = 0; j < NP; ++j) *reinterpret_cast<float4*>(tile + toff[j]) = cur[j];
      __syncthreads();
    }
    float lsum = 0.f;
    float4 outv[NP];
#pragma unroll
    for (int j = 0; j < NP; ++j) {
      const int g4 = tid + j * nt;
      float4 v = cur[j];
      if (KSP == 3) {
        // 3x3: the row's float4 from the tile, its left / right neighbours from the adjacent
        // lanes (adjacent float4 groups of the same image row) or from the zero halo
        float a0 = bsp, a1 = bsp, a2 = bsp, a3 = bsp;
#pragma unroll
        for (int di = 0; di < 3; ++di) {
          const float* rp = tile + toff[j] + (di - 1) * RS;
          const float4 mid = *reinterpret_cast<const float4*>(rp);
          float lf = __shfl_up_sync(0xffffffffu, mid.w, 1);
          float rt = __shfl_down_sync(0xffffffffu, mid.x, 1);
          if (left_edge[j]) lf = rp[-1];
          if (right_edge[j]) rt = rp[4];
          const float w0 = wsp[di * 3], w1 = wsp[di * 3 + 1], w2 = wsp[di * 3 + 2];
          a0 = fmaf(w0, lf, a0);    a0 = fmaf(w1, mid.x, a0); a0 = fmaf(w2, mid.y, a0);
          a1 = fmaf(w0, mid.x, a1); a1 = fmaf(w1, mid.y, a1); a1 = fmaf(w2, mid.z, a1);
          a2 = fmaf(w0, mid.y, a2); a2 = fmaf(w1, mid.z, a2); a2 = fmaf(w2, mid.w, a2);
          a3 = fmaf(w0, mid.z, a3); a3 = fmaf(w1, mid.w, a3); a3 = fmaf(w2, rt, a3);
        }
        v = make_float4(a0, a1, a2, a3);
      } else if (KSP > 0) {
        constexpr int LO = (KSP - 1) / 2;
        float a0 = bsp, a1 = bsp, a2 = bsp, a3 = bsp;
#pragma unroll
        for (int di = 0; di < KSP; ++di) {
          const float* rp = tile + toff[j] + (di - LO) * RS;
          float win[4 + 2 * LO];
          const float4 mid = *reinterpret_cast<const float4*>(rp);
          win[LO] = mid.x; win[LO + 1] = mid.y; win[LO + 2] = mid.z; win[LO + 3] = mid.w;
#pragma unroll
          for (int e = 0; e < LO; ++e) { win[e] = rp[e - LO]; win[LO + 4 + e] = rp[4 + e]; }
#pragma unroll
          for (int dj = 0; dj < KSP; ++dj) {
            const float wv = wsp[di * KSP + dj];
            a0 = fmaf(wv, win[dj], a0); a1 = fmaf(wv, win[dj + 1], a1);
            a2 = fmaf(wv, win[dj + 2], a2); a3 = fmaf(wv, win[dj + 3], a3);
          }
        }
        v = make_float4(a0, a1, a2, a3);
      }
      float4 o = v;
      if (KT > 0) {
        o = make_float4(btv + wt[KT - 1] * v.x, btv + wt[KT - 1] * v.y, btv + wt[KT - 1] * v.z,
                        btv + wt[KT - 1] * v.w);
        // hist[j][k] holds s_{t-1-k}; tap index of s_{t-1-k} is KT-2-k
#pragma unroll
        for (int k = 0; k < NHIST; ++k) {
          const float wv = wt[KT - 2 - k];
          o.x = fmaf(wv, hist[j][k].x, o.x); o.y = fmaf(wv, hist[j][k].y, o.y);
          o.z = fmaf(wv, hist[j][k].z, o.z); o.w = fmaf(wv, hist[j][k].w, o.w);
        }
#pragma unroll
        for (int k = NHIST - 1; k > 0; --k) hist[j][k] = hist[j][k - 1];
        if (NHIST > 0) hist[j][0] = v;
      }
      if (s.act) { o.x = silu_f(o.x); o.y = silu_f(o.y); o.z = silu_f(o.z); o.w = silu_f(o.w); }
      if (s.post) {
        const float* pp = s.post + ((size_t)(b * s.T + t) * HW + (size_t)(ANY ? min(g4, groups - 1) : g4) * 4) * s.post_stride + s.post_off;
        o.x *= pp[0]; o.y *= pp[s.post_stride]; o.z *= pp[2 * s.post_stride]; o.w *= pp[3 * s.post_stride];
      }
      outv[j] = o;
      if (!ANY || g4 < groups) lsum += (o.x + o.y) + (o.z + o.w);
    }
    // stores after all shared-memory reads of this step (generic-pointer stores would otherwise
    // pin the following loads behind them)
#pragma unroll
    for (int j = 0; j < NP; ++j)
      if (!ANY || tid + j * nt < groups) reinterpret_cast<float4*>(p)[tid + j * nt] = outv[j];
    if (s.sums) {
      for (int off = 16; off > 0; off >>= 1) lsum += __shfl_down_sync(0xffffffffu, lsum, off);
      if (lane == 0) red[t * nw + warp] = lsum;
    }
    if (KSP > 0) __syncthreads();      // all conv reads done before the tile is overwritten
#pragma unroll
    for (int j = 0; j < NP; ++j) cur[j] = nxt[j];
  }
  if (s.sums) {
    __syncthreads();
    for (int t = tid; t < s.T; t += nt) {
      float tot = 0.f;
      for (int w = 0; w < nw; ++w) tot += red[t * nw + w];
      s.sums[(size_t)(b * s.T + t) * s.C + c] = tot;
    }
  }
}

// The plane stencil for planes of up to about 4096 pixels of any shape (3x3 or no spatial taps, four temporal
// ones): what the walk above spends its time on is one load in flight per thread, divisions and edge
// branches per tap and a history in shared memory.  Here a plane belongs to one warp (eight planes a CTA,
// no CTA barrier) or to one CTA; a thread keeps J <= 8 pixels with their history in registers and
// requests the next frame's pixels before it works on this one.  With 3x3 taps its pixels are a strip of a
// column, so that a tile value read from shared memory serves up to three of them; the tile has a zero
// halo and there are two in turn (one barrier per frame).
// (Larger planes of rows of whole float4 groups: the fast path above.)
// Bound: instruction issue and the shared-memory reads of the taps (floor 8 bytes a pixel: 24 us here).
// 48 x 8 frames of 14x14x256, 3x3 and four taps: 365 us by the walk above, 121 with pixels dealt out a warp
// wide, 73 as strips; 16 x 8 x 56x56 x 32: 100 -> 65 us.
template <int KSP, int J, bool WARP>
__global__ void __launch_bounds__(WARP ? 256 : 512, WARP ? 3 : 1) plane_stencil_small_kernel(const StencilArgs s) {
  constexpr int KT = 4;
  extern __shared__ __align__(16) float sm[];
  const int W = s.W, HW = s.H * W, RS = W + 2, strips = (s.H + J - 1) / J, TS = (strips * J + 2) * RS;
  const int nt = WARP ? 32 : blockDim.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int me = WARP ? lane : threadIdx.x, plane = WARP ? blockIdx.x * 8 + warp : blockIdx.x;
  float* tile = KSP > 0 ? sm + (WARP ? warp * 2 * TS : 0) : nullptr;      // [2][TS]
  float* red = sm + (KSP > 0 ? 2 * TS : 0);                               // [T][warps], CTA form only
  auto sync = [&]() { if (WARP) __syncwarp(); else __syncthreads(); };
  pdl_sync();
  if (WARP && plane >= s.B * s.C) return;
  const int b = plane / s.C, c = plane - b * s.C;

  // pixels i0 + j * step, j < cnt
  int i0 = me, step = nt, cnt = me < HW ? (HW - me + nt - 1) / nt : 0, toff = 0;
  if (KSP > 0) {
    const int st = me / W, w = me - st * W;
    i0 = st * J * W + w; step = W;
    cnt = min(J, s.H - st * J);                         // negative past the last strip
    toff = (cnt > 0 ? st * J * RS : 0) + w;             // top left of the first pixel's window
  }
  float wsp[KSP > 0 ? KSP * KSP : 1], wt[KT];
#pragma unroll
  for (int i = 0; i < KSP * KSP; ++i) wsp[i] = __ldg(s.wsp + (size_t)i * s.C + c);
  const float bsp = KSP > 0 ? __ldg(s.bsp + c) : 0.f;
#pragma unroll
  for (int j = 0; j < KT; ++j) wt[j] = __ldg(s.wt + (size_t)j * s.C + c);
  const float btv = __ldg(s.bt + c);

  const size_t pstride = (size_t)s.planes_per_frame * HW;
  float* p = s.buf + ((size_t)(b * s.T) * s.planes_per_frame + s.plane0 + c) * HW + i0;
  float cur[J], nxt[J], hist[J][KT - 1];      // hist[j][k] = s_{t-1-k}
#pragma unroll
  for (int j = 0; j < J; ++j) {
    cur[j] = j < cnt ? p[j * step] : 0.f;
    nxt[j] = 0.f;
#pragma unroll
    for (int k = 0; k < KT - 1; ++k) hist[j][k] = 0.f;
  }
  if (KSP > 0) {
    for (int i = me; i < 2 * TS; i += nt) tile[i] = 0.f;
    sync();
  }
  for (int t = 0; t < s.T; ++t) {
    if (t + 1 < s.T) {
#pragma unroll
      for (int j = 0; j < J; ++j)
        if (j < cnt) nxt[j] = p[pstride + j * step];
    }
    float v[J];
    if (KSP > 0) {
      float* tl = tile + (t & 1) * TS + toff;
#pragma unroll
      for (int j = 0; j < J; ++j)
        if (j < cnt) tl[(j + 1) * RS + 1] = cur[j];
      sync();
#pragma unroll
      for (int j = 0; j < J; ++j) v[j] = bsp;
#pragma unroll
      for (int r = 0; r < J + 2; ++r) {
        const float x0 = tl[r * RS], x1 = tl[r * RS + 1], x2 = tl[r * RS + 2];
#pragma unroll
        for (int di = 0; di < 3; ++di) {
          const int j = r - di;
          if (j < 0 || j >= J) continue;
          v[j] = fmaf(wsp[KSP > 0 ? di * 3 : 0], x0, v[j]);
          v[j] = fmaf(wsp[KSP > 0 ? di * 3 + 1 : 0], x1, v[j]);
          v[j] = fmaf(wsp[KSP > 0 ? di * 3 + 2 : 0], x2, v[j]);
        }
      }
    } else {
#pragma unroll
      for (int j = 0; j < J; ++j) v[j] = cur[j];
    }
    const float* post = s.post ? s.post + ((size_t)(b * s.T + t) * HW + i0) * s.post_stride + s.post_off : nullptr;
    float lsum = 0.f;
#pragma unroll
    for (int j = 0; j < J; ++j) {
      float o = btv + wt[KT - 1] * v[j];
#pragma unroll
      for (int k = KT - 2; k >= 0; --k) o = fmaf(wt[KT - 2 - k], hist[j][k], o);
#pragma unroll
      for (int k = KT - 2; k > 0; --k) hist[j][k] = hist[j][k - 1];
      hist[j][0] = v[j];
      if (s.act) o = silu_f(o);
      if (j < cnt) {
        if (post) o *= __ldg(post + (size_t)(j * step) * s.post_stride);
        p[j * step] = o;
        lsum += o;
      }
      cur[j] = nxt[j];
    }
    p += pstride;
    if (s.sums) {
      for (int off = 16; off > 0; off >>= 1) lsum += __shfl_down_sync(0xffffffffu, lsum, off);
      if (lane == 0) {
        if (WARP) s.sums[(size_t)(b * s.T + t) * s.C + c] = lsum;
        else red[t * (nt >> 5) + warp] = lsum;
      }
    }
  }
  if (!WARP && s.sums) {
    __syncthreads();
    for (int t = threadIdx.x; t < s.T; t += nt) {
      float tot = 0.f;
      for (int w = 0; w < (nt >> 5); ++w) tot += red[t * (nt >> 5) + w];
      s.sums[(size_t)(b * s.T + t) * s.C + c] = tot;
    }
  }
}

// the fewest threads (one warp, else a CTA) that hold the plane with at most eight pixels each
template <int KSP>
static int launch_stencil_small(const StencilArgs& s, cudaStream_t st, bool* handled) {
  const int HW = s.H * s.W;
  static const int sizes[4] = {32, 128, 256, 512}, js[4] = {2, 4, 7, 8};
  int nt = 0, J = 0;
  for (int k = 0; k < 4 && J == 0; ++k)
    for (int i = 0; i < 4 && J == 0; ++i) {
      const int j = js[i];
      if (KSP > 0 ? (long long)s.W * ((s.H + j - 1) / j) <= sizes[k] : HW <= j * sizes[k]) { nt = sizes[k]; J = j; }
    }
  const bool warp = nt == 32;
  const size_t tiles = KSP > 0 && J > 0 ? (size_t)2 * ((s.H + J - 1) / J * J + 2) * (s.W + 2) * (warp ? 8 : 1) : 0;
  const size_t smem = (tiles + (warp ? 0 : (size_t)s.T * (nt / 32))) * sizeof(float);
  *handled = J > 0 && smem <= 64 * 1024;
  if (!*handled) return CSSM_OK;
  auto go = [&](auto kern) -> int {
    cudaError_t e = func_smem(kern, smem);
    if (e != cudaSuccess) { set_cuda_error(e); return CSSM_ERR_CUDA; }
    launch_k(kern, warp ? (s.B * s.C + 7) / 8 : s.B * s.C, warp ? 256 : nt, smem, st, s);
    return check_launch();
  };
  if (warp) {
    if (J == 2) return go(plane_stencil_small_kernel<KSP, 2, true>);
    if (J == 4) return go(plane_stencil_small_kernel<KSP, 4, true>);
    if (J == 7) return go(plane_stencil_small_kernel<KSP, 7, true>);
    return go(plane_stencil_small_kernel<KSP, 8, true>);
  }
  if (J == 2) return go(plane_stencil_small_kernel<KSP, 2, false>);
  if (J == 4) return go(plane_stencil_small_kernel<KSP, 4, false>);
  if (J == 7) return go(plane_stencil_small_kernel<KSP, 7, false>);
  return go(plane_stencil_small_kernel<KSP, 8, false>);
}

template <int KSP, int KT, int NP, bool ANY = false>
static int launch_stencil_fast(const StencilArgs& s, cudaStream_t st, int nt = ST_THREADS) {
  const size_t smem = ((KSP > 0 ? (size_t)(s.H + 2) * (s.W + 8) : 0) + (size_t)s.T * (nt / 32)) * sizeof(float);
  if (smem > 200 * 1024) return CSSM_ERR_UNSUPPORTED;
  auto kern = plane_stencil_fast_kernel<KSP, KT, NP, ANY>;
  cudaError_t e = func_smem(kern, smem);
  if (e != cudaSuccess) { set_cuda_error(e); return CSSM_ERR_CUDA; }
  launch_k(kern, s.B * s.C, nt, smem, st, s);
  return check_launch();
}

template <int NP>
static int dispatch_stencil_fast(const StencilArgs& s, cudaStream_t st, bool* handled) {
  *handled = true;
  if (s.ksp == 3 && s.kt == 4) return launch_stencil_fast<3, 4, NP>(s, st);
  if (s.ksp == 0 && s.kt == 4) return launch_stencil_fast<0, 4, NP>(s, st);
  if (s.ksp == 3 && s.kt == 0) return launch_stencil_fast<3, 0, NP>(s, st);
  if (s.ksp == 0 && s.kt == 0) return launch_stencil_fast<0, 0, NP>(s, st);
  *handled = false;
  return CSSM_OK;
}

// Rows of whole float4 groups, four temporal taps and 3x3 or no spatial ones: the groups dealt out to a CTA of as few idle threads as can be.
// From 192 pixels on; below that the form with a plane a warp is as good or better (122 x 8 x 8 x 8 x 64 87 us a pass, 93 so; 173 x 1 x 12 x 12 x 32
// 38.4, 39.6; but 30 x 8 x 16 x 16 x 64 72.5, 64.4; 3 x 8 x 48 x 48 x 64 85, 71; of 39 shapes from 16 x 16 to 60 x 60 none more than 1 % behind); a
// single frame, whose CTAs are over before their loads pay, from 1280 on (33 x 1 x 16 x 16 x 256 twice in the classifier: 620 us a pass, 632 so).
template <int KSP>
static int launch_stencil_groups(const StencilArgs& s, cudaStream_t st, bool* handled) {
  const int groups = s.H * s.W / 4;
  int best = 0, nt = 0;
  for (int np = 1; np <= 4; ++np) {
    const int n = ((groups + np - 1) / np + 31) / 32 * 32;
    if (n > 512) continue;
    if (best == 0 || n * np < nt * best || (n * np == nt * best && n >= 128)) { best = np; nt = n; }
  }
  *handled = best > 0 && groups >= (s.T > 1 ? 48 : 320);
  if (!*handled) return CSSM_OK;
  if (best == 1) return launch_stencil_fast<KSP, 4, 1, true>(s, st, nt);
  if (best == 2) return launch_stencil_fast<KSP, 4, 2, true>(s, st, nt);
  if (best == 3) return launch_stencil_fast<KSP, 4, 3, true>(s, st, nt);
  return launch_stencil_fast<KSP, 4, 4, true>(s, st, nt);
}

// One source frame for a whole clip: the spatial conv is the same for every frame, and frame f of the temporal one sees
// f + 1 equal frames (after kt - 1 frames nothing changes any more: the caller asks for T <= kt).  So a plane is read and
// convolved once, by G threads from a zero-bordered tile, and written for the T frames that differ (48 clips of 8 frames,
// 14 x 14 x 256 twice and 7 x 7 x 384: three launches 184 us frame by frame, 56 so).
// KSP, KT: tap counts, -1: at run time (up to 7 x 7 and 8).
template <int G, int KSP, int KT>
__global__ void __launch_bounds__(256) repeat_stencil_kernel(const StencilArgs s, FastDiv dw) {
  extern __shared__ __align__(16) float sm[];
  __shared__ float red[8][8];
  constexpr int TF = KT > 0 ? KT : 8;                  // frames at most
  const int ksp = KSP >= 0 ? KSP : s.ksp, kt = KT >= 0 ? KT : s.kt, lo = ksp > 0 ? (ksp - 1) / 2 : 0;
  const int HW = s.H * s.W, pitch = s.W + (ksp > 0 ? ksp - 1 : 0), rows = s.H + (ksp > 0 ? ksp - 1 : 0);
  const int lt = threadIdx.x % G, pl = threadIdx.x / G, lane = threadIdx.x & 31;
  const int plane = blockIdx.x * (256 / G) + pl, total = s.B * s.C;
  const bool on = plane < total;
  const int b = on ? plane / s.C : 0, c = on ? plane - b * s.C : 0;
  float* raw = sm + pl * pitch * rows;
  const size_t fstride = (size_t)s.planes_per_frame * HW;
  float* __restrict__ p = s.buf + ((size_t)b * s.T * s.planes_per_frame + s.plane0 + c) * HW;
  float wsp[KSP > 0 ? KSP * KSP : 49], wt[TF];
#pragma unroll
  for (int i = 0; i < (KSP >= 0 ? KSP * KSP : 49); ++i) wsp[i] = i < ksp * ksp ? __ldg(s.wsp + (size_t)i * s.C + c) : 0.f;
#pragma unroll
  for (int j = 0; j < TF; ++j) wt[j] = j < kt ? __ldg(s.wt + (size_t)j * s.C + c) : 0.f;
  const float bsp = ksp > 0 ? __ldg(s.bsp + c) : 0.f, bt = kt > 0 ? __ldg(s.bt + c) : 0.f;
  for (int i = lt; i < pitch * rows; i += G) raw[i] = 0.f;
  if (G == 32) __syncwarp(); else __syncthreads();
  pdl_sync();
  if (on)
    for (int i0 = lt; i0 < HW; i0 += 8 * G) {
      float v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = i0 + u * G < HW ? p[i0 + u * G] : 0.f;
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int i = i0 + u * G, h = dw.div(i);
        if (i < HW) raw[(h + lo) * pitch + i - h * s.W + lo] = v[u];
      }
    }
  if (G == 32) __syncwarp(); else __syncthreads();
  float sum[TF];
#pragma unroll
  for (int f = 0; f < TF; ++f) sum[f] = 0.f;
  if (on)
    for (int i = lt; i < HW; i += G) {
      const int h = dw.div(i), w = i - h * s.W;
      const float* r = raw + h * pitch + w;
      float v;
      if (ksp > 0) {
        v = bsp;
        if constexpr (KSP >= 0) {
#pragma unroll
          for (int di = 0; di < KSP; ++di)
#pragma unroll
            for (int dj = 0; dj < KSP; ++dj) v = fmaf(wsp[di * KSP + dj], r[di * pitch + dj], v);
        } else {
          int q = 0;
          for (int di = 0; di < ksp; ++di)
            for (int dj = 0; dj < ksp; ++dj) v = fmaf(__ldg(s.wsp + (size_t)q++ * s.C + c), r[di * pitch + dj], v);
        }
      } else {
        v = *r;
      }
#pragma unroll
      for (int f = 0; f < TF; ++f) {
        if (f >= s.T) continue;
        float o = v;
        if (kt > 0) {
          // tap j reads frame f - (kt - 1) + j, the newest first
          if constexpr (KT > 0) o = fmaf(wt[KT - 1], v, bt);
          else {
#pragma unroll
            for (int j = 0; j < TF; ++j) if (j == kt - 1) o = fmaf(wt[j], v, bt);
          }
#pragma unroll
          for (int j = 0; j < TF - 1; ++j) if (j < kt - 1 && j >= kt - 1 - f) o = fmaf(wt[j], v, o);
        }
        if (s.act) o = silu_f(o);
        p[(size_t)f * fstride + i] = o;
        sum[f] += o;
      }
    }
  if (s.sums == nullptr) return;
#pragma unroll
  for (int f = 0; f < TF; ++f) {
    if (f >= s.T) continue;
    float t = sum[f];
    for (int off = 16; off > 0; off >>= 1) t += __shfl_down_sync(0xffffffffu, t, off);
    if (G == 32) { if (lane == 0 && on) s.sums[((size_t)b * s.T + f) * s.C + c] = t; }
    else if (lane == 0) red[f][threadIdx.x >> 5] = t;
  }
  if (G == 32) return;
  __syncthreads();
  if (on && lt < s.T) {
    float t = 0.f;
    for (int i = 0; i < 8; ++i) t += red[lt][i];
    s.sums[((size_t)b * s.T + lt) * s.C + c] = t;
  }
}

int launch_repeat_stencil(const StencilArgs& s, cudaStream_t st) {
  const int halo = s.ksp > 0 ? s.ksp - 1 : 0;
  const size_t plane = (size_t)(s.H + halo) * (s.W + halo) * sizeof(float);
  if (s.T > 8 || s.kt > 8 || s.ksp > 7 || s.T > (s.kt > 1 ? s.kt : 1) || s.post != nullptr || plane > 200 * 1024) return CSSM_ERR_UNSUPPORTED;
  const bool warp = 8 * plane <= 48 * 1024;            // a plane a warp up to 37 x 37 and a 3 x 3 conv, else a CTA
  const size_t smem = warp ? 8 * plane : plane;
  auto kern = s.ksp == 3 && s.kt == 4 ? (warp ? repeat_stencil_kernel<32, 3, 4> : repeat_stencil_kernel<256, 3, 4>)
                                      : (warp ? repeat_stencil_kernel<32, -1, -1> : repeat_stencil_kernel<256, -1, -1>);
  const cudaError_t e = func_smem(kern, smem);
  if (e != cudaSuccess) { set_cuda_error(e); return CSSM_ERR_CUDA; }
  const long long planes = (long long)s.B * s.C;
  launch_k(kern, (unsigned)(warp ? (planes + 7) / 8 : planes), 256, smem, st, s, FastDiv(s.W));
  return check_launch();
}

int launch_plane_stencil(const StencilArgs& s, cudaStream_t st) {
  if (s.ksp > 7 || s.kt > 8) return CSSM_ERR_UNSUPPORTED;
  if (s.W % 4 == 0 && (s.H * s.W == 4096 || s.H * s.W == 1024) &&
      (reinterpret_cast<uintptr_t>(s.buf) & 15u) == 0) {
    bool handled = false;
    const int rc = s.H * s.W == 4096 ? dispatch_stencil_fast<4>(s, st, &handled)
                                     : dispatch_stencil_fast<1>(s, st, &handled);
    if (handled) return rc;
  }
  if (s.kt == 4 && (s.ksp == 0 || s.ksp == 3) && s.W % 4 == 0 && (reinterpret_cast<uintptr_t>(s.buf) & 15u) == 0) {
    bool handled = false;
    const int rc = s.ksp == 3 ? launch_stencil_groups<3>(s, st, &handled) : launch_stencil_groups<0>(s, st, &handled);
    if (handled) return rc;
  }
  if (s.kt == 4 && (s.ksp == 0 || s.ksp == 3)) {
    bool handled = false;
    const int rc = s.ksp == 3 ? launch_stencil_small<3>(s, st, &handled) : launch_stencil_small<0>(s, st, &handled);
    if (handled) return rc;
  }
  const int nh = s.kt > 0 ? s.kt - 1 : 0;
  const size_t smem = (size_t)(1 + nh) * s.H * s.W * sizeof(float);
  if (smem > 200 * 1024) return CSSM_ERR_UNSUPPORTED;
  auto go = [&](auto kern) -> int {
    cudaError_t e = func_smem(kern, smem);
    if (e != cudaSuccess) { set_cuda_error(e); return CSSM_ERR_CUDA; }
    launch_k(kern, s.B * s.C, ST_THREADS, smem, st, s);
    return check_launch();
  };
  if (s.ksp == 3 && s.kt == 4) return go(plane_stencil_kernel<3, 4>);
  if (s.ksp == 0 && s.kt == 4) return go(plane_stencil_kernel<0, 4>);
  if (s.ksp == 3 && s.kt == 0) return go(plane_stencil_kernel<3, 0>);
  if (s.ksp == 0 && s.kt == 0) return go(plane_stencil_kernel<0, 0>);
  return go(plane_stencil_kernel<-1, -1>);
}

// ------------------------------------------- temporal conv on q, k, v (GDN) ----
// Causal depthwise temporal conv (KT taps) + SiLU + optional per-pixel input gate on the 3C planar
// planes of q, k and v in ONE elementwise launch: a thread owns four consecutive pixels of one
// plane and walks t with the KT-1 previous raw values in registers and the next frame's load in
// flight, so every plane is read once and written once at full occupancy.  Gate planes (channel gates) are multiplied on the way.
template <int KT, bool PLANES>
__global__ void __launch_bounds__(256) qkv_temporal_conv_kernel(const QkvTconvArgs a) {
  pdl_sync();
  const int HW4 = a.HW >> 2;
  const long long gid = (long long)blockIdx.x * 256 + threadIdx.x;
  const long long total = (long long)a.B * 3 * a.C * HW4;
  if (gid >= total) return;
  const int g4 = (int)(gid % HW4);
  const int p = (int)((gid / HW4) % (3 * a.C));
  const int b = (int)(gid / ((long long)HW4 * 3 * a.C));
  const int grp = p / a.C, c = p - grp * a.C;
  const float* wtp = grp == 0 ? a.wt[0] : grp == 1 ? a.wt[1] : a.wt[2];
  const float* btp = grp == 0 ? a.bt[0] : grp == 1 ? a.bt[1] : a.bt[2];
  float w[KT];
#pragma unroll
  for (int j = 0; j < KT; ++j) w[j] = wtp[(size_t)j * a.C + c];
  const float bias = btp[c];
  const int poff = grp - 1;                                   // k: B_k, v: B_v, q: none
  const bool gated = !PLANES && a.bkv != nullptr && grp > 0, planes = PLANES && grp > 0;
  float4 hist[KT - 1];
#pragma unroll
  for (int k = 0; k < KT - 1; ++k) hist[k] = make_float4(0.f, 0.f, 0.f, 0.f);
  const size_t fstride = (size_t)3 * a.C * HW4;               // float4 units between frames
  float4* ptr = reinterpret_cast<float4*>(a.buf) + ((size_t)b * a.T * 3 * a.C + p) * HW4 + g4;
  const size_t gstride = (size_t)2 * a.C * HW4;
  const float4* gpl = planes ? reinterpret_cast<const float4*>(a.gsp) + ((size_t)b * a.T * 2 * a.C + p - a.C) * HW4 + g4 : nullptr;
  constexpr int AH = PLANES ? 2 : 1;                          // frames on their way (two without gate planes: 1.5 % of a pass slower)
  const float4 one = make_float4(1.f, 1.f, 1.f, 1.f);
  float4 ring[AH], gr[AH];
#pragma unroll
  for (int i = 0; i < AH; ++i) {
    ring[i] = ptr[(size_t)min(i, a.T - 1) * fstride];
    gr[i] = planes ? __ldg(gpl + (size_t)min(i, a.T - 1) * gstride) : one;
  }
  for (int t = 0; t < a.T; ++t) {
    const float4 cur = ring[0], gc = gr[0];
#pragma unroll
    for (int i = 0; i + 1 < AH; ++i) { ring[i] = ring[i + 1]; gr[i] = gr[i + 1]; }
    if (t + AH < a.T) {
      ring[AH - 1] = ptr[AH * fstride];
      if (planes) gr[AH - 1] = __ldg(gpl + (size_t)(t + AH) * gstride);
    }
    // out[t] = bias + sum_j w[j] * s[t - (KT-1) + j]; hist[k] holds s[t - (KT-1) + k]
    float4 o = make_float4(fmaf(w[KT - 1], cur.x, bias), fmaf(w[KT - 1], cur.y, bias),
                           fmaf(w[KT - 1], cur.z, bias), fmaf(w[KT - 1], cur.w, bias));
#pragma unroll
    for (int k = 0; k < KT - 1; ++k) {
      o.x = fmaf(w[k], hist[k].x, o.x); o.y = fmaf(w[k], hist[k].y, o.y);
      o.z = fmaf(w[k], hist[k].z, o.z); o.w = fmaf(w[k], hist[k].w, o.w);
    }
#pragma unroll
    for (int k = 0; k + 1 < KT - 1; ++k) hist[k] = hist[k + 1];
    if (KT > 1) hist[KT - 2] = cur;
    o = make_float4(silu_f(o.x), silu_f(o.y), silu_f(o.z), silu_f(o.w));
    if (gated) {
      const float4* gp = reinterpret_cast<const float4*>(a.bkv + ((size_t)(b * a.T + t) * a.HW + 4 * g4));
      const float4 g0 = __ldg(gp), g1 = __ldg(gp + 1);        // {Bk,Bv} of pixels 0,1 and 2,3
      o.x *= poff ? g0.y : g0.x; o.y *= poff ? g0.w : g0.z;
      o.z *= poff ? g1.y : g1.x; o.w *= poff ? g1.w : g1.z;
    }
    if (planes) { o.x *= gc.x; o.y *= gc.y; o.z *= gc.z; o.w *= gc.w; }
    *ptr = o;
    ptr += fstride;
  }
}

int launch_qkv_temporal_conv(const QkvTconvArgs& a, cudaStream_t st) {
  if (a.HW % 4 != 0 || a.kt < 1) return CSSM_ERR_UNSUPPORTED;
  const long long total = (long long)a.B * 3 * a.C * (a.HW >> 2);
  const unsigned grid = (unsigned)((total + 255) / 256);
  auto go = [&](auto plain, auto planes) { launch_k(a.gsp != nullptr ? planes : plain, grid, 256, 0, st, a); };
  switch (a.kt) {
    case 2: go(qkv_temporal_conv_kernel<2, false>, qkv_temporal_conv_kernel<2, true>); break;
    case 3: go(qkv_temporal_conv_kernel<3, false>, qkv_temporal_conv_kernel<3, true>); break;
    case 4: go(qkv_temporal_conv_kernel<4, false>, qkv_temporal_conv_kernel<4, true>); break;
    default: return CSSM_ERR_UNSUPPORTED;
  }
  return check_launch();
}

// ----------------------------------------------------------- gated gate maps ----
// One CTA per (b,t).  ctx = ctx_sum / (H*W).  Writes, per bin, the float4
// {exp(-D), (D+1e-8)*Bg, Cg/(H*W), 1e-7*(D+1e-8)} at bin_index(path, kh, kw).

__device__ __forceinline__ float gate_act(float x, int act) {
  if (act == CSSM_ACT_SIGMOID2) return 2.0f / (1.0f + expf(-x));
  if (act == CSSM_ACT_EXP_CLIP) return expf(fminf(fmaxf(x, -4.f), 2.f));
  return x > 20.f ? x : log1pf(expf(x));
}

__device__ __forceinline__ float4 gated_map(float rd, float rb, float rc, int act, float inv) {
  const float D = gate_act(rd, act);
  return make_float4(expf(-D), (D + 1e-8f) * rb, rc * inv, 1e-7f * (D + 1e-8f));
}

// Factored gates of FR frames a CTA (the bins of a frame are split over gridDim.y CTAs when there are few frames).  The entries of the six
// vectors go to the lanes, four a lane, the channels in S slices to the warps, so that a weight read serves FR frames and a warp's weights are
// some 16 loads a lane and entry: those of the first 16 channels are on their way before the kernel waits for the one before it (weights are
// older than the chain).  Then the slices' sums meet in shared memory and all threads write the maps.
// (Before: one frame a CTA with all loads behind the wait, 12 us of a pass with 33 frames of 16 x 16 x 256, now 5.5; four frames with the
// matrices copied to shared memory first, 18 us a launch for 192 frames of 14 x 14 x 256, now 6.4.)
constexpr int GF_THREADS = 512, GF_E = 4, GF_U = 16;
struct GateSplit { int S, EC; };           // slices of the channels, chunks of 32 * GF_E entries
template <int FR>
__global__ void __launch_bounds__(GF_THREADS) gated_gates_factored_kernel(const GatedGateArgs g, const GateSplit q) {
  extern __shared__ __align__(16) float sh[];
  const int Wf = g.W / 2 + 1, NB = g.H * Wf, per = g.H + Wf, E = 3 * per, C = g.C;
  float* ctx = sh;                          // [C][FR]
  float* part = sh + C * FR;                // [S][E][FR]
  float* vec = part + q.S * E * FR;         // [E][FR]
  const float inv = 1.0f / (float)(g.H * g.W);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, f0 = blockIdx.x * FR, nf = min(FR, g.BT - f0);
  const int step = (GF_THREADS / 32) / q.S, sl = warp % q.S, c0 = sl * C / q.S, c1 = (sl + 1) * C / q.S;
  auto column = [&](int e, const float*& w, int& ld, const float*& bias) {
    const int m = e / per, r = e - m * per, h = r < g.H ? 0 : 1, col = h ? r - g.H : r;
    const float* k = g.gk[0];
    const float* bp = g.gb[0];
#pragma unroll
    for (int i = 1; i < 6; ++i)
      if (i == 2 * m + h) { k = g.gk[i]; bp = g.gb[i]; }
    w = k + col; bias = bp + col; ld = h ? Wf : g.H;
  };
  const float* wp[GF_E];
  int ld[GF_E];
  float w[GF_E][GF_U];
  auto point = [&](int ec) {
#pragma unroll
    for (int i = 0; i < GF_E; ++i) {
      const float* b;
      column(min((ec * GF_E + i) * 32 + lane, E - 1), wp[i], ld[i], b);
    }
  };
  auto fetch = [&](int c) {
#pragma unroll
    for (int u = 0; u < GF_U; ++u)
#pragma unroll
      for (int i = 0; i < GF_E; ++i) w[i][u] = __ldg(wp[i] + (size_t)min(c + u, C - 1) * ld[i]);
  };
  int ec = warp / q.S;
  const bool busy = ec < step && ec < q.EC;
  point(min(ec, q.EC - 1));
  fetch(c0);
  pdl_sync();
  for (int i = tid; i < C * FR; i += GF_THREADS) {
    const int f = i / C, c = i - f * C;
    ctx[c * FR + f] = f < nf ? __ldg(g.ctx_sum + (size_t)(f0 + f) * C + c) * inv : 0.f;
  }
  __syncthreads();
  if (busy) {
    for (bool first = true; ec < q.EC; ec += step, first = false) {
      if (!first) { point(ec); fetch(c0); }
      float acc[GF_E][FR];
#pragma unroll
      for (int i = 0; i < GF_E; ++i)
#pragma unroll
        for (int f = 0; f < FR; ++f) acc[i][f] = 0.f;
      for (int c = c0; c < c1; c += GF_U) {
        if (c > c0) fetch(c);
#pragma unroll
        for (int u = 0; u < GF_U; ++u) {
          if (c + u >= c1) break;
#pragma unroll
          for (int f = 0; f < FR; ++f) {
            const float x = ctx[(c + u) * FR + f];
#pragma unroll
            for (int i = 0; i < GF_E; ++i) acc[i][f] = fmaf(x, w[i][u], acc[i][f]);
          }
        }
      }
#pragma unroll
      for (int i = 0; i < GF_E; ++i) {
        const int e = (ec * GF_E + i) * 32 + lane;
        if (e < E) {
#pragma unroll
          for (int f = 0; f < FR; ++f) part[(sl * E + e) * FR + f] = acc[i][f];
        }
      }
    }
  }
  __syncthreads();
  for (int i = tid; i < E * FR; i += GF_THREADS) {
    const int e = i / FR;
    const float *k, *b;
    int l;
    column(e, k, l, b);
    float v = __ldg(b);
    for (int t = 0; t < q.S; ++t) v += part[t * E * FR + i];
    vec[i] = v;
  }
  __syncthreads();
  const int per_cta = (NB + gridDim.y - 1) / gridDim.y, b0 = blockIdx.y * per_cta, nb = min(per_cta, NB - b0);
  for (int i = tid; i < nf * nb; i += GF_THREADS) {
    const int f = i / nb, bin = b0 + i - f * nb, kh = bin / Wf, kw = bin - kh * Wf;
    float r[3];
#pragma unroll
    for (int gi = 0; gi < 3; ++gi) r[gi] = vec[(gi * per + kh) * FR + f] * vec[(gi * per + g.H + kw) * FR + f];
    g.maps[(size_t)(f0 + f) * NB + bin_index(g.path, kh, kw, g.H, Wf)] = gated_map(r[0], r[1], r[2], g.act, inv);
  }
}

// Dense gates: a thread owns one bin of G frames, so that a weight read serves all of them (one frame per
// read moved 80 MB of weights through L2 for 128 frames of 56 x 56 x 32).
template <int G>
__global__ void __launch_bounds__(128) gated_gates_dense_kernel(const GatedGateArgs g) {
  extern __shared__ __align__(16) float sh[];
  const int Wf = g.W / 2 + 1, NB = g.H * Wf, f0 = blockIdx.x * G, nf = min(G, g.BT - f0);
  const float inv = 1.0f / (float)(g.H * g.W);
  pdl_sync();
  const GateCtxSrc src = {g.ctx_sum, nullptr, nullptr, 1, g.C, g.H, 0, inv};
  gate_ctx(src, f0, nf, sh, sh + G * g.C);
  const int bin = blockIdx.y * 128 + threadIdx.x;
  if (bin >= NB) return;
  float r[3][G];
  gate_dense<3, G>(g.gk, g.gb, NB, bin, g.C, sh, r);
  const int kh = bin / Wf, o = bin_index(g.path, kh, bin - kh * Wf, g.H, Wf);
#pragma unroll
  for (int f = 0; f < G; ++f)
    if (f < nf) g.maps[(size_t)(f0 + f) * NB + o] = gated_map(r[0][f], r[1][f], r[2][f], g.act, inv);
}

int launch_gated_gates(const GatedGateArgs& g, cudaStream_t st) {
  const int Wf = g.W / 2 + 1, NB = g.H * Wf;
  if (g.gate_type == CSSM_GATE_FACTORED) {
    const int E = 3 * (g.H + Wf), sms = sm_count();
    GateSplit q;
    q.EC = (E + 32 * GF_E - 1) / (32 * GF_E);
    q.S = q.EC < GF_THREADS / 32 ? GF_THREADS / 32 / q.EC : 1;
    // Frames a CTA: the classifier's pass with 1, 2, 4: 32 images 488, 490, 492 us; 48 images of T = 8 (192 frames) 774, 762, 765; 256
    // images 1922, 1911, 1912; 512 3590, 3565, 3552.
    const int FR = g.BT >= 3 * sms ? 4 : g.BT >= sms ? 2 : 1;
    const size_t smem = (size_t)FR * (g.C + (q.S + 1) * E) * sizeof(float);
    const dim3 grid((g.BT + FR - 1) / FR, gate_chunks((g.BT + FR - 1) / FR, NB));
    return launch_gates(FR == 4 ? gated_gates_factored_kernel<4> : FR == 2 ? gated_gates_factored_kernel<2> : gated_gates_factored_kernel<1>, grid,
                        GF_THREADS, smem, st, g, q);
  }
  const int chunks = (NB + 127) / 128, G = gate_dense_frames(g.BT, chunks, g.C);
  const dim3 grid((g.BT + G - 1) / G, chunks);
  const size_t smem = (size_t)(G * g.C + 128) * sizeof(float);
  return launch_gates(G == 8 ? gated_gates_dense_kernel<8> : G == 4 ? gated_gates_dense_kernel<4> : gated_gates_dense_kernel<1>,
                      grid, 128, smem, st, g);
}

}  // namespace cssm
