// GDN block, kernels ahead of the spectral stage: RoPE + channels-last depthwise conv with
// per-row context sums, and the gate maps (alpha, beta per frequency bin; B_k, B_v per pixel).
#include <type_traits>
#include "kernels.cuh"
#include "bf16_ops.cuh"
#include "gates.cuh"

namespace cssm {

// ------------------------------------------------- RoPE + depthwise KxK, channels-last ----
// One CTA per (frame, band of DW_ROWS output rows, group of 16 channels).  The band's input
// rows (+ halo) are rotated (RoPE) while they are staged in shared memory as [row][w][16];
// each thread then produces DW_ROWS x 4 outputs for one channel from there.  The CTA also
// writes, per centre row and channel, the sum over w of the ROTATED INPUT (ctx is the mean of
// the block input, cssm.py:4785-4786), not of the conv output.
constexpr int DW_ROWS = 8, DW_THREADS = 256;

// Position of (padded column col, channel c) inside a staged row.  With 16 channels per pixel two
// pixels share a 32-float line; the halves swap with bit 2 of the column, so that the two
// half-warps of a window read (columns col and col + 4, same channels) hit different banks.
template <int DW_CG>
__device__ __forceinline__ int dw_pos(int col, int c) {
  if (DW_CG == 16) return ((col >> 1) << 5) + ((((col & 1) ^ ((col >> 2) & 1))) << 4) + c;
  return col * DW_CG + c;
}

// BC: one source frame for all T frames of a clip (a.x_bcast).  The frames differ by the t part of the
// angle alone, one rotation per pair for the whole plane, and that commutes with the sums of the conv up
// to the two channels' weights: with p = conv(w_e, x_e | w_o, x_o) and q = conv(w_e, x_o | w_o, x_e) of the
// plane rotated by (h, w),  out_e = p_e cos - q_e sin,  out_o = p_o cos + q_o sin.  So a CTA stages and
// convolves once (two products) for all T frames instead of T times; what is left is the output's write.
// 5x5, one 64x64 image over eight frames, batch 128, 64 channels: 1021 -> 372 us; the frames' stores without a bound and an address each 267.
template <int K, int DW_CG, bool BC>
__global__ void __launch_bounds__(DW_THREADS, (K <= 5 ? 2 : 1)) rope_dwconv_cl_kernel(const GdnDwArgs a) {
  pdl_sync();
  extern __shared__ __align__(16) float sm[];
  constexpr int LO = (K - 1) / 2, NR = DW_ROWS + K - 1;
  const int W = a.W, C = a.C, n2 = C / 2;
  const int WP = (W + K - 1 + 1) & ~1;                 // padded columns per staged row (even)
  const int rpitch = WP * DW_CG;                        // floats per staged row
  const int bands = (a.H + DW_ROWS - 1) / DW_ROWS, cgs = C / DW_CG;
  int bid = blockIdx.x;
  const int cg = bid % cgs; bid /= cgs;
  const int band = bid % bands;
  const int fr = bid / bands;
  const int t = fr % a.T, h0 = band * DW_ROWS, c0 = cg * DW_CG;
  const int fsrc = !BC && a.x_bcast ? fr / a.T : fr;   // BC: fr counts clips
  const int tid = threadIdx.x;
  // ---- zero the pad columns (left LO, right up to WP) of every staged row ----
  for (int i = tid; i < NR * (WP - W) * DW_CG; i += DW_THREADS) {
    const int r = i / ((WP - W) * DW_CG), rem = i - r * (WP - W) * DW_CG;
    const int pc = rem / DW_CG, c = rem - pc * DW_CG;
    const int col = pc < LO ? pc : W + pc;               // 0..LO-1, then W+LO..WP-1
    sm[r * rpitch + dw_pos<DW_CG>(col, c)] = 0.f;
  }
  // ---- stage rows h0-LO .. h0+DW_ROWS-1+(K-1-LO), DW_CG channels, rotated ----
  // DW_THREADS is a multiple of the pairs per pixel, so a thread keeps its channel pair and walks
  // columns wb, wb + WSTEP of every staged row: the t part of the angle is loaded once, the w part
  // once per column, the h part once per row.  Four rows x two columns are fetched per trip, every
  // load issued before the first is used.
  constexpr int PP = DW_CG / 2;                         // pairs per pixel in this channel group
  constexpr int WSTEP = DW_THREADS / PP;
  const int pl = tid % PP, pi = c0 / 2 + pl;
  const bool rope = a.rope_t != nullptr;
  float2 ct = make_float2(1.f, 0.f);
  if (rope && !BC) ct = a.rope_t[t * n2 + pi];
  const float* xf = a.x + (size_t)fsrc * a.H * W * C + c0 + 2 * pl;
  for (int wb = tid / PP; wb < W; wb += 2 * WSTEP) {
    float2 cw[2];
    int spos[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int w = wb + k * WSTEP;
      cw[k] = (rope && w < W) ? __ldg(&a.rope_w[w * n2 + pi]) : make_float2(1.f, 0.f);
      spos[k] = dw_pos<DW_CG>(min(w, W - 1) + LO, 2 * pl);
    }
#pragma unroll
    for (int r0 = 0; r0 < NR; r0 += 4) {
      float2 v[4][2];
#pragma unroll
      for (int r4 = 0; r4 < 4; ++r4) {
        const int hh = h0 + r0 + r4 - LO;
        const bool rin = r0 + r4 < NR && hh >= 0 && hh < a.H;
#pragma unroll
        for (int k = 0; k < 2; ++k)
          v[r4][k] = (rin && wb + k * WSTEP < W)
                         ? __ldg(reinterpret_cast<const float2*>(xf + ((size_t)hh * W + wb + k * WSTEP) * C))
                         : make_float2(0.f, 0.f);
      }
#pragma unroll
      for (int r4 = 0; r4 < 4; ++r4) {
        if (r0 + r4 >= NR) continue;
        const int hh = h0 + r0 + r4 - LO;
        float cth = 1.f, sth = 0.f;
        if (rope && hh >= 0 && hh < a.H) {
          const float2 ch = __ldg(&a.rope_h[hh * n2 + pi]);
          cth = ct.x * ch.x - ct.y * ch.y; sth = ct.x * ch.y + ct.y * ch.x;
        }
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          if (wb + k * WSTEP >= W) continue;
          const float c2 = cth * cw[k].x - sth * cw[k].y, s2 = cth * cw[k].y + sth * cw[k].x;
          const float2 o = make_float2(v[r4][k].x * c2 - v[r4][k].y * s2, v[r4][k].x * s2 + v[r4][k].y * c2);
          *reinterpret_cast<float2*>(sm + (r0 + r4) * rpitch + spos[k]) = o;
        }
      }
    }
  }
  __syncthreads();
  // ---- context partial sums of the centre rows ----
  if (BC && a.ctx_part != nullptr) {
    // four lanes per (row, pair) of the row sums, each frame rotated by its t part
    constexpr int NI = DW_ROWS * PP * 4;
    for (int i = tid; i < NI; i += DW_THREADS) {         // NI is a multiple of the warp size
      const int qd = i & 3, pr = (i >> 2) % PP, r = (i >> 2) / PP;
      float se = 0.f, so = 0.f;
      const float* srow = sm + (r + LO) * rpitch;
      for (int w = qd; w < W; w += 4) {
        const float2 v = *reinterpret_cast<const float2*>(srow + dw_pos<DW_CG>(w + LO, 2 * pr));
        se += v.x; so += v.y;
      }
#pragma unroll
      for (int off = 1; off < 4; off <<= 1) {
        se += __shfl_xor_sync(0xffffffffu, se, off); so += __shfl_xor_sync(0xffffffffu, so, off);
      }
      if (h0 + r < a.H)
        for (int f = qd; f < a.T; f += 4) {
          const float2 cf2 = rope ? __ldg(&a.rope_t[f * n2 + c0 / 2 + pr]) : make_float2(1.f, 0.f);
          *reinterpret_cast<float2*>(a.ctx_part + (((size_t)fr * a.T + f) * a.H + h0 + r) * C + c0 + 2 * pr) =
              make_float2(se * cf2.x - so * cf2.y, se * cf2.y + so * cf2.x);
        }
    }
  }
  if (!BC && a.ctx_part != nullptr && tid < DW_ROWS * DW_CG) {
    const int r = tid / DW_CG, c = tid % DW_CG;
    if (h0 + r < a.H) {
      float s = 0.f;
      const float* srow = sm + (r + LO) * rpitch;
      for (int w = 0; w < W; ++w) s += srow[dw_pos<DW_CG>(w + LO, c)];
      a.ctx_part[((size_t)fr * a.H + h0 + r) * C + c0 + c] = s;
    }
  }
  if (a.out == nullptr) return;
  // ---- conv: thread = (channel pair, two consecutive w), all DW_ROWS rows; packed f32x2 FMAs ----
  // The staged pairs are read with 8-byte loads as they lie.  With eight pairs per pixel a warp holds
  // four column pairs; they are taken in the order 0, 2, 1, 3 so that the two of a half-warp are four
  // columns apart and land in different halves of the swizzled 128-byte lines.
  unsigned long long wk2[K * K];
#pragma unroll
  for (int i = 0; i < K * K; ++i) {
    const float2 w2 = *reinterpret_cast<const float2*>(a.wk + (size_t)i * C + c0 + 2 * pl);
    wk2[i] = pk2(w2.x, w2.y);
  }
  const float2 b2 = *reinterpret_cast<const float2*>(a.bias + c0 + 2 * pl);
  const unsigned long long bias2 = pk2(b2.x, b2.y);
  const int q = tid / PP;
  const int qs = PP == 8 ? ((q & ~3) | ((q & 1) << 1) | ((q >> 1) & 1)) : q;
  for (int wg = qs; wg * 2 < W; wg += WSTEP) {
    const int w0 = wg * 2;
    // offsets of the window's padded columns w0 .. w0+K inside a staged row (same for all rows)
    int off[2 + K - 1];
#pragma unroll
    for (int j = 0; j < 2 + K - 1; ++j) off[j] = dw_pos<DW_CG>(min(w0 + j, WP - 1), 2 * pl);
    if (BC) {
      constexpr int RC = DW_ROWS / 2;                    // output rows at a time (registers)
#pragma unroll 1
      for (int rc = 0; rc < DW_ROWS && h0 + rc < a.H; rc += RC) {
        unsigned long long p[RC][2], qx[RC][2];
#pragma unroll
        for (int r = 0; r < RC; ++r) p[r][0] = p[r][1] = qx[r][0] = qx[r][1] = 0ull;
#pragma unroll
        for (int ir = 0; ir < RC + K - 1; ++ir) {
          const float* srow = sm + (rc + ir) * rpitch;
          unsigned long long win[2 + K - 1], swp[2 + K - 1];
#pragma unroll
          for (int j = 0; j < 2 + K - 1; ++j) {
            const float2 v = *reinterpret_cast<const float2*>(srow + off[j]);
            win[j] = pk2(v.x, v.y); swp[j] = pk2(v.y, v.x);
          }
#pragma unroll
          for (int di = 0; di < K; ++di) {
            const int r = ir - di;
            if (r < 0 || r >= RC) continue;
#pragma unroll
            for (int dj = 0; dj < K; ++dj)
#pragma unroll
              for (int j = 0; j < 2; ++j) {
                p[r][j] = fma2(wk2[di * K + dj], win[dj + j], p[r][j]);
                qx[r][j] = fma2(wk2[di * K + dj], swp[dj + j], qx[r][j]);
              }
          }
        }
        // (whole windows, as all are of planes of a multiple of eight rows and even width, without a test at every store)
        float* orow = a.out + (((size_t)fr * a.T * a.H + h0 + rc) * W + w0) * C + c0 + 2 * pl;
        const size_t fstep = (size_t)a.H * W * C;
        const int wc = W * C;
        auto frames = [&](auto all) {
          float* o = orow;
          float2 cn = rope ? __ldg(&a.rope_t[pi]) : make_float2(1.f, 0.f);
#pragma unroll 1
          for (int f = 0; f < a.T; ++f, o += fstep) {
            const float2 cf2 = cn;
            if (rope && f + 1 < a.T) cn = __ldg(&a.rope_t[(f + 1) * n2 + pi]);
            const unsigned long long c2 = pk2(cf2.x, cf2.x), s2 = pk2(-cf2.y, cf2.y);
#pragma unroll
            for (int r = 0; r < RC; ++r)
#pragma unroll
              for (int j = 0; j < 2; ++j)
                if (decltype(all)::value || (h0 + rc + r < a.H && w0 + j < W))
                  *reinterpret_cast<unsigned long long*>(o + r * wc + j * C) = fma2(s2, qx[r][j], fma2(c2, p[r][j], bias2));
          }
        };
        if (h0 + rc + RC <= a.H && w0 + 1 < W) frames(std::true_type());
        else frames(std::false_type());
      }
      continue;
    }
    unsigned long long acc[DW_ROWS][2];
#pragma unroll
    for (int r = 0; r < DW_ROWS; ++r) { acc[r][0] = bias2; acc[r][1] = bias2; }
#pragma unroll
    for (int ir = 0; ir < NR; ++ir) {
      const float* srow = sm + ir * rpitch;
      unsigned long long win[2 + K - 1];
#pragma unroll
      for (int j = 0; j < 2 + K - 1; ++j)
        win[j] = *reinterpret_cast<const unsigned long long*>(srow + off[j]);   // pad columns hold zeros
      // input row ir feeds output row r = ir - di for tap row di
#pragma unroll
      for (int di = 0; di < K; ++di) {
        const int r = ir - di;
        if (r < 0 || r >= DW_ROWS) continue;
#pragma unroll
        for (int dj = 0; dj < K; ++dj) {
          acc[r][0] = fma2(wk2[di * K + dj], win[dj], acc[r][0]);
          acc[r][1] = fma2(wk2[di * K + dj], win[dj + 1], acc[r][1]);
        }
      }
    }
    float* orow = a.out + (((size_t)fr * a.H + h0) * W + w0) * C + c0 + 2 * pl;
#pragma unroll
    for (int r = 0; r < DW_ROWS; ++r) {
      if (h0 + r >= a.H) continue;
#pragma unroll
      for (int j = 0; j < 2; ++j)
        if (w0 + j < W) {
          float ox, oy;
          upk2(acc[r][j], ox, oy);
          *reinterpret_cast<float2*>(orow + ((size_t)r * W + j) * C) = make_float2(ox, oy);
        }
    }
  }
}

// ------------------------------------------- context row sums without a conv (K = 1) ----
// ctx_part[(frame, h, c)] = sum over w of the rotated input.  One warp per image row of a source frame: a lane owns one
// or more float4 channel groups, 32 / (C / 4) pixels side by side where C < 128, and walks the row eight 16-byte loads at a time.
// Rotations commute, so the loop turns by the w part of the angle alone; the h and t parts turn the finished sums,
// for every frame t of the clip where one source frame stands for all.
// Bound: HBM (with 8-byte loads, four in flight, and the whole angle per element the kernel before ran at a quarter of its
// rate): 128 x 32 frames of 32x32x64 316 -> 192 us (floor 165), 12 x 8 of 64x64x64 57 -> 27.
constexpr int CTX_WARPS = 4;
__global__ void __launch_bounds__(CTX_WARPS * 32) rope_ctx_rowsum_kernel(const GdnDwArgs a) {
  pdl_sync();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int copies = a.x_bcast ? a.T : 1, frames = a.BT / copies;
  const long long row = (long long)blockIdx.x * CTX_WARPS + warp;        // (source frame, h)
  if (row >= (long long)frames * a.H) return;
  const int fr = (int)(row / a.H), h = (int)(row % a.H);
  const int n2 = a.C / 2, c4 = a.C / 4, wide = c4 < 32 ? 32 / c4 : 1, sub = c4 < 32 ? lane / c4 : 0;
  const bool rope = a.rope_t != nullptr;
  const float4* xr = reinterpret_cast<const float4*>(a.x + (size_t)row * a.W * a.C);
  for (int j0 = 0; j0 < c4; j0 += 32) {
    const int j = j0 + (c4 < 32 ? lane - sub * c4 : lane);
    const bool on = j < c4 && sub < wide;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    if (on) {
      const float4* rw = reinterpret_cast<const float4*>(a.rope_w) + j;
#pragma unroll 1
      for (int w0 = sub; w0 < a.W; w0 += 8 * wide) {
        float4 v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int w = w0 + u * wide;
          v[u] = w < a.W ? __ldg(xr + (size_t)w * c4 + j) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int w = w0 + u * wide;
          if (rope) {
            const float4 c = __ldg(rw + (size_t)min(w, a.W - 1) * c4);
            s.x = fmaf(v[u].x, c.x, fmaf(-v[u].y, c.y, s.x)); s.y = fmaf(v[u].x, c.y, fmaf(v[u].y, c.x, s.y));
            s.z = fmaf(v[u].z, c.z, fmaf(-v[u].w, c.w, s.z)); s.w = fmaf(v[u].z, c.w, fmaf(v[u].w, c.z, s.w));
          } else {
            s.x += v[u].x; s.y += v[u].y; s.z += v[u].z; s.w += v[u].w;
          }
        }
      }
    }
    for (int k = 1; k < wide; ++k) {                  // sums of the other pixels side by side
      const int from = (lane + k * c4) & 31;
      const float4 o = make_float4(__shfl_sync(0xffffffffu, s.x, from), __shfl_sync(0xffffffffu, s.y, from),
                                   __shfl_sync(0xffffffffu, s.z, from), __shfl_sync(0xffffffffu, s.w, from));
      if (sub == 0) { s.x += o.x; s.y += o.y; s.z += o.z; s.w += o.w; }
    }
    if (on && sub == 0) {
      if (rope) {
        const float4 c = __ldg(reinterpret_cast<const float4*>(a.rope_h + (size_t)h * n2) + j);
        s = make_float4(s.x * c.x - s.y * c.y, s.x * c.y + s.y * c.x, s.z * c.z - s.w * c.w, s.z * c.w + s.w * c.z);
      }
      for (int k = 0; k < copies; ++k) {
        float4 o = s;
        if (rope) {
          const int t = a.x_bcast ? k : fr % a.T;
          const float4 c = __ldg(reinterpret_cast<const float4*>(a.rope_t + (size_t)t * n2) + j);
          o = make_float4(s.x * c.x - s.y * c.y, s.x * c.y + s.y * c.x, s.z * c.z - s.w * c.w, s.z * c.w + s.w * c.z);
        }
        *reinterpret_cast<float4*>(a.ctx_part + (((size_t)fr * copies + k) * a.H + h) * a.C + 4 * j) = o;
      }
    }
  }
}

template <int K, int DW_CG, bool BC>
static int launch_dw_cg(const GdnDwArgs& a, cudaStream_t st) {
  const size_t smem = (size_t)(DW_ROWS + K - 1) * ((a.W + K - 1 + 1) & ~1) * DW_CG * sizeof(float);
  if (smem > 200 * 1024) return CSSM_ERR_UNSUPPORTED;
  cudaError_t e = func_smem(rope_dwconv_cl_kernel<K, DW_CG, BC>, smem);
  if (e != cudaSuccess) { set_cuda_error(e); return CSSM_ERR_CUDA; }
  const int bands = (a.H + DW_ROWS - 1) / DW_ROWS;
  launch_k(rope_dwconv_cl_kernel<K, DW_CG, BC>, (BC ? a.BT / a.T : a.BT) * bands * (a.C / DW_CG), DW_THREADS, smem, st, a);
  return check_launch();
}

// 16-channel groups (64-byte segments per pixel) when C allows, else 4-channel groups
template <int K>
static int launch_dw(const GdnDwArgs& a, cudaStream_t st) {
  // one source frame for four or more frames: the doubled conv costs less than the repeated ones
  if (K > 1 && a.x_bcast && a.T >= 4 && a.C % 16 == 0) return launch_dw_cg<K, 16, K != 1>(a, st);
  return a.C % 16 == 0 ? launch_dw_cg<K, 16, false>(a, st) : launch_dw_cg<K, 4, false>(a, st);
}

int launch_rope_dwconv_cl(const GdnDwArgs& a, cudaStream_t st) {
  if (a.C % 4 != 0) return CSSM_ERR_UNSUPPORTED;
  if (a.ksz <= 1 && a.out == nullptr) {
    if (a.ctx_part == nullptr) return CSSM_OK;
    const long long rows = (long long)(a.x_bcast ? a.BT / a.T : a.BT) * a.H;
    launch_k(rope_ctx_rowsum_kernel, (unsigned)((rows + CTX_WARPS - 1) / CTX_WARPS), CTX_WARPS * 32, 0, st, a);
    return check_launch();
  }
  switch (a.ksz > 1 ? a.ksz : 1) {
    case 1: return launch_dw<1>(a, st);
    case 3: return launch_dw<3>(a, st);
    case 5: return launch_dw<5>(a, st);
    case 7: return launch_dw<7>(a, st);
    default: return CSSM_ERR_UNSUPPORTED;
  }
}

// ------------------------------------------------------------------- GDN gate maps ----
// One CTA per frame.  ctx = (sum over rows of ctx_part) / (H*W) + tcode[t].
// alpha/beta: sigmoid(row[h] + col[kw]) (factored) or sigmoid(Dense(H*Wf)) (dense);
// alpha = 0.1 + 0.89 * raw.  Stored as float2 {alpha, beta} at bin_index(path, kh, kw).
// B_k / B_v: same over (h, w) pixels, float2 {B_k, B_v} at h*W + w.  cssm.py:4798-4848, 4864-4865.
__global__ void __launch_bounds__(256, 5) gdn_gates_kernel(const GdnGateArgs g) {
  extern __shared__ __align__(16) float sh[];
  const int Wf = g.W / 2 + 1, NB = g.H * Wf, HW = g.H * g.W;
  float* ctx = sh;                       // [C]
  float* scratch = sh + g.C;             // [256]
  float* vec = scratch + 256;            // factored: alpha_h, alpha_w, beta_h, beta_w, Bk_h, Bk_w, Bv_h, Bv_w
  const int fr = blockIdx.x, tid = threadIdx.x;
  pdl_sync();
  const GateCtxSrc src = {nullptr, g.ctx_part, g.tcode, g.T, g.C, g.H, g.ctx_per_clip, 1.0f / (float)HW};
  gate_ctx(src, fr, 1, ctx, scratch);
  const int ngate = g.use_input_gates ? 4 : 2;
  if (g.gate_type == CSSM_GATE_FACTORED) {
    // segment offsets inside vec
    int off[9];
    off[0] = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int wd = q < 2 ? Wf : g.W;
      off[2 * q + 1] = off[2 * q] + g.H;
      off[2 * q + 2] = off[2 * q + 1] + wd;
    }
    if (g.use_input_gates) gate_vectors<8>(g.gk, g.gb, off, 8, ctx, g.C, vec, scratch);
    else gate_vectors<8>(g.gk, g.gb, off, 4, ctx, g.C, vec, scratch);
    for (int bin = tid; bin < NB; bin += blockDim.x) {
      const int kh = bin / Wf, kw = bin % Wf;
      const float ra = sigmoid_f(vec[off[0] + kh] + vec[off[1] + kw]);
      const float rb = sigmoid_f(vec[off[2] + kh] + vec[off[3] + kw]);
      g.ab[(size_t)fr * NB + bin_index(g.path, kh, kw, g.H, Wf)] = make_float2(0.1f + 0.89f * ra, rb);
    }
    if (g.use_input_gates)
      for (int px = tid; px < HW; px += blockDim.x) {
        const int h = px / g.W, w = px % g.W;
        g.bkv[(size_t)fr * HW + px] = make_float2(sigmoid_f(vec[off[4] + h] + vec[off[5] + w]),
                                                  sigmoid_f(vec[off[6] + h] + vec[off[7] + w]));
      }
  } else {
    // scalar: one value per frame and gate, Dense(1)(ctx) (cssm.py:4825-4833).  channel: alpha, beta
    // per head, Dense(n_h)(ctx) (cssm.py:4808-4810); its spatial gates are a 1x1 conv of the block
    // input and are applied elsewhere.  The maps are constant over the bins.
    const bool chan = g.gate_type == CSSM_GATE_CHANNEL;
    const int nout = chan ? g.nh : 1, nvec = chan ? 2 : ngate;
    const int off[9] = {0, nout, 2 * nout, 3 * nout, 4 * nout, 0, 0, 0, 0};
    gate_vectors<8>(g.gk, g.gb, off, nvec, ctx, g.C, vec, scratch);
    for (int o = tid; o < nvec * nout; o += blockDim.x) vec[o] = sigmoid_f(vec[o]);
    __syncthreads();
    for (int i = tid; i < nout * NB; i += blockDim.x) {
      const int hh = i / NB;
      g.ab[((size_t)fr * nout + hh) * NB + (i - hh * NB)] = make_float2(0.1f + 0.89f * vec[hh], vec[nout + hh]);
    }
    if (!chan && g.use_input_gates)
      for (int px = tid; px < HW; px += blockDim.x) g.bkv[(size_t)fr * HW + px] = make_float2(vec[2], vec[3]);
  }
}

// Dense gates: a thread owns one bin (blockIdx.y < bin_chunks) or one pixel of G frames.
template <int G>
__global__ void __launch_bounds__(128) gdn_gates_dense_kernel(const GdnGateArgs g, int bin_chunks) {
  extern __shared__ __align__(16) float sh[];
  const int Wf = g.W / 2 + 1, NB = g.H * Wf, HW = g.H * g.W, f0 = blockIdx.x * G, nf = min(G, g.BT - f0);
  pdl_sync();
  const GateCtxSrc src = {nullptr, g.ctx_part, g.tcode, g.T, g.C, g.H, g.ctx_per_clip, 1.0f / (float)HW};
  gate_ctx(src, f0, nf, sh, sh + G * g.C);
  const bool bins = (int)blockIdx.y < bin_chunks;
  const int i = (blockIdx.y - (bins ? 0 : bin_chunks)) * 128 + threadIdx.x, n = bins ? NB : HW;
  if (i >= n) return;
  float r[2][G];
  gate_dense<2, G>(g.gk + (bins ? 0 : 2), g.gb + (bins ? 0 : 2), n, i, g.C, sh, r);
  const int kh = i / Wf, o = bin_index(g.path, kh, i - kh * Wf, g.H, Wf);
#pragma unroll
  for (int f = 0; f < G; ++f) {
    if (f >= nf) continue;
    const float a = sigmoid_f(r[0][f]), b = sigmoid_f(r[1][f]);
    if (bins) g.ab[(size_t)(f0 + f) * NB + o] = make_float2(0.1f + 0.89f * a, b);
    else g.bkv[(size_t)(f0 + f) * HW + i] = make_float2(a, b);
  }
}

int launch_gdn_gates(const GdnGateArgs& g, cudaStream_t st) {
  const int Wf = g.W / 2 + 1;
  if (g.gate_type == CSSM_GATE_DENSE) {
    const int bc = (g.H * Wf + 127) / 128, chunks = bc + (g.use_input_gates ? (g.H * g.W + 127) / 128 : 0);
    const int G = gate_dense_frames(g.BT, chunks, g.C);
    const dim3 grid((g.BT + G - 1) / G, chunks);
    const size_t smem = (size_t)(G * g.C + 128) * sizeof(float);
    return launch_gates(G == 8 ? gdn_gates_dense_kernel<8> : G == 4 ? gdn_gates_dense_kernel<4> : gdn_gates_dense_kernel<1>,
                        grid, 128, smem, st, g, bc);
  }
  const size_t smem = (size_t)(g.C + 256 + 4 * g.H + 2 * Wf + 2 * g.W + 4 * g.nh + 8) * sizeof(float);
  // (it starts beside or behind a projection; packed, 8 frames of 64 x 64 x 64: the SimpleCSSM pass 244 -> 237 us without)
  return launch_gates(gdn_gates_kernel, g.BT, 256, spread_smem(smem, g.BT), st, g);
}

}  // namespace cssm
