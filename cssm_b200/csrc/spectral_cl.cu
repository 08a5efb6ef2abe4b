// Fused spectral kernel of the gated block for the small planes of the CSSM-SHViT stages
// (14 x 14 and 7 x 7) at T = 1, on bf16 channels-last activations:
//   y[n, p, c] = irfft2( C * floor((Delta + 1e-8) * B * rfft2(x[n, :, c])) )[p] * z[n, p, c]
// (at T = 1 the state is h_1 = U_1, so the kernel spectrum K_hat does not enter; z arrives already
// through SiLU).  TPP threads per (sample, channel) plane, PL channels of one sample per CTA: a thread takes pairs of rows h and
// h + ceil(N / 2), packed into one complex FFT (csrc/lane_fft.cuh) and separated in its registers, and whole spectrum columns.  The half
// spectrum of the plane (N x (N/2+1) complex) waits in shared memory between
// the passes as fp16 pairs [bin][plane] (conflict-free; the row pass scales by 1/N so that the
// values stay in range, fp16's 11 significant bits are finer than the bf16 output): 55 KB per CTA of 64 planes
// instead of 84 KB with fp32, four CTAs = 16 warps per SM instead of 4 warps.  The input tile, the z
// tile and the output tile share one [pixel][PL] bf16 buffer that is filled and drained with
// 16-byte accesses, so HBM sees x, z and y once each as full rows.
//
// Bound at full batches: the FMA pipe (about 27 operations a value).  14 x 14 x 256, 512 images: 7-point DFTs of every row and column by their
// definition 80 us a launch, lane FFTs of row pairs 50; the classifier's pass 3619 -> 3566 us.  Few images: a thread's chain of transforms, so
// sixteen channels a CTA with a thread for every row pair and column (one image 209 -> 200 us a pass).
#include <cuda_fp16.h>
#include "kernels.cuh"
#include "bf16_ops.cuh"
#include "lane_fft.cuh"

namespace cssm {

constexpr int SCL_PL = 64;             // the channels are a multiple of this

template <int N, int PL, int TPP>
__global__ void __launch_bounds__(PL * TPP)
gated_spectral_cl_kernel(const __nv_bfloat16* __restrict__ xz, int ld, int C,
                         const float4* __restrict__ gates, __nv_bfloat16* __restrict__ y, int ldy) {
  pdl_sync();
  constexpr int Wf = N / 2 + 1, P = N * N, NB = N * Wf, TPB = PL * TPP, V = PL / 8;
  constexpr int RP = (N + 1) / 2;                    // row pairs
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __half2* R = reinterpret_cast<__half2*>(smem_raw);                      // [NB][PL] (re, im)
  __nv_bfloat16* tile = reinterpret_cast<__nv_bfloat16*>(R + NB * PL);    // [P][PL]
  float4* gs = reinterpret_cast<float4*>(tile + P * PL);                  // [NB]
  const int tid = threadIdx.x, pl = tid % PL, part = tid / PL;
  const int slices = C / PL;
  const int n = blockIdx.x / slices, c0 = (blockIdx.x % slices) * PL;
  const __nv_bfloat16* xin = xz + (size_t)n * P * ld + c0;

  // ---- stage x tile and the sample's gate map ----
  // (asynchronous 16-byte copies: every request of the tile is in flight at once)
  auto fill = [&](const __nv_bfloat16* src) {
    for (int q = tid; q < P * V; q += TPB) {
      const int p = q / V, j = q % V;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;"
                   ::"r"((uint32_t)__cvta_generic_to_shared(tile + p * PL + j * 8)),
                     "l"(src + (size_t)p * ld + j * 8) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fill(xin);
  for (int i = tid; i < NB; i += TPB) gs[i] = __ldg(gates + (size_t)n * NB + i);
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();

  // ---- forward rows, scaled by 1/N (and 1/2 for the separation) ----
#pragma unroll 1
  for (int h = part; h < RP; h += TPP) {
    const bool two = h + RP < N;
    cf z[N];
#pragma unroll
    for (int w = 0; w < N; ++w) {
      const float a = __bfloat162float(tile[(h * N + w) * PL + pl]), b = two ? __bfloat162float(tile[((h + RP) * N + w) * PL + pl]) : 0.f;
      z[w] = mk(a * (0.5f / N), b * (0.5f / N));
    }
    lane_dft<N>(z);
#pragma unroll
    for (int k = 0; k < Wf; ++k) {
      const cf u = z[k], v = z[(N - k) % N];
      R[(h * Wf + k) * PL + pl] = __floats2half2_rn(u.x + v.x, u.y - v.y);
      if (two) R[((h + RP) * Wf + k) * PL + pl] = __floats2half2_rn(u.y + v.y, v.x - u.x);
    }
  }
  __syncthreads();                      // x tile consumed; row spectra of all threads visible
  // ---- z tile (already through SiLU) into the same buffer ----
  // (asynchronous copies again: they land while the column pass runs)
  fill(xin + C);

  // ---- columns: forward DFT, gates (T = 1: h = U), inverse DFT (the forward one of the values with their parts exchanged) ----
#pragma unroll 1
  for (int k = part; k < Wf; k += TPP) {
    cf v[N];
#pragma unroll 1
    for (int back = 0; back < 2; ++back) {
      if (back == 0) {
#pragma unroll
        for (int h = 0; h < N; ++h) {
          const float2 t = __half22float2(R[(h * Wf + k) * PL + pl]);
          v[h] = mk(t.x, t.y);
        }
      }
      lane_dft<N>(v);
      if (back == 0) {
#pragma unroll
        for (int kh = 0; kh < N; ++kh) {
          const float4 g = gs[kh * Wf + k];          // {exp(-D), (D+1e-8)B, C/(HW), 1e-7(D+1e-8)}
          const float gy = g.y * (float)N;           // undoes the row pass's 1/N
          float ur = gy * v[kh].x, ui = gy * v[kh].y;
          if (ur * ur + ui * ui < g.w * g.w) { ur = g.w; ui = 0.f; }
          v[kh] = mk(g.z * ui, g.z * ur);
        }
      }
    }
#pragma unroll
    for (int h = 0; h < N; ++h) R[(h * Wf + k) * PL + pl] = __floats2half2_rn(v[h].y, v[h].x);
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();                      // z tile complete; columns of all threads visible

  // ---- inverse rows (C2R: imaginary parts of the DC and Nyquist bins are ignored), * z ----
#pragma unroll 1
  for (int h = part; h < RP; h += TPP) {
    const bool two = h + RP < N;
    cf z[N];
#pragma unroll
    for (int k = 0; k < Wf; ++k) {
      const float2 a = __half22float2(R[(h * Wf + k) * PL + pl]);
      float2 b = make_float2(0.f, 0.f);
      if (two) b = __half22float2(R[((h + RP) * Wf + k) * PL + pl]);
      // Z[k] = A[k] + i B[k], Z[N - k] = conj A[k] + i conj B[k], parts exchanged
      if (k == 0 || 2 * k == N) z[k] = mk(b.x, a.x);
      else { z[k] = mk(a.y + b.x, a.x - b.y); z[N - k] = mk(b.x - a.y, a.x + b.y); }
    }
    lane_dft<N>(z);
#pragma unroll
    for (int w = 0; w < N; ++w) {
      const int i = (h * N + w) * PL + pl, j = i + RP * N * PL;
      tile[i] = __float2bfloat16(z[w].y * __bfloat162float(tile[i]));
      if (two) tile[j] = __float2bfloat16(z[w].x * __bfloat162float(tile[j]));
    }
  }
  __syncthreads();
  __nv_bfloat16* yo = y + (size_t)n * P * ldy + c0;
  for (int q = tid; q < P * V; q += TPB) {
    const int p = q / V, j = q % V;
    *reinterpret_cast<uint4*>(yo + (size_t)p * ldy + j * 8) =
        *reinterpret_cast<const uint4*>(tile + p * PL + j * 8);
  }
}

bool spectral_cl_supported(int H, int W, int C, int T) {
  return T == 1 && H == W && (H == 14 || H == 7) && C % SCL_PL == 0;
}

template <int N, int PL, int TPP>
static int spectral_cl_launch(const __nv_bfloat16* xz, int ld, int Nimg, int C, const float* gates, __nv_bfloat16* y, int ldy, cudaStream_t st) {
  constexpr int NB = N * (N / 2 + 1);
  constexpr size_t smem = (size_t)NB * PL * 4 + (size_t)N * N * PL * 2 + (size_t)NB * 16;
  auto kern = gated_spectral_cl_kernel<N, PL, TPP>;
  const cudaError_t e = func_smem(kern, smem);
  if (e != cudaSuccess) { set_cuda_error(e); return CSSM_ERR_CUDA; }
  launch_k(kern, Nimg * (C / PL), PL * TPP, smem, st, xz, ld, C, reinterpret_cast<const float4*>(gates), y, ldy);
  return check_launch();
}

// xz: (Nimg, H*W, ld) bf16 with x_main in columns [0, C) and silu(z) in [C, 2C); gates: the
// (Nimg, H*Wf) float4 maps of launch_gated_gates in row-major bin order; y: (Nimg, H*W, ldy).
int launch_gated_spectral_cl(const __nv_bfloat16* xz, int ld, int Nimg, int H, int W, int C,
                             const float* gates, __nv_bfloat16* y, int ldy, cudaStream_t st) {
  if (!spectral_cl_supported(H, W, C, 1) || ld % 8 != 0 || ldy % 8 != 0) return CSSM_ERR_UNSUPPORTED;
  // Up to two CTAs of 64 planes an SM the smaller ones are ahead (32 images 500 -> 493 us a pass, 64 701 -> 699), above it not (96: 891, 891).
  const bool few = (long long)Nimg * (C / SCL_PL) < 2LL * sm_count();
  if (H == 14) return few ? spectral_cl_launch<14, 16, 8>(xz, ld, Nimg, C, gates, y, ldy, st) : spectral_cl_launch<14, SCL_PL, 2>(xz, ld, Nimg, C, gates, y, ldy, st);
  return few ? spectral_cl_launch<7, 16, 4>(xz, ld, Nimg, C, gates, y, ldy, st) : spectral_cl_launch<7, SCL_PL, 2>(xz, ld, Nimg, C, gates, y, ldy, st);
}

}  // namespace cssm
