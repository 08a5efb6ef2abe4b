// GDN fused spectral kernel for 64x64 planes, d_k = d_v = 4 (static images: csrc/gdn_spectral_r64.cu): persistent CTAs of eight warps,
// one per SM, that take the steps of one (batch, head) after another.  A step has two parts with a barrier after each:
//   transforms  sixteen planes, two a warp (csrc/fft64.cuh: whole 64-point FFTs in a lane's registers), each in place in its region of
//               shared memory: TMA brings it, the row spectra and then the half-spectrum go over it.  Warps 0-3 transform an output
//               plane of the step before back (TMA store over the v plane in global memory, and v of this step into its region) and
//               then a k plane, warps 4-7 a q plane and then v;
//   bins        all threads: a lane owns eight or nine of the 2112 frequency bins, normalises k and q as it reads them and updates
//               all four rows of a bin's 4x4 state (packed f32x2 over pairs of rows), which streams through L2 a bin ahead, 16 bytes
//               a lane and access (270 KB a head: more than the registers or what the planes leave of shared memory); the
//               readout's spectrum replaces v's.
// So a plane crosses shared memory five times (in, rows out, columns in and out, bins) and no FFT exchanges anything.
// (Two warps a scheduler at 255 registers; twelve at 168, one a plane, spill, and the inverse and v one after another are the longest chain:
// 3174 against 2353 us, same bins.)
// Bound: the transforms (1.13 ms of 2.13) issue 59 % of the time, the bins 39 %: dependent packed multiply-adds of two warps, instruction
// fetch, state reads.  128 x 8 x 64 x 64 x 64: 3764 (FFTs shared by eight lanes, shared-memory pipe 80 % busy) -> 2130 us; one head, T = 1
// 36 -> 27; 10 x 64 channels, T = 1 66 -> 43; 2 x 16 clips 522 -> 295; last frame only, 64 x 8 1389 -> 797.
// Every wait is bounded; on expiry the kernel records an error code (cssm_device_error) and winds down.

// Complex adds as scalar pairs: a lane's FFT is all register renaming then (packed 2418 against 2353 us, before the bins' last form).
#define CSSM_F32X2 0
#include <cuda.h>
#include <string.h>
#include "fft64.cuh"
#include "kernels.cuh"
#include "bf16_ops.cuh"
#include "gdn_common.cuh"
#include "tc05.cuh"

namespace cssm {

__device__ int g_p64_error = 0;

constexpr int GQ_THREADS = 8 * 32;
constexpr uint32_t GQ_REGION = P64_PLANE_CF * 8u;                          // one plane: raw, row spectra or half-spectrum
constexpr uint32_t GQ_NRM_OFF = 12u * GQ_REGION;
constexpr uint32_t GQ_SMEM = GQ_NRM_OFF + 32u + 128u;                       // (+ alignment)
static_assert(GQ_REGION % 128 == 0 && P64_RAW <= GQ_REGION && GQ_SMEM + 1024 <= 227 * 1024, "one CTA per SM");

// The regions, 128-byte aligned as TMA wants them; behind them half the scales of the q and k planes.
__device__ __forceinline__ unsigned char* p64_smem() {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  return smem_raw + ((128u - (tc::smem_u32(smem_raw) & 127u)) & 127u);
}

// One step of all bins.  A call, so that its registers and those of the transforms are allocated apart (inlined, 280 bytes of spills a
// thread, which miss L1 beside this much shared memory).
__device__ __noinline__ void p64_bins(const float2* ab, const float2* wh, ulonglong2* S, bool first, bool last, bool emit) {
  typedef unsigned long long u64;
  constexpr int NB = 64 * 33;
  cf* base = reinterpret_cast<cf*>(p64_smem());
  const float4* nrm = reinterpret_cast<const float4*>(p64_smem() + GQ_NRM_OFF);
  ulonglong2 st[2][8];
  float2 gw[2][2];
  auto fetch = [&](int r, int w) {
    const int i = threadIdx.x + r * GQ_THREADS;
    if (i >= NB) return;
    gw[w][0] = __ldg(ab + i);
    gw[w][1] = __ldg(wh + i);
#pragma unroll
    for (int c = 0; c < 8; ++c) st[w][c] = make_ulonglong2(0ull, 0ull);
    if (!first) {
#pragma unroll
      for (int c = 0; c < 8; ++c) st[w][c] = __ldcg(S + c * NB + i);
    }
  };
  auto bin = [&](int r, int w) {
    const int i = threadIdx.x + r * GQ_THREADS;
    if (i >= NB) return;
    const int si = p64_slot(i);
    u64 Sx[2][4], Sy[2][4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      Sx[0][c] = st[w][c].x; Sx[1][c] = st[w][c].y;
      Sy[0][c] = st[w][4 + c].x; Sy[1][c] = st[w][4 + c].y;
    }
    const float4 nk = nrm[1];
    const float nkv[4] = {nk.x, nk.y, nk.z, nk.w};
    cf kk[4], v[4];
    float ks = 0.f;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const cf k = base[(4 + c) * P64_PLANE_CF + si];
      v[c] = base[(8 + c) * P64_PLANE_CF + si];
      kk[c] = mk(k.x * nkv[c], k.y * nkv[c]);
      ks += kk[c].x * kk[c].x + kk[c].y * kk[c].y;
    }
    const float kn = rsqrtf(ks + 1e-6f);
#pragma unroll
    for (int c = 0; c < 4; ++c) kk[c] = mk(kk[c].x * kn, kk[c].y * kn);
    const float beta = gw[w][0].y, bv = 0.5f * beta;                       // v is doubled
#pragma unroll
    for (int c = 0; c < 4; ++c) v[c] = mk(bv * v[c].x, bv * v[c].y);
    const cf aw = mk(gw[w][0].x * gw[w][1].x, gw[w][0].x * gw[w][1].y);
    gdn_rows_update(Sx, Sy, kk, v, aw, beta);
    if (!last) {
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        __stcg(S + c * NB + i, make_ulonglong2(Sx[0][c], Sx[1][c]));
        __stcg(S + (4 + c) * NB + i, make_ulonglong2(Sy[0][c], Sy[1][c]));
      }
    }
    if (emit) {
      const float4 nq = nrm[0];
      const float nqv[4] = {nq.x, nq.y, nq.z, nq.w};
      cf qq[4], o[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const cf q = base[c * P64_PLANE_CF + si];
        const float sc = nqv[c] * (1.0f / 4096.0f);
        qq[c] = mk(q.x * sc, q.y * sc);
      }
      gdn_rows_read(Sx, Sy, qq, o);
#pragma unroll
      for (int c = 0; c < 4; ++c) base[(8 + c) * P64_PLANE_CF + si] = o[c];
    }
  };
  // One copy of the body and register moves: two copies are more than the instruction caches like (2398 against 2150 us); the state
  // two bins ahead is no faster (2364 against 2352).
  fetch(0, 0);
#pragma unroll 1
  for (int r = 0; r * GQ_THREADS < NB; ++r) {
    fetch(r + 1, 1);
    bin(r, 0);
#pragma unroll
    for (int c = 0; c < 8; ++c) st[0][c] = st[1][c];
    gw[0][0] = gw[1][0]; gw[0][1] = gw[1][1];
  }
}

// LAST: only the last step's output planes are produced: the q planes, the readout and the inverse of earlier steps are skipped.
template <bool LAST>
__global__ void __launch_bounds__(GQ_THREADS, 1) gdn_spectral_p64(const GdnSpectralArgs a, const __grid_constant__ CUtensorMap map) {
  unsigned char* smem = p64_smem();
  float* nrm = reinterpret_cast<float*>(smem + GQ_NRM_OFF);
  __shared__ __align__(8) uint64_t raw_full[12];
  __shared__ int s_bad;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr int DK = 4, NB = 64 * 33;
  const int nh = a.C / DK, heads = a.B * nh, T = a.T;
  if (tid == 0) {
    for (int i = 0; i < 12; ++i) tc::mbar_init(&raw_full[i], 1);
    tc::fence_mbar_init();
    s_bad = 0;
  }
  __syncthreads();
  pdl_sync();
  const int steps = (heads - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x * T;
  // first row pair of plane p (q 0-3, k 4-7, v 8-11) in step s
  auto plane_row = [&](int p, int s) {
    const int hi = s / T, t = s - hi * T, head = blockIdx.x + hi * gridDim.x, b = head / nh, hd = head - b * nh;
    return ((b * T + t) * 3 * a.C + (p >> 2) * a.C + hd * DK + (p & 3)) * 32;
  };
  auto load = [&](int p, int s) {
    tc::mbar_expect_tx(&raw_full[p], P64_RAW);
    tc::tma_load_2d(smem + p * GQ_REGION, &map, 0, plane_row(p, s), &raw_full[p]);
  };
  for (int s = 0; s <= steps; ++s) {
    const int hi = s / T, t = s - hi * T;
    const bool emit = !LAST || t == T - 1, emitted = s > 0 && (!LAST || t == 0);       // this step, the one before: the same for all
    if (lane == 0 && s < steps) {
      if (warp < 4) load(4 + warp, s);
      else {
        if (emit) load(warp - 4, s);
        tc::tma_prefetch_2d(&map, 0, plane_row(warp + 4, s));
      }
    }
    __syncwarp();
    // one copy of the FFT's code for all passes: forward rows and columns, or inverse columns and rows with real and imaginary parts
    // exchanged before and after
#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
      const bool fwd = warp >= 4 || half == 1;
      const int p = warp < 4 ? (half ? 4 + warp : 8 + warp) : (half ? 4 + warp : warp - 4);
      unsigned char* own = smem + p * GQ_REGION;
      cf* sp = reinterpret_cast<cf*>(own);
      if (fwd ? s < steps && (p >= 4 || emit) : emitted) {
        cf z[64];
        if (fwd) {
          const int n = LAST && p < 4 ? hi : s;                            // copies into this region before
          if (__any_sync(0xffffffffu, !tc::mbar_wait_spin(&raw_full[p], n & 1)) && lane == 0) { atomicExch(&g_p64_error, 1); s_bad = 1; }
          p64_load_rows(own, lane, z);
        } else {
          p64_pack_columns(sp, lane);
          __syncwarp();
          p64_get_columns_swapped(sp, lane, z);
        }
#pragma unroll 1
        for (int pass = 0; pass < 2; ++pass) {
          fft64_lane(z);
          __syncwarp();                                                    // every lane has read what is written now
          if (pass == 0) {
            if (fwd) {
              p64_put_rows(sp, lane, z);
              __syncwarp();
#pragma unroll
              for (int h = 0; h < 64; ++h) z[h] = sp[p64_row(h) * P64_PITCH + lane];
            } else {
#pragma unroll
              for (int h = 0; h < 64; ++h) sp[p64_row(h) * P64_PITCH + lane] = mk(z[h].y, z[h].x);
              __syncwarp();
              p64_get_rows_swapped(sp, lane, z);
            }
          } else if (fwd) {
            if (p < 8) {
              float e0 = 0.f, e1 = 0.f;
#pragma unroll
              for (int k = 0; k < 64; ++k) { e0 = fmaf(z[k].x, z[k].x, e0); e1 = fmaf(z[k].y, z[k].y, e1); }
              float e = (e0 + e1) * (lane == 0 ? 1.f : 0.25f);             // (the packed column is not doubled)
#pragma unroll
              for (int o = 16; o; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
              if (lane == 0) nrm[p] = a.use_l2 ? 0.5f * rsqrtf(e + 1e-6f) : 0.5f;
            }
            p64_put_columns(sp, lane, z);
            __syncwarp();
            p64_unpack_columns(sp, lane);
          } else {
            p64_store_rows_swapped(own, lane, z);
            tc::fence_proxy_async();
            __syncwarp();
            if (lane == 0) {
              tc::tma_store_2d(&map, own, 0, plane_row(p, s - 1));
              asm volatile("cp.async.bulk.commit_group;" ::: "memory");
              asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            }
          }
        }
      }
      if (!fwd && lane == 0 && s < steps) load(p, s);                      // v, for warp + 4
      __syncwarp();
    }
    if (s == steps) break;
    __syncthreads();
    if (s_bad) break;                                                      // the same for all: nobody waits before the next barrier
    const int head = blockIdx.x + hi * gridDim.x, b = head / nh, hd = head - b * nh;
    p64_bins(a.ab + ((size_t)(b * T + t) * a.ab_heads + (a.ab_heads > 1 ? hd : 0)) * NB, reinterpret_cast<const float2*>(a.what) + (size_t)hd * NB,
             reinterpret_cast<ulonglong2*>(a.state) + (size_t)blockIdx.x * 8 * NB, t == 0, t + 1 == T, emit);
    tc::fence_proxy_async();                                               // these accesses come before the copies into the regions
    __syncthreads();
  }
  if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  // error path only: copies that may still be in flight get a bounded time (~1 ms) to land
  if (s_bad)
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
}

// Row pairs of 128 floats; a box of 132 leaves the pairs of a plane 528 bytes apart (the four columns past the end are outside the
// map: zeros on the way in, skipped on the way out).
static bool pair_map(CUtensorMap* map, float* base, uint64_t pairs) {
  const tc::EncodeTiledFn enc = tc::encode_fn();
  if (!enc) return false;
  const cuuint64_t dims[2] = {128, pairs}, strides[1] = {512};
  const cuuint32_t box[2] = {132, 32}, es[2] = {1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, base, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int launch_gdn_spectral_p64(const GdnSpectralArgs& a, cudaStream_t st) {
  if (a.static_image || a.dk != 4 || a.H != 64 || a.W != 64) return CSSM_ERR_UNSUPPORTED;
  const long long pairs = (long long)a.B * a.T * 3 * a.C * 32;
  if (pairs >= (1LL << 31)) return CSSM_ERR_UNSUPPORTED;
  CUtensorMap map;
  memset(&map, 0, sizeof(map));
  if (!pair_map(&map, a.qkv, (uint64_t)pairs)) return CSSM_ERR_CUDA;
  auto kern = a.last_only ? gdn_spectral_p64<true> : gdn_spectral_p64<false>;
  const cudaError_t e = func_smem(kern, GQ_SMEM);
  if (e != cudaSuccess) { set_cuda_error(e); return CSSM_ERR_CUDA; }
  const int heads = a.B * (a.C / 4), sms = sm_count();
  launch_k(kern, heads < sms ? heads : sms, GQ_THREADS, (size_t)GQ_SMEM, st, a, map);
  return check_launch();
}

int read_p64_error(int* out, int clear) {
  cudaError_t e = cudaMemcpyFromSymbol(out, g_p64_error, sizeof(int));
  if (e == cudaSuccess && clear && *out != 0) {
    const int zero = 0;
    e = cudaMemcpyToSymbol(g_p64_error, &zero, sizeof(int));
  }
  if (e != cudaSuccess) { set_cuda_error(e); return CSSM_ERR_CUDA; }
  return CSSM_OK;
}

}  // namespace cssm
