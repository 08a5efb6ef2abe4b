// Shared helpers for the cssm_b200 CUDA sources (sm_100a).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <stddef.h>
#include "../../include/cssm_b200.h"

#ifndef CSSM_F32X2
#define CSSM_F32X2 1
#endif

namespace cssm {

struct __align__(8) cf {
  float x, y;
};

__device__ __forceinline__ cf mk(float x, float y) { cf r; r.x = x; r.y = y; return r; }
// Complex add / subtract as one packed fp32x2 instruction (sm_100): halves the issue slots of
// the FFT butterflies, which are mostly complex additions.
__device__ __forceinline__ cf operator+(cf a, cf b) {
#if CSSM_F32X2
  unsigned long long pa, pb, pr;
  asm("mov.b64 %0, {%1, %2};" : "=l"(pa) : "f"(a.x), "f"(a.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(pb) : "f"(b.x), "f"(b.y));
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(pr) : "l"(pa), "l"(pb));
  cf r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(pr));
  return r;
#else
  return mk(a.x + b.x, a.y + b.y);
#endif
}
__device__ __forceinline__ cf operator-(cf a, cf b) {
#if CSSM_F32X2
  unsigned long long pa, pb, pr;
  asm("mov.b64 %0, {%1, %2};" : "=l"(pa) : "f"(a.x), "f"(a.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(pb) : "f"(b.x), "f"(b.y));
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(pr) : "l"(pa), "l"(pb));
  cf r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(pr));
  return r;
#else
  return mk(a.x - b.x, a.y - b.y);
#endif
}
__device__ __forceinline__ cf cmul(cf a, cf b) {
  return mk(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// a * conj(b)
__device__ __forceinline__ cf cmulc(cf a, cf b) {
  return mk(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}
// SiLU / sigmoid through an approximate reciprocal (rcp.approx: within 1 ulp, far inside the block's 1e-4 tolerance) instead of an
// IEEE division, which measured several times as long over activations with many zeros.
__device__ __forceinline__ float rcp_fast(float d) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
  return r;
}
// e^v and log v without the scaling of subnormal results and arguments that the intrinsics wrap around the same instructions (three more
// each): for sums 1 + e^v, which subnormals do not change, and logarithms of at least 1.
__device__ __forceinline__ float exp_ftz(float v) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v * 1.44269504088896340736f));
  return r;
}
__device__ __forceinline__ float log_ftz(float v) {
  float r;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r * 0.69314718055994530942f;
}
__device__ __forceinline__ float silu_f(float v) { return v * rcp_fast(1.0f + exp_ftz(-v)); }
__device__ __forceinline__ float sigmoid_f(float v) { return rcp_fast(1.0f + exp_ftz(-v)); }

// n / d for 0 <= n < 2^31 by one multiply-high with d's rounded-up reciprocal, 2^l >= d (division by invariant integers,
// Granlund and Montgomery 1994).
struct FastDiv {
  uint32_t mul, shift, one;
  FastDiv() = default;
  explicit FastDiv(int d) {
    shift = 0;
    while ((1u << shift) < (uint32_t)d) ++shift;
    mul = (uint32_t)((((uint64_t)1 << 32) * (((uint64_t)1 << shift) - (uint64_t)d)) / (uint64_t)d + 1);
    one = d == 1 ? 1 : 0;
  }
  __device__ __forceinline__ int div(int n) const {
    return one ? n : (int)((__umulhi((uint32_t)n, mul) + (uint32_t)n) >> shift);
  }
};

// ---- launches ----
// Programmatic dependent launch: inside a PdlScope every kernel but the first is launched so that its
// CTAs may become resident while the one before still runs.  Each kernel waits (pdl_wait) before it
// touches anything an earlier kernel writes or reads, and only then lets the next one start
// (pdl_trigger), so at most two kernels of a chain overlap and what a kernel does ahead of its wait
// (barriers, TMEM, tables, weights) may rely on everything before the chain's first kernel.
// It pays where launches are short (CSSM-SHViT, one image: 630 -> 487 us); with activations of 1 GB, launches of
// 0.5 ms and more, passes got 3 % slower, so the block drivers turn it on up to PDL_MAX_BYTES a tensor.  The classifiers
// keep it on at every size, for the mixer blocks in them too: it wins throughout (2 images 362 against 466 us without, 64
// 821 / 941, 512 4054 / 4118, 768 5885 / 5925).  Exceptions within a scope: PdlOff, spread_smem.
int sm_count();                           // of the current device
extern thread_local int g_pdl;            // 0 off, 1 first launch of a scope pending, 2 on
constexpr size_t PDL_MAX_BYTES = (size_t)256 << 20;
struct PdlScope {
  int prev;
  explicit PdlScope(bool on) : prev(g_pdl) { if (g_pdl == 0 && on) g_pdl = 1; }
  ~PdlScope() { g_pdl = prev; }
};
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_sync() { pdl_wait(); pdl_trigger(); }

// A launch that waits for everything before it, also inside a scope, for persistent kernels of many rounds: in an overlapped
// launch the CTAs take SMs in the order in which those come free, so neighbours in the grid, which work on neighbouring
// tiles, sit far apart, and the CTAs that have a round more than others end up two on an SM (24 DeltaNet clips of 8 frames of
// 28x28x64: the pass 451 us, 429 so; 10 of 40x40x64: 463, 447).
struct PdlOff {
  int prev;
  explicit PdlOff(bool off) : prev(g_pdl) { if (off && g_pdl == 2) g_pdl = 1; }
  ~PdlOff() { if (prev == 2) g_pdl = 2; }
};

// Whether the CTAs that take one group more than others, `groups` dealt out to `occ` CTAs on every SM, would share SMs
// with one another in an overlapped launch where they need not.
inline bool uneven_rounds(long long groups, int occ) {
  const long long sms = sm_count(), rest = groups % (sms * occ);
  return groups > sms * occ && rest > 0 && (rest + sms - 1) / sms < occ;
}

template <class... P, class... A>
inline void launch_k(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = st;
  cfg.attrs = at; cfg.numAttrs = g_pdl == 2 ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);     // errors are read by check_launch
  if (g_pdl == 1) g_pdl = 2;
}
// cudaFuncAttributeMaxDynamicSharedMemorySize of the current device is at least `bytes` from here on: it only ever
// rises (smem_limit.h)
cudaError_t func_smem_set(const void* kern, size_t bytes);
template <class F> inline cudaError_t func_smem(F* kern, size_t bytes) {
  return func_smem_set(reinterpret_cast<const void*>(kern), bytes);
}
// Shared memory to ask for where a kernel of `ctas` long CTAs (a recurrence over T) needs `smem`: in an overlapped
// launch at least as much as keeps a CTA more than the even share off an SM.  Launched early such a kernel finds the
// CTAs of the one before on most SMs and goes two or four at a time to the few with room, where it then stays for its whole run
// while others are idle.  Block by block (packed, so): GDN 4 x 4 x 48 x 48 x 32 (32 CTAs) 1541, 942 us; gated 4 x 8 x
// 60 x 60 x 32 226, 170; gated SimpleCSSM, 7 clips of 16 frames (112 CTAs) 216, 172.
inline size_t spread_smem(size_t smem, long long ctas) {
  constexpr size_t SM_BYTES = 228 * 1024, CTA_BYTES = 1024;         // of an SM; reserved by each CTA
  const size_t share = (size_t)((ctas + sm_count() - 1) / sm_count());
  if (g_pdl != 2 || share > 8) return smem;
  const size_t least = SM_BYTES / (share + 1) - CTA_BYTES + 128;
  return smem > least ? smem : least;
}

// Host-side record of the last CUDA error seen on this thread.
void set_cuda_error(cudaError_t e);
int check_launch();

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
inline size_t round_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

// ---- plan layouts (device memory prepared by *_plan_init) ----
struct GatedPlan {
  size_t khat;     // cf [C][H*Wf] in the bin order of the spectral kernel in use
  size_t rope_t;   // float2 [T][C/2]  (cos, sin)
  size_t rope_h;   // float2 [H][C/2]
  size_t rope_w;   // float2 [W][C/2]
  size_t rope_nz;  // float  [C/2]  1 = pair rotated on some axis, 0 = angle identically zero
  size_t total;
};
GatedPlan gated_plan_layout(const cssm_gated_desc& d);

// Which spectral kernel handles an (H, W) plane.
enum SpectralPath { PATH_GENERIC = 0, PATH_R64 = 1, PATH_R32 = 2 };
SpectralPath spectral_path(int H, int W);

// Position of frequency bin (kh, kw) inside a per-(b,t) gate map / per-channel K_hat.
__host__ __device__ inline int bin_index(int path, int kh, int kw, int H, int Wf) {
  if (path == PATH_R64) return (((kh >> 3) * 33 + kw) << 3) + (kh & 7);
  if (path == PATH_R32) return ((((((kh >> 2) & 1) << 2) | (kh >> 3)) * 17 + kw) << 2) + (kh & 3);
  return kh * Wf + kw;
}

}  // namespace cssm

// Caller-owned state of the streaming host entry points (cssm_host_pipe_create / _destroy; the type
// is opaque in the public header): one copy stream, its events, and which host buffer was prefetched
// into which of the two input buffers of which workspace.
struct cssm_host_pipe {
  cudaStream_t copy;
  cudaEvent_t copied[2];       // the copy into input buffer j has finished
  cudaEvent_t computed;        // orders a cold copy behind the work already queued on the caller's stream
  const void* src;             // host address whose batch sits (or is arriving) in buffer `buf`
  const void* ws;              // ... of this workspace
  int buf;
};

namespace cssm {
// First half of a streaming host call: makes `stream` wait for the batch x_host in input buffer
// *j of the workspace (already prefetched by the previous call on this pipe, or copied now), and
// starts the copy of x_next_host (may be null) into the other buffer on the pipe's stream.
inline int host_pipe_stage(cssm_host_pipe* p, void* workspace, char* xbuf0, char* xbuf1, size_t xbytes,
                           const void* x_host, const void* x_next_host, cudaStream_t st, int* j_out) {
  cudaError_t e = cudaSuccess;
  char* xb[2] = {xbuf0, xbuf1};
  int j;
  if (p->src == x_host && p->ws == workspace) {
    j = p->buf;                                        // prefetched by the previous call
  } else {
    j = 0;
    // after whatever the caller queued on its stream, and after any copy still running on the pipe
    e = cudaEventRecord(p->computed, st);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(p->copy, p->computed, 0);
    if (e == cudaSuccess) e = cudaMemcpyAsync(xb[0], x_host, xbytes, cudaMemcpyHostToDevice, p->copy);
    if (e == cudaSuccess) e = cudaEventRecord(p->copied[0], p->copy);
  }
  p->src = nullptr;
  if (x_next_host != nullptr && e == cudaSuccess) {
    // buffer 1 - j was last read by the previous call's forward, which that call waited for
    e = cudaMemcpyAsync(xb[1 - j], x_next_host, xbytes, cudaMemcpyHostToDevice, p->copy);
    if (e == cudaSuccess) e = cudaEventRecord(p->copied[1 - j], p->copy);
    if (e == cudaSuccess) { p->src = x_next_host; p->ws = workspace; p->buf = 1 - j; }
  }
  if (e == cudaSuccess) e = cudaStreamWaitEvent(st, p->copied[j], 0);
  *j_out = j;
  if (e != cudaSuccess) { set_cuda_error(e); return CSSM_ERR_CUDA; }
  return CSSM_OK;
}
// Error path of a streaming host call: leave no copy running into a workspace the caller may free.
inline void host_pipe_abort(cssm_host_pipe* p) {
  cudaStreamSynchronize(p->copy);
  p->src = nullptr;
}
}  // namespace cssm
