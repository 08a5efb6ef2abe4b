// Arguments of the float32 1x1 channel projections (csrc/gemm_tc.cu, csrc/gemm_split.cu), with the layout changes and
// pointwise work of the blocks fused into their load and store:
//   A side: channels-last rows (optionally rotated by RoPE on load), or planar planes
//           (optionally RMS-normalised over channels, scaled and gated on load);
//   C side: channels-last rows, or planar planes (optionally through SiLU / sigmoid).
// out[m, n] = sum_k A[m, k] * Wk[k, n] + bias[n],  m = frame*HW + pixel.
#pragma once
#include "common.cuh"

namespace cssm {

struct GemmArgs {
  int M, N, K, HW;
  const float* A;         // channels-last: (M, K).  planar: plane (frame*a_planes + a_plane0 + k)
  int a_planes, a_plane0;
  // source frame of output frame f, both A layouts: (f / a_fdiv) * a_fmul + a_fadd, where
  // a_fdiv <= 1 means no division and a_fmul == a_fadd == 0 means the identity.
  //   last frame of every clip : a_fmul = T, a_fadd = T-1  (output frames = clips)
  //   one frame repeated over T: a_fdiv = T, a_fmul = 1    (output frames = (clip, t))
  int a_fdiv, a_fmul, a_fadd;
  int rope_tlast;         // 1: every output frame is rotated as t = T-1; 0: t = output frame % T
  const float* Wk;        // (K, N) row-major
  const void* wsplit;       // Wk as launch_split_weights left it, or nullptr (gemm_split only; no RMS prologue)
  const float* bias;      // (N) or nullptr
  float* out;             // channels-last (M, N) or planar plane (frame*o_planes + o_plane0 + n)
  int o_planes, o_plane0;
  // RoPE on a channels-last A (nullptr = off): float2 (cos, sin) tables
  const float2* rope_t; const float2* rope_h; const float2* rope_w;
  const float* rope_nz;     // (K/2) 1 = pair is rotated, 0 = identity (may be nullptr: rotate all)
  int T, H, W;
  // planar-A prologue of the GDN output: a <- a * rsqrt(mean_k a^2 + eps) * scale[k] * gate
  const float* rms_scale;   // (K) or nullptr (no normalisation)
  const float* gate;        // planar, plane (frame*g_planes + g_plane0 + k), or nullptr
  int g_planes, g_plane0;
  int g_compact;            // 1: the gate is indexed by the OUTPUT frame, 0: by the source frame
  int out_act;              // 0 none, 1 silu, 2 sigmoid; applied to output columns n >= act_n0
  int act_n0;
  // planar output, gemm_tc only: columns n < mul_n multiply plane (frame*mul_planes + mul_plane0 + n) of mul in place and are not stored
  float* mul; int mul_planes, mul_plane0, mul_n;
  int z_last_only;          // planar output: columns n >= act_n0 are only stored for frames with t == T-1
  const float* sub;         // channels-last output only: (M, N) tensor subtracted from the result, or nullptr
};

// Two tf32 parts (three bf16 ones under the RMS prologue), K = 64 only; three bf16 parts, any size.
bool gemm_tc_supported(const GemmArgs& g, bool a_planar);
// whether gemm_tc takes a channels-last (M, K) by (K, N) projection of frames of HW pixels that multiplies planes in place (mul)
bool gemm_tc_in_place(int K, int N, int HW, int mul_n);
int launch_gemm_tc(const GemmArgs& g, bool a_planar, cudaStream_t st);
int launch_gemm_split(const GemmArgs& g, bool a_planar, cudaStream_t st);
// The weights of up to two projections (K, N0), (K, N1) split once for all CTAs of their launches, in the layout of an operand
// block; split_weights_bytes(K, N) each, 16-byte aligned.  0 bytes: K so short that every CTA keeps its share of the weights anyway.
size_t split_weights_bytes(int K, int N);
int launch_split_weights(int K, const float* w0, int N0, void* out0, const float* w1, int N1, void* out1, cudaStream_t st);
int read_tc_error(int* out, int clear);
int read_split_error(int* out, int clear);

template <bool A_PLANAR, bool O_PLANAR>
inline int launch_gemm(const GemmArgs& g, cudaStream_t st) {
  static_assert(A_PLANAR != O_PLANAR, "projections change layout");
  if (gemm_tc_supported(g, A_PLANAR)) return launch_gemm_tc(g, A_PLANAR, st);
  return launch_gemm_split(g, A_PLANAR, st);
}

}  // namespace cssm
