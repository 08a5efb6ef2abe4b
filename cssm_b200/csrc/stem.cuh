// Stem layer arguments and helpers shared by csrc/simple_model.cu and csrc/stem_tc.cu.
#pragma once
#include "common.cuh"

namespace cssm {

__device__ __forceinline__ float softplus_f(float a) {
  return fmaxf(a, 0.f) + log_ftz(1.0f + exp_ftz(-fabsf(a)));
}

struct StemArgs {
  const float* x; float* out;           // (N,Hin,Win,Cin) -> (N,Ho,Wo,C), channels-last
  const float* wk; const float* bk;     // (KS,KS,Cin,C), (C)
  const float* scale; const float* bias;
  int N, Hin, Win, Cin, C, Ho, Wo;
  int w_in_smem;                        // conv kernel staged in shared memory
};

// 3x3 pooled layers of C to C channels, C = 32 or 64, on the tensor cores; `scratch` holds the weights as
// launch_stem_split_weights leaves them (16-byte aligned)
size_t stem_tc_scratch_bytes(int C);
bool stem_tc_supported(const StemArgs& a);
int launch_stem_split_weights(const float* wk, void* scratch, int C, cudaStream_t st);
int launch_stem_layer_tc(const StemArgs& a, const void* scratch, cudaStream_t st);
int read_stem_error(int* out, int clear);

}  // namespace cssm
