// GDN on square planes with whole FFTs in a lane's registers, key dimension 2 (csrc/gdn_spectral_fft.cuh)
#define CSSM_F32X2 0
#include "gdn_spectral_fft.cuh"

namespace cssm {
int launch_gdn_spectral_fft2(const GdnSpectralArgs& a, cudaStream_t st) { return launch_gdn_fft_dk<2>(a, st); }
}  // namespace cssm
