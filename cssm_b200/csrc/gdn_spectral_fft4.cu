// GDN on square planes with whole FFTs in a lane's registers, key dimension 4 (csrc/gdn_spectral_fft.cuh)
#define CSSM_F32X2 0
#include "gdn_spectral_fft.cuh"

namespace cssm {
int launch_gdn_spectral_fft4(const GdnSpectralArgs& a, cudaStream_t st) { return launch_gdn_fft_dk<4>(a, st); }
}  // namespace cssm
