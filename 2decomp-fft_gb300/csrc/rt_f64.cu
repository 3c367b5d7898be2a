// The runtime-planned smooth-length passes (fft_rt.cuh) in fixed point (FP64).
#include "fft_rt.cuh"

namespace gbfft {
cudaError_t launch_rt_f64(int kind, bool contiguous, const PassArgs& a, cudaStream_t s) {
  return rt::launch<rt::Fixed>(kind, contiguous, a, s);
}
}  // namespace gbfft
