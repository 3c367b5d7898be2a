// The runtime-planned smooth-length passes (fft_rt.cuh) in FP32.
#include "fft_rt.cuh"

namespace gbfft {
cudaError_t launch_rt_f32(int kind, bool contiguous, const PassArgs& a, cudaStream_t s) {
  return rt::launch<rt::F32>(kind, contiguous, a, s);
}
}  // namespace gbfft
