// Instantiations of the two-stage FP32 passes (fft_mixed.cuh).  The build
// compiles this file once for every part -- a second radix and a line kind
// (GBFFT_MIXED_R1, GBFFT_MIXED_KIND) -- and once without, for the dispatch.
#ifdef GBFFT_MIXED_R1
#include "fft_mixed.cuh"

namespace gbfft {

namespace {
template <int R0>
cudaError_t launch_r0(bool contiguous, const PassArgs& a, cudaStream_t s) {
  constexpr int R1 = GBFFT_MIXED_R1, kKind = GBFFT_MIXED_KIND, N = R0 * R1;
  if constexpr (mixed_length(N) && mixed_r0(N) == R0)
    if (a.n == N)
      return contiguous ? mixed::launch_n<kKind, true, N>(a, s) : mixed::launch_n<kKind, false, N>(a, s);
  if constexpr (R0 < R1) return launch_r0<R0 + 1>(contiguous, a, s);
  return cudaErrorNotSupported;
}
}  // namespace

template <>
cudaError_t launch_mixed_part<GBFFT_MIXED_R1, GBFFT_MIXED_KIND>(bool contiguous, const PassArgs& a, cudaStream_t s) {
  return launch_r0<2>(contiguous, a, s);
}

}  // namespace gbfft
#else
#include "gbfft_internal.h"

namespace gbfft {

#define GBFFT_MIXED_DECL(r)                                                                  \
  template <> cudaError_t launch_mixed_part<r, K_C2C>(bool, const PassArgs&, cudaStream_t);  \
  template <> cudaError_t launch_mixed_part<r, K_R2C>(bool, const PassArgs&, cudaStream_t);  \
  template <> cudaError_t launch_mixed_part<r, K_C2R>(bool, const PassArgs&, cudaStream_t);
GBFFT_MIXED_R1S(GBFFT_MIXED_DECL)

cudaError_t launch_mixed_f32(int kind, bool contiguous, const PassArgs& a, cudaStream_t s) {
  switch (a.tpl) {
#define GBFFT_MIXED_CASE(r)                                                     \
  case r:                                                                       \
    return kind == K_C2C   ? launch_mixed_part<r, K_C2C>(contiguous, a, s)      \
           : kind == K_R2C ? launch_mixed_part<r, K_R2C>(contiguous, a, s)      \
                           : launch_mixed_part<r, K_C2R>(contiguous, a, s);
    GBFFT_MIXED_R1S(GBFFT_MIXED_CASE)
#undef GBFFT_MIXED_CASE
    default: return cudaErrorNotSupported;
  }
}

}  // namespace gbfft
#endif
