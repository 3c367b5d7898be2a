// Instantiations of the compile-time fixed-point passes (fft_fxc.cuh).  The
// build compiles this file once for every part: a line kind, a layout and a
// group of lengths (GBFFT_FXC_PART = group * 6 + kind * 2 + contiguous), and
// once without, for the dispatch.
#ifdef GBFFT_FXC_PART
#include "fft_fxc.cuh"

#define GBFFT_CAT2(a, b) a##b
#define GBFFT_CAT(a, b) GBFFT_CAT2(a, b)

namespace gbfft {

cudaError_t GBFFT_CAT(launch_fxc_part, GBFFT_FXC_PART)(const PassArgs& a, cudaStream_t s) {
  constexpr int kGroup = GBFFT_FXC_PART / 6, kKind = GBFFT_FXC_PART % 6 / 2;
  constexpr bool kContig = GBFFT_FXC_PART % 2 == 1;
#define GBFFT_FXC_CASE(g, N, T, r0, r1, r2, r3)                                              \
  if constexpr (g == kGroup)                                                                 \
    if (a.n == N) return fx::launch_p<fx::Plan<N, T, r0, r1, r2, r3>, kKind, kContig>(a, s);
  GBFFT_FXC_PLANS(GBFFT_FXC_CASE)
#undef GBFFT_FXC_CASE
  return cudaErrorNotSupported;
}

}  // namespace gbfft
#else
#include "gbfft_internal.h"

namespace gbfft {

#define GBFFT_FXC_DECL(p) cudaError_t launch_fxc_part##p(const PassArgs& a, cudaStream_t s);
#define GBFFT_FXC_PARTS(X) X(0) X(1) X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11)
GBFFT_FXC_PARTS(GBFFT_FXC_DECL)

cudaError_t launch_fxc(int kind, bool contiguous, const PassArgs& a, cudaStream_t s) {
  int group = -1;
#define GBFFT_FXC_GROUP(g, N, T, r0, r1, r2, r3) \
  if (a.n == N) group = g;
  GBFFT_FXC_PLANS(GBFFT_FXC_GROUP)
#undef GBFFT_FXC_GROUP
  if (group < 0) return cudaErrorNotSupported;
  switch (group * 6 + kind * 2 + (contiguous ? 1 : 0)) {
#define GBFFT_FXC_CALL(p) \
  case p: return launch_fxc_part##p(a, s);
    GBFFT_FXC_PARTS(GBFFT_FXC_CALL)
#undef GBFFT_FXC_CALL
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace gbfft
#endif
