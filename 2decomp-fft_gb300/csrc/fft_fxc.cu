// Instantiations of the compile-time fixed-point passes (fft_fxc.cuh).  The
// build compiles this file once for every part: a line kind, a layout and a
// group of lengths (GBFFT_FXC_PART = group * 8 + kind * 2 + contiguous, kind
// 3 the real-to-real passes), and
// once without, for the dispatch.
#ifdef GBFFT_FXC_PART
#include "fft_fxc.cuh"

#define GBFFT_CAT2(a, b) a##b
#define GBFFT_CAT(a, b) GBFFT_CAT2(a, b)

namespace gbfft {

namespace {
constexpr int kGroup = GBFFT_FXC_PART / 8, kKind = GBFFT_FXC_PART % 8 / 2;
constexpr bool kContig = GBFFT_FXC_PART % 2 == 1;
#if GBFFT_FXC_PART % 8 / 2 == 3
using Args = DttArgs;
int length(const Args& a) { return a.M; }
template <class P>
cudaError_t launch(const Args& a, cudaStream_t s) { return fx::launch_r2r_p<P, kContig>(a, s); }
#else
using Args = PassArgs;
int length(const Args& a) { return a.n; }
template <class P>
cudaError_t launch(const Args& a, cudaStream_t s) { return fx::launch_p<P, kKind, kContig>(a, s); }
#endif
}  // namespace

cudaError_t GBFFT_CAT(launch_fxc_part, GBFFT_FXC_PART)(const Args& a, cudaStream_t s) {
#define GBFFT_FXC_CASE(g, N, T, r0, r1, r2, r3)                                  \
  if constexpr (g == kGroup)                                                     \
    if (length(a) == N) return launch<fx::Plan<N, T, r0, r1, r2, r3>>(a, s);
  GBFFT_FXC_PLANS(GBFFT_FXC_CASE)
#undef GBFFT_FXC_CASE
  return cudaErrorNotSupported;
}

}  // namespace gbfft
#else
#include "gbfft_internal.h"

namespace gbfft {

#define GBFFT_FXC_PARTS(X) \
  X(0) X(1) X(2) X(3) X(4) X(5) X(8) X(9) X(10) X(11) X(12) X(13) X(16) X(17) X(18) \
  X(19) X(20) X(21) X(24) X(25) X(26) X(27) X(28) X(29) X(32) X(33) X(34) X(35) X(36) X(37)
#define GBFFT_FXC_R2R_PARTS(X) X(6) X(7) X(14) X(15) X(22) X(23) X(30) X(31) X(38) X(39)
#define GBFFT_FXC_DECL(p) cudaError_t launch_fxc_part##p(const PassArgs& a, cudaStream_t s);
#define GBFFT_FXC_R2R_DECL(p) cudaError_t launch_fxc_part##p(const DttArgs& a, cudaStream_t s);
GBFFT_FXC_PARTS(GBFFT_FXC_DECL)
GBFFT_FXC_R2R_PARTS(GBFFT_FXC_R2R_DECL)
#define GBFFT_FXC_CALL(p) \
  case p: return launch_fxc_part##p(a, s);

namespace {
int group_of(int n) {
  int group = -1;
#define GBFFT_FXC_GROUP(g, N, T, r0, r1, r2, r3) \
  if (n == N) group = g;
  GBFFT_FXC_PLANS(GBFFT_FXC_GROUP)
#undef GBFFT_FXC_GROUP
  return group;
}
}  // namespace

cudaError_t launch_fxc(int kind, bool contiguous, const PassArgs& a, cudaStream_t s) {
  switch (group_of(a.n) * 8 + kind * 2 + (contiguous ? 1 : 0)) {
    GBFFT_FXC_PARTS(GBFFT_FXC_CALL)
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_fxc_r2r(bool contiguous, const DttArgs& a, cudaStream_t s) {
  switch (group_of(a.M) * 8 + 6 + (contiguous ? 1 : 0)) {
    GBFFT_FXC_R2R_PARTS(GBFFT_FXC_CALL)
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace gbfft
#endif
