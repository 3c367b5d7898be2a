// Shared-memory ping-pong Stockham stages with a runtime radix, used by the
// runtime-planned axis kernel (fft_axis.cu) and the real-to-real kernel
// (dtt.cu).  The line sits in a padded shared buffer (LineCtx::sidx); the
// twiddles come from a full-length table exp(-2 pi i m / N) (LineCtx::tw).
#pragma once

#include "fft_common.cuh"

namespace gbfft {
namespace dev {

// One Stockham stage of radix R, shared buffer A -> B.  Butterfly b
// (0 <= b < n/R) reads points b + r n/R, multiplies by
// W_{Ns R}^{(b mod Ns) r}, transforms, and writes points
// (b - b mod Ns) R + b mod Ns + r Ns.  One butterfly in flight per thread.
// Ctx: a LineCtx (or a type derived from it that supplies its own twiddle()).
template <typename T, int KIND, bool CONTIG, int R, class Ctx = LineCtx<T, KIND, CONTIG>>
__device__ __forceinline__ void stage_pp(const Ctx& c, const Cx<T>* A, Cx<T>* B, int Ns) {
  using C = Cx<T>;
  const int nb = c.N / R;
  const int tstride = c.N / (Ns * R);
#pragma unroll 1
  for (int b = c.t; b < nb; b += c.tpl) {
    C v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = A[c.sidx(b + r * nb)];
    const int k = b % Ns;
    if (k != 0) {
#pragma unroll
      for (int r = 1; r < R; ++r) v[r] = cmul(v[r], c.twiddle(k * r * tstride));
    }
    dftg<R>(v);
    const int base = (b - k) * R + k;
#pragma unroll
    for (int r = 0; r < R; ++r) B[c.sidx(base + r * Ns)] = v[r];
  }
}

// A stage of any radix (primes above 7): each output point is a direct sum
// over its R inputs, O(n R) per line.
template <typename T, int KIND, bool CONTIG, class Ctx = LineCtx<T, KIND, CONTIG>>
__device__ void stage_pp_generic(const Ctx& c, const Cx<T>* A, Cx<T>* B, int R, int Ns) {
  using C = Cx<T>;
  const int N = c.N, nb = N / R, tstride = N / (Ns * R);
#pragma unroll 1
  for (int o = c.t; o < N; o += c.tpl) {
    const int k = o % Ns;
    const int r = (o / Ns) % R;
    const int q = o / (Ns * R);
    const int b = q * Ns + k;
    const int step = (k * tstride + r * nb) % N;
    C acc = cmk<C>(T(0), T(0));
    int e = 0;
#pragma unroll 1
    for (int j = 0; j < R; ++j) {
      const C x = A[c.sidx(b + j * nb)], w = c.twiddle(e);
      acc.x += x.x * w.x - x.y * w.y;
      acc.y += x.x * w.y + x.y * w.x;
      e += step;
      if (e >= N) e -= N;
    }
    B[c.sidx(o)] = acc;
  }
}

// The radix stages of the lines in shared buffer A, ping-ponging with B; A is
// the last buffer written when it returns.
template <typename T, int KIND, bool CONTIG, class Ctx>
__device__ __forceinline__ void run_stages_pp(const Ctx& c, int nst, const int* radix, Cx<T>*& A, Cx<T>*& B) {
  using C = Cx<T>;
  int Ns = 1;
#pragma unroll 1
  for (int s = 0; s < nst; ++s) {
    const int R = radix[s];
    if (R == 16) stage_pp<T, KIND, CONTIG, 16>(c, A, B, Ns);
    else if (R == 8) stage_pp<T, KIND, CONTIG, 8>(c, A, B, Ns);
    else if (R == 4) stage_pp<T, KIND, CONTIG, 4>(c, A, B, Ns);
    else if (R == 2) stage_pp<T, KIND, CONTIG, 2>(c, A, B, Ns);
    else if (R == 3) stage_pp<T, KIND, CONTIG, 3>(c, A, B, Ns);
    else if (R == 5) stage_pp<T, KIND, CONTIG, 5>(c, A, B, Ns);
    else if (R == 7) stage_pp<T, KIND, CONTIG, 7>(c, A, B, Ns);
    else if (R == 11) stage_pp<T, KIND, CONTIG, 11>(c, A, B, Ns);
    else if (R == 13) stage_pp<T, KIND, CONTIG, 13>(c, A, B, Ns);
    else if (R == 17) stage_pp<T, KIND, CONTIG, 17>(c, A, B, Ns);
    else if (R == 19) stage_pp<T, KIND, CONTIG, 19>(c, A, B, Ns);
    else if (R == 23) stage_pp<T, KIND, CONTIG, 23>(c, A, B, Ns);
    else if (sizeof(T) == 4 && (R == 29 || R == 31)) {
      // in FP64 a butterfly of 29 or 31 points does not fit the registers
      if constexpr (sizeof(T) == 4) {
        if (R == 29) stage_pp<T, KIND, CONTIG, 29>(c, A, B, Ns);
        else stage_pp<T, KIND, CONTIG, 31>(c, A, B, Ns);
      }
    } else {
      stage_pp_generic<T, KIND, CONTIG>(c, A, B, R, Ns);
    }
    __syncthreads();
    C* tmp = A;
    A = B;
    B = tmp;
    Ns *= R;
  }
}

// The runtime-planned pass of a CTA's lines (e points in all): loaded into
// shared buffer 0, each stage ping-pongs between the two buffers, the result
// is stored from the last buffer written.
template <typename T, int KIND, bool CONTIG>
__device__ __forceinline__ void run_pp_lines(const LineCtx<T, KIND, CONTIG>& c, const PassArgs& a, Cx<T>* buf0,
                                             size_t e) {
  using C = Cx<T>;
  C* buf1 = buf0 + (e + (e >> 4) + 1);

#pragma unroll 1
  for (int n = c.t; n < c.N; n += c.tpl) buf0[c.sidx(n)] = c.gload(n);
  __syncthreads();

  C* A = buf0;
  C* B = buf1;
  run_stages_pp<T, KIND, CONTIG>(c, a.nst, a.radix, A, B);

  if (KIND == K_R2C) {
    c.store_r2c(A);
  } else {
#pragma unroll 1
    for (int n = c.t; n < c.N; n += c.tpl) c.gstore(n, A[c.sidx(n)]);
  }
}

}  // namespace dev
}  // namespace gbfft
