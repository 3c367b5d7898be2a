// Compile-time two-stage axis passes for FP32 lengths that are not powers of
// two: every n = R0 * R1 with R0 <= R1 <= 32 and R1 <= 3 R0 of the primes up
// to 13 (mixed_length in gbfft_internal.h), TPL = R1 threads a line:
//   stage 0: radix R0, thread t's butterfly from points t + r R1 as they are
//            loaded (c2r: both half spectra, combined in shared memory);
//   stage 1: radix R1 after R0 points: threads t < R0 own one butterfly each,
//            twiddles W_n^{t r} from the stage-major table, and store points
//            t + r R0 from their registers (r2c: through shared memory, which
//            splits the two real lines' spectra).
//
// What bounds them is memory: two stages are one exchange, the fewest that
// lines of 12 to 1024 points can have, the radices and strides are compile-time
// constants, and 20 to 32 points in flight a thread cover the latency.  Runtime
// plans of radices up to 16 spend 1.2 to 2.2 times as long in index arithmetic
// and in more exchanges.  Passes of 24 M points, us (28 at the copy rate), and in
// brackets the runtime plan (24, 225, 900) or the balanced three-stage one (360):
//   225  r2c x 47 (82)  c2r x 47 (84)  r2c z 43 (52)  c2r z 39 (72)  c2c y 38 (46)
//   360  r2c x 49 (73)  c2r x 49 (70)  r2c z 46 (76)  c2r z 40 (64)  c2c y 40 (73)
//   24   r2c x 54 (68)  c2r x 55 (79)  r2c z 45 (45)  c2r z 43 (58)  c2c y 36 (41)
//   900  r2c x 43 (93)  c2r x 44 (105) r2c z 53 (89)  c2r z 49 (126) c2c y 48 (81)
// The rel-L2 error against 64 bits is that of the runtime and balanced plans,
// roundings in another order: 0.965 of it on average over the passes of 177
// lengths on noise and on modes (0.88 to 1.04 for single lengths), 0.98 over 68
// random boxes (0.87 to 1.15 for single ones).
#pragma once

#include <type_traits>

#include "fft_io.cuh"

namespace gbfft {
namespace mixed {

using namespace dev;

// Shared-memory slots.  The exchange is an R1 x R0 matrix (row t holds stage
// 0's outputs of thread t) whose pitch is odd, so that both its column-wise
// writes and its row-wise reads touch each bank once; the line in natural
// order (c2r inputs, r2c outputs) lies dense in the same place.
template <int N, bool CONTIG>
struct Slots {
  static constexpr int R0 = mixed_r0(N), R1 = N / R0, P = R0 | 1;
  int line, L;
  __device__ __forceinline__ int natural(int n) const { return CONTIG ? line * (R1 * P) + n : n * L + line; }
  __device__ __forceinline__ int matrix(int row, int col) const { return natural(row * P + col); }
};

template <int N, class Ctx>
__device__ __forceinline__ void run_mixed(const Ctx& c, float2* Sm) {
  constexpr int KIND = Ctx::kind;
  constexpr bool CONTIG = Ctx::contiguous;
  constexpr int R0 = mixed_r0(N), R1 = N / R0, H = N / 2 + 1, J = (H + R1 - 1) / R1;
  const rt::Io<float, KIND, CONTIG, Ctx> io(c);
  const Slots<N, CONTIG> slot{c.line, c.L};
  const int t = c.t;
  // a backward transform conjugates on the way in (c2r: in its inputs) and out
  const int back = KIND == K_C2R || (KIND == K_C2C && c.inverse) ? (int)0x80000000 : 0;
  auto turn = [back](float2 z) { return make_float2(z.x, __int_as_float(__float_as_int(z.y) ^ back)); };
  float2 v[R1];
  if constexpr (KIND == K_C2R) {
    float2 x[J], y[J];
#pragma unroll
    for (int i = 0; i < J; ++i) {
      x[i] = y[i] = io.zero();
      if (H % R1 == 0 || i < J - 1 || t + i * R1 < H) io.halves(i * R1, x[i], y[i]);
    }
#pragma unroll
    for (int i = 0; i < J; ++i) {
      const int j = t + i * R1;
      if (j == 0 || 2 * j == N) x[i].y = y[i].y = 0.f;  // Im of the DC and Nyquist bins is ignored
      if (j < H) {
        // z = x1 + i x2, conjugated for the inverse-by-conjugation
        Sm[slot.natural(j)] = make_float2(x[i].x - y[i].y, -(x[i].y + y[i].x));
        if (j > 0 && 2 * j < N) Sm[slot.natural(N - j)] = make_float2(x[i].x + y[i].y, x[i].y - y[i].x);
      }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < R0; ++r) v[r] = Sm[slot.natural(t + r * R1)];
    __syncthreads();
  } else {
#pragma unroll
    for (int r = 0; r < R0; ++r) v[r] = io.load(r * R1);
    if constexpr (KIND == K_C2C) {
#pragma unroll
      for (int r = 0; r < R0; ++r) v[r] = turn(v[r]);
    }
  }
  rt::dft_f32<R0>(v);
#pragma unroll
  for (int r = 0; r < R0; ++r) Sm[slot.matrix(t, r)] = v[r];
  __syncthreads();
  const bool act = t < R0;
  if (act) {
#pragma unroll
    for (int r = 0; r < R1; ++r) v[r] = Sm[slot.matrix(r, t)];
#pragma unroll
    for (int r = 1; r < R1; ++r) v[r] = cmul(v[r], c.twiddle((R0 - 1) + (r - 1) * R0 + t));
    rt::dft_f32<R1>(v);
  }
  if constexpr (KIND == K_R2C) {
    __syncthreads();
    if (act) {
#pragma unroll
      for (int r = 0; r < R1; ++r) Sm[slot.natural(t + r * R0)] = v[r];
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < J; ++i) {
      const int k = t + i * R1;
      if (k < H) {
        const float2 zk = Sm[slot.natural(k)], zm = Sm[slot.natural(k == 0 ? 0 : N - k)];
        io.put_halves(i * R1, make_float2((zk.x + zm.x) * 0.5f, (zk.y - zm.y) * 0.5f),
                      make_float2((zk.y + zm.y) * 0.5f, (zm.x - zk.x) * 0.5f));
      }
    }
  } else if (act) {
#pragma unroll
    for (int r = 0; r < R1; ++r) io.store(r * R0, turn(v[r]));
  }
}

// Registers: 64 a thread for butterflies of at most 16 points, 80 up to 24,
// 128 beyond.
template <int KIND, bool CONTIG, int N>
__global__ void __launch_bounds__(256, N / mixed_r0(N) <= 16 ? 4 : N / mixed_r0(N) <= 24 ? 3 : 2)
    mixed_pass_kernel(const __grid_constant__ PassArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  chained_entry();
  LineCtx<float, KIND, CONTIG> c;
  c.init(a);
  run_mixed<N>(c, reinterpret_cast<float2*>(smem_raw));
}

template <int KIND, bool CONTIG, int N>
cudaError_t launch_n(const PassArgs& a, cudaStream_t stream) {
  constexpr int R0 = mixed_r0(N), R1 = N / R0;
  const size_t smem = mixed_smem_bytes(R0, R1, a.L);
  if (a.tpl != R1 || a.L < 1 || a.L * a.tpl > 256 || smem > kFxMaxSmem) return cudaErrorInvalidValue;
  auto kern = mixed_pass_kernel<KIND, CONTIG, N>;
  if (smem > 48 * 1024) {
    cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err != cudaSuccess) return err;
  }
  const dim3 block = CONTIG ? dim3(a.tpl, a.L) : dim3(a.L, a.tpl);
  const dim3 grid((unsigned)((a.nlines + a.L - 1) / a.L), CONTIG ? 1u : (unsigned)a.nv);
  const cudaError_t err = launch_chained(kern, grid, block, smem, stream, a);
  add_launches(1);
  return err != cudaSuccess ? err : cudaGetLastError();
}

}  // namespace mixed
}  // namespace gbfft
