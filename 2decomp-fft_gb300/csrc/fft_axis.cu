// Batched 1D FFT passes along one axis of an x-fastest 3D array, for sm_103a.
//
// This file replaces the 1D transforms of the reference backends -- the
// Glassman loops c2c_1m_{x,y,z} / r2c_1m_{x,z} / c2r_1m_{x,z} of
// src/fft_generic.f90:112-384 and the cuFFT plans of
// src/fft_cufft.f90:73-258 -- with one kernel family:
//
//  * A CTA owns L whole lines.  Each line is transformed by `tpl` threads
//    with a mixed-radix Stockham (self-sorting) FFT: every stage reads the
//    line at stride n/R, applies twiddles and a radix-R butterfly in
//    registers and writes it back in sorted order.  Between stages the line
//    sits in shared memory, padded by one slot every 32 to keep strided
//    accesses bank-conflict free.
//  * This file holds the runtime-planned kernel, which handles any length up
//    to kMaxN: lines are loaded into shared memory, each stage ping-pongs
//    between two shared buffers, and the result is stored from the last one.
//    FP32 powers of two and smooth lengths run compile-time plans
//    (fft_fast.cuh, fft_mixed.cuh) or the smooth-length kernel (fft_rt.cuh)
//    instead, and FP64 lines the fixed-point kernels (fft_fx.cuh).
//  * Along y and z the lanes of a warp walk neighbouring x positions, so the
//    strided transforms still read and write contiguous x segments.
//  * r2c/c2r carry two real lines in one complex line (z = a + i b) and
//    separate / combine the two half spectra in the last / first stage, which
//    halves the FFT work and keeps the reference's c2r rule that the
//    imaginary parts of the DC and Nyquist bins are ignored
//    (src/fft_generic.f90:318-330: buf(i) = conjg(buf(d1+2-i)), real part).
//  * Backward transforms run as conj(F(conj(x))), so only forward butterflies
//    and one table of forward twiddles exp(-2 pi i m/n) exist.
#include <atomic>

#include "fft_common.cuh"
#include "fft_pp.cuh"
#include "gbfft_internal.h"

namespace gbfft {

namespace {

using namespace dev;

std::atomic<long long> g_launches{0};

// Runtime-planned pass: any length up to kMaxN, any factorisation (run_pp_lines,
// fft_pp.cuh).
template <typename T, int KIND, bool CONTIG>
__global__ void __launch_bounds__(kMaxThreads)
    axis_pass_kernel(const __grid_constant__ PassArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  chained_entry();
  LineCtx<T, KIND, CONTIG> c;
  c.init(a);
  run_pp_lines<T, KIND, CONTIG>(c, a, reinterpret_cast<Cx<T>*>(smem_raw), (size_t)a.n * a.L);
}

template <typename T, int KIND, bool CONTIG>
cudaError_t launch_typed(const PassArgs& a, cudaStream_t stream) {
  const size_t smem = pass_smem_bytes(sizeof(T), a.n, a.L);
  auto kern = axis_pass_kernel<T, KIND, CONTIG>;
  // the limit is a per-device attribute of the kernel: set it on every
  // launch that needs it (cheap), so a second device is covered too
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  const dim3 block = CONTIG ? dim3(a.tpl, a.L) : dim3(a.L, a.tpl);
  const dim3 grid((unsigned)((a.nlines + a.L - 1) / a.L), CONTIG ? 1u : (unsigned)a.nv);
  const cudaError_t err = launch_chained(kern, grid, block, smem, stream, a);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return err != cudaSuccess ? err : cudaGetLastError();
}

// Identity copy.  A block of 1024 threads moves 2048 consecutive words of the
// widest type both arrays are aligned to, two a thread, both loads in flight;
// the last block also moves the bytes after the last whole word.  One block
// per 32 KB instead of a grid that strides over the array: the blocks reach
// DRAM in address order (256^3 complex128, 268 MB: 90.4 -> 79.2 us, 6.8 TB/s;
// 256 x 4, 256 x 8, 512 x 4 words, 32-byte words and streaming hints measured
// 79.7 to 80.7), and a chain of small copies overlaps its launches.
constexpr int kCopyThreads = 1024;
template <typename V>
__global__ void __launch_bounds__(kCopyThreads) copy_kernel(const V* s, V* d, size_t n, int tail) {
  chained_entry();
  const size_t i = (size_t)blockIdx.x * (2 * kCopyThreads) + threadIdx.x;
  const bool two = i + kCopyThreads < n;
  V a, b;
  if (i < n) a = s[i];
  if (two) b = s[i + kCopyThreads];
  if (i < n) d[i] = a;
  if (two) d[i + kCopyThreads] = b;
  if (blockIdx.x + 1 == gridDim.x && (int)threadIdx.x < tail)
    reinterpret_cast<unsigned char*>(d + n)[threadIdx.x] = reinterpret_cast<const unsigned char*>(s + n)[threadIdx.x];
}

template <typename V>
cudaError_t launch_copy_as(const void* src, void* dst, size_t bytes, cudaStream_t stream) {
  const size_t n = bytes / sizeof(V), blocks = (n + 2 * kCopyThreads - 1) / (2 * kCopyThreads);
  const cudaError_t err =
      launch_chained(copy_kernel<V>, dim3((unsigned)(blocks ? blocks : 1)), dim3(kCopyThreads), 0, stream,
                     reinterpret_cast<const V*>(src), reinterpret_cast<V*>(dst), n, (int)(bytes % sizeof(V)));
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return err != cudaSuccess ? err : cudaGetLastError();
}

}  // namespace

size_t pass_smem_bytes(int prec_bytes, int n, int L) {
  const size_t e = (size_t)n * (size_t)L;
  return 2 * (e + (e >> 4) + 1) * (size_t)(2 * prec_bytes);
}

namespace {
cudaError_t launch_axis_one(int prec_bytes, int kind, bool contiguous, const PassArgs& a, cudaStream_t stream) {
  if (a.tma) {
    if (!tma_pass_supported(prec_bytes, kind, contiguous, a)) return cudaErrorInvalidValue;
    return launch_tma_pass(a, stream);
  }
  if (a.fast == 5) {
    if (!tc_pass_supported(prec_bytes, kind, contiguous, a)) return cudaErrorInvalidValue;
    return launch_tc_pass(a, stream);
  }
  if (a.fast == 8)
    return prec_bytes == 4 ? launch_rt_f32(kind, contiguous, a, stream) : launch_rt_f64(kind, contiguous, a, stream);
  if (a.fast == 7) return prec_bytes == 8 ? launch_fxc(kind, contiguous, a, stream) : cudaErrorInvalidValue;
  if (a.fast == 6) return prec_bytes == 8 ? launch_fx(kind, contiguous, a, stream) : cudaErrorInvalidValue;
  if (a.fast && prec_bytes != 4) return cudaErrorInvalidValue;  // the other compile-time kernels are FP32's
  if (a.fast == 4) return launch_gen_f32(kind, contiguous, a, stream);
  if (a.fast == 3) return launch_split_f32(kind, contiguous, a, stream);
  if (a.fast == 2) return launch_mixed_f32(kind, contiguous, a, stream);
  if (a.fast)
    return kind == K_C2C ? launch_fast_f32_c2c(kind, contiguous, a, stream)
                         : launch_fast_f32_real(kind, contiguous, a, stream);
#define GB_DISPATCH(T)                                                              \
  switch (kind) {                                                                   \
    case K_C2C: return contiguous ? launch_typed<T, K_C2C, true>(a, stream)         \
                                  : launch_typed<T, K_C2C, false>(a, stream);       \
    case K_R2C: return contiguous ? launch_typed<T, K_R2C, true>(a, stream)         \
                                  : launch_typed<T, K_R2C, false>(a, stream);       \
    case K_C2R: return contiguous ? launch_typed<T, K_C2R, true>(a, stream)         \
                                  : launch_typed<T, K_C2R, false>(a, stream);       \
    default: return cudaErrorInvalidValue;                                          \
  }
  if (prec_bytes == 4) {
    GB_DISPATCH(float)
  } else if (prec_bytes == 8) {
    GB_DISPATCH(double)
  }
#undef GB_DISPATCH
  return cudaErrorInvalidValue;
}
}  // namespace

// Strided one-shot passes with more planes than a grid's y extent allows
// run as several launches of at most kMaxGridY planes, each side's array
// offset by the planes already done (a line (u, v) starts at u + v * s_l, in
// elements of that side's type).  The persistent bulk-copy pass walks any
// number of planes itself.
cudaError_t launch_axis_pass(int prec_bytes, int kind, bool contiguous, const PassArgs& a,
                             cudaStream_t stream) {
  if (contiguous || a.tma || a.fast == 5 || a.nv <= kMaxGridY)  // persistent kernels take any plane count
    return launch_axis_one(prec_bytes, kind, contiguous, a, stream);
  const size_t cs = 2 * (size_t)prec_bytes, rs = (size_t)prec_bytes;
  const size_t src_e = kind == K_R2C ? rs : cs, dst_e = kind == K_C2R ? rs : cs;
  for (long long v0 = 0; v0 < a.nv; v0 += kMaxGridY) {
    PassArgs b = a;
    b.nv = (int)(a.nv - v0 < kMaxGridY ? a.nv - v0 : kMaxGridY);
    b.src = static_cast<const char*>(a.src) + v0 * a.s_src_l * src_e;
    b.dst = static_cast<char*>(a.dst) + v0 * a.s_dst_l * dst_e;
    cudaError_t err = launch_axis_one(prec_bytes, kind, contiguous, b, stream);
    if (err != cudaSuccess) return err;
  }
  return cudaSuccess;
}

cudaError_t launch_copy(const void* src, void* dst, size_t bytes, cudaStream_t stream) {
  if (bytes == 0 || src == dst) return cudaSuccess;
  const uintptr_t at = (uintptr_t)src | (uintptr_t)dst;
  if (at % 16 == 0) return launch_copy_as<uint4>(src, dst, bytes, stream);
  if (at % 8 == 0) return launch_copy_as<uint2>(src, dst, bytes, stream);
  if (at % 4 == 0) return launch_copy_as<unsigned>(src, dst, bytes, stream);
  // blocks of 2 KB of single bytes: up to 4 TB in one grid
  return launch_copy_as<unsigned char>(src, dst, bytes, stream);
}

long long launch_counter() { return g_launches.load(); }
void add_launches(long long n) { g_launches.fetch_add(n); }

}  // namespace gbfft
