// Internal declarations shared by the kernels and the host engine of the
// GB300 3D FFT backend.  Nothing here is part of the C ABI (include/gbfft.h).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

struct gbfft_engine_s;

namespace gbfft {

constexpr int kMaxStages = 16;    // radix stages of one axis plan
constexpr int kMaxE = 16;         // complex values a thread holds in one stage
constexpr int kMaxThreads = 512;  // threads in one CTA of an axis pass
constexpr int kMaxN = 8192;       // longest axis a single-tile pass supports
constexpr int kMaxGridY = 65535;  // planes (grid.y) of one strided launch
constexpr int kSmsDefault = 152;  // SMs of a GB300: the occupancy targets of small grids
constexpr int kMaxDevices = 64;   // per-device caches of launch parameters

// What one axis pass does to each line.
enum Kind : int {
  K_C2C = 0,  // complex line -> complex line
  K_R2C = 1,  // two real lines -> two half spectra (n/2+1 values each)
  K_C2R = 2,  // two half spectra -> two real lines
};

// Radices with a hand-written butterfly; any other factor runs through the
// generic direct-sum stage.
__host__ __device__ constexpr bool radix_is_special(int r) {
  return r == 2 || r == 3 || r == 4 || r == 5 || r == 7 || r == 8 || r == 16;
}

// Arguments of one batched-line FFT pass along one axis of a 3D array.
//
// A "line" is one 1D transform.  Two addressings exist:
//   contiguous (the x axis): line l starts at l * s_l, point n at + n * s_n;
//   strided   (the y and z axes): lines are indexed by (u, v) with u the
//     x index (unit stride, so a warp reads neighbouring lines in one
//     transaction) and v the remaining axis; line (u, v) starts at
//     u + v * s_l and point n sits at + n * s_n.
// For K_R2C / K_C2R two neighbouring real lines (2c, 2c+1 along l or u) are
// carried by one complex line c.  All strides are in elements of the
// array's own type (real elements for the real side of r2c/c2r).
// Chirp-z (Bluestein) tables of one axis whose length has a large prime
// factor: the length-n transform is a circular convolution of length m (a
// power of two >= 2n - 1) between the input times a chirp and the
// conjugate chirp, done as two forward m-point FFTs.  Device pointers; the
// struct itself lives on the host, in the engine's axis plan.
struct BlueTables {
  int m;                    // convolution length
  int nst;                  // radix stages of the m-point FFTs
  int radix[kMaxStages];
  const void* chirp;        // w_j = exp(-i pi j^2 / n), j < n
  const void* filt;         // FFT_m of b (b_j = conj w_j at j and m - j, 0 between), divided by m
  const void* twm;          // exp(-2 pi i k / m), k < m
};

// Axes whose largest prime factor exceeds this run the chirp-z path: a
// direct-sum stage costs that many multiply-adds a point.
constexpr int kBluePrime = 256;

// Plan of one axis for the fixed-point FP64 kernels (fft_fx.cu) and the
// smooth-length kernels (fft_rt.cuh): radix stages after ns points, and for
// the scale of a fixed-point line, per stage, the exponent that bounds how
// many inputs a value then sums (lg) and the powers of two it was divided
// by (shift).  Built by the engine for one length; the struct lives on the
// host and travels as a kernel argument.
struct FxPlan {
  int nst;
  int radix[kMaxStages];
  int ns[kMaxStages];
  unsigned magic[kMaxStages];  // ceil(2^32 / ns)
  int lg[kMaxStages];
  int shift[kMaxStages];
  const void* tw;    // stage-major roots (stage_twiddles order), Q62 or FP32
  const void* root;  // the n roots in Q62, for direct-sum stages
  int tpl;           // threads a line (runtime plans: at least n / kFxPoints)
  int ct;            // 1: a compile-time plan (fft_fxc.cuh)
  int rt;            // 1: a smooth-length runtime plan (fft_rt.cuh)
};
constexpr int kFxPoints = 8;        // points a thread loads at most
constexpr int kFxMaxThreads = 512;  // threads of a CTA
constexpr size_t kFxMaxSmem = 200 * 1024;
constexpr size_t kFxWordBytes = 48;  // scale words of a line (fx::Words)
// Shared memory of L lines of n points: two padded buffers and the lines'
// scale words.
__host__ __device__ constexpr size_t fx_smem_bytes(int n, int L) {
  const size_t e = (size_t)n * (size_t)L;
  return 2 * (e + (e >> 4) + 1) * 16 + (size_t)L * kFxWordBytes;
}
// ... and of the compile-time plans (fft_fxc.cuh): one buffer, padded by an
// entry in eight; a single line keeps room for the two of its FP64 fallback.
__host__ __device__ constexpr size_t fxc_smem_bytes(int n, int L) {
  const size_t one = ((size_t)n + n / 8 + 2) * (size_t)L;
  return (L == 1 ? 2 * one : one) * 16 + 32 + (size_t)L * kFxWordBytes;
}
// Lengths with a compile-time plan (fft_fxc.cuh): X(group, n, threads a line,
// radices).  The radices stay at most 10 (64 registers a thread, four CTAs
// of 256 threads an SM) but for 1024, 2048 and 4096 points, and the threads a line
// are those that leave the fewest idle over the stages.  `group` splits the
// instantiations over translation units.
// The list is a choice, not a rule: the powers of two, and of the smooth
// lengths those of the grids that this library is tested and measured on and
// round ones like them.  The other 7-smooth lengths (112, 140, 168, 224, 252, 280,
// 336, 448, 504, 672, 840, 896 and 60 odd more up to 1024) would gain as much as
// these did over the runtime plans (fft_rt.cuh), 1.1 to 1.3 times, for 5 MB of
// library each.  r2c / c2r x passes of 24 M points, us, here and on the runtime
// plan, as measured when the list was made:
//   72  118 / 117   144 / 158      450  205 / 208   238 / 254
//   144 146 / 148   188 / 209      540  192 / 196   218 / 236
//   225 176 / 174   203 / 222      720  189 / 187   225 / 233
//   360 183 / 178   216 / 231      960  194 / 189   223 / 244
// 600 points have no plan of ten points a thread that keeps three stages: with
// four (10 10 3 2) 242 / 242, on the runtime plan 203 / 220.
#define GBFFT_FXC_PLANS(X)         \
  X(0, 16, 4, 4, 4, 1, 1)          \
  X(0, 32, 4, 8, 4, 1, 1)          \
  X(0, 48, 8, 8, 6, 1, 1)          \
  X(0, 64, 8, 8, 8, 1, 1)          \
  X(0, 96, 12, 8, 4, 3, 1)         \
  X(0, 126, 14, 9, 7, 2, 1)        \
  X(0, 128, 16, 8, 4, 4, 1)        \
  X(0, 160, 20, 10, 4, 4, 1)       \
  X(0, 180, 20, 10, 9, 2, 1)       \
  X(0, 192, 24, 8, 8, 3, 1)        \
  X(1, 243, 27, 9, 9, 3, 1)        \
  X(1, 256, 32, 8, 8, 4, 1)        \
  X(1, 320, 40, 10, 8, 4, 1)       \
  X(1, 384, 48, 8, 8, 6, 1)        \
  X(1, 400, 50, 10, 8, 5, 1)       \
  X(1, 512, 64, 8, 8, 8, 1)        \
  X(1, 1024, 64, 16, 8, 8, 1)      \
  X(1, 2048, 128, 16, 16, 8, 1)    \
  X(1, 4096, 256, 16, 16, 16, 1)   \
  X(2, 72, 9, 9, 8, 1, 1)          \
  X(2, 100, 10, 10, 10, 1, 1)      \
  X(2, 144, 24, 6, 6, 4, 1)        \
  X(2, 200, 20, 10, 10, 2, 1)      \
  X(2, 225, 25, 9, 5, 5, 1)        \
  X(2, 270, 30, 10, 9, 3, 1)       \
  X(2, 324, 41, 9, 9, 4, 1)        \
  X(2, 450, 50, 10, 9, 5, 1)       \
  X(2, 540, 60, 10, 9, 3, 2)       \
  X(2, 640, 80, 10, 8, 8, 1)       \
  X(2, 768, 96, 8, 8, 4, 3)        \
  X(2, 960, 120, 10, 8, 4, 3)      \
  X(3, 80, 10, 10, 8, 1, 1)        \
  X(3, 108, 18, 6, 6, 3, 1)        \
  X(3, 150, 30, 6, 5, 5, 1)        \
  X(3, 210, 42, 7, 6, 5, 1)        \
  X(3, 240, 30, 10, 8, 3, 1)       \
  X(3, 288, 36, 9, 8, 4, 1)        \
  X(3, 360, 45, 10, 9, 4, 1)       \
  X(3, 480, 60, 10, 4, 4, 3)       \
  X(3, 576, 72, 9, 8, 8, 1)        \
  X(3, 648, 108, 6, 6, 6, 3)       \
  X(3, 800, 100, 10, 10, 8, 1)     \
  X(3, 1000, 100, 10, 10, 10, 1)   \
  X(4, 90, 10, 10, 9, 1, 1)        \
  X(4, 120, 15, 10, 4, 3, 1)       \
  X(4, 162, 18, 9, 9, 2, 1)        \
  X(4, 216, 36, 6, 6, 6, 1)        \
  X(4, 250, 25, 10, 5, 5, 1)       \
  X(4, 300, 34, 10, 10, 3, 1)      \
  X(4, 432, 72, 6, 6, 6, 2)        \
  X(4, 500, 50, 10, 10, 5, 1)      \
  X(4, 720, 90, 10, 9, 8, 1)       \
  X(4, 900, 100, 10, 10, 9, 1)
// threads of a CTA: 256, or what four lines (64-byte rows of a strided tile)
// take
__host__ __device__ constexpr int fxc_max_threads(int tpl) { return tpl <= 64 ? 256 : tpl <= 128 ? 4 * tpl : 512; }
struct FxcShape {
  int tpl, r[4];  // tpl 0: no compile-time plan
};
__host__ __device__ constexpr FxcShape fxc_shape(int n) {
#define GBFFT_FXC_SHAPE(g, N, T, a, b, c, d) \
  if (n == N) return FxcShape{T, {a, b, c, d}};
  GBFFT_FXC_PLANS(GBFFT_FXC_SHAPE)
#undef GBFFT_FXC_SHAPE
  return FxcShape{0, {0, 0, 0, 0}};
}

struct PassArgs {
  const void* src;
  void* dst;
  const void* tw;  // n complex roots exp(-2 pi i m / n), m = 0..n-1
  long long s_src_n, s_src_l;
  long long s_dst_n, s_dst_l;
  int n;           // transform length
  int nst;         // number of radix stages (0 when n == 1)
  int L;           // complex lines per CTA
  int tpl;         // threads per line
  int inverse;     // 1: backward (+i) transform, done as conj(F(conj(x)))
  int nlines;      // complex lines along l (contiguous) or u (strided)
  int real_lines;  // r2c/c2r: real lines along l or u (may be odd)
  int nv;          // strided: extent of v (grid.y)
  int first_fused; // stage 0 reads global memory directly
  int last_fused;  // last stage writes global memory directly
  int fast;        // 1: compile-time power-of-two kernel, 2: mixed-radix kernel,
                   // 3: split-precision tensor-core kernel (mma.sync), 4:
                   // balanced non-power-of-two plan, 5: split-precision
                   // tcgen05 kernel (fft_tc.cu), 6: fixed-point FP64 kernel
                   // (fft_fx.cu), 7: its compile-time plans (fft_fxc.cuh),
                   // 8: runtime plans of smooth lengths (fft_rt.cuh)
  int pair_vec;    // r2c/c2r on strided lines, bit 0: the two real lines of a
                   // pair are adjacent and aligned (read/write as one pair);
                   // bit 1 (FP32): so are their two complex lines, 16-byte
                   // aligned (one 16-byte access for both)
  int csize;       // fast == 1, one-shot: 0, or launch CTAs in clusters of
                   // csize neighbours (co-scheduled: their row segments
                   // reach DRAM together)
  int csync;       // with csize: the CTAs of a cluster start with a
                   // cluster barrier
  int row_w;       // strided, nv == 1: 0, or the lines are the positions
                   // of whole (x, y) planes taken flat: line u is point
                   // (u % row_w, u / row_w) of the plane and starts at
                   // u % row_w + (u / row_w) * s_src_r (s_dst_r), so that
                   // a tile's row segments are as aligned as the plane
  long long s_src_r, s_dst_r;
  int tma;         // strided FP32 c2c pass (fast == 1) run by the persistent
                   // kernel whose tiles arrive by bulk tensor copies
                   // (fft_tma.cu); needs tma_pass_supported()
  int* status;     // device word set to 1 when a bounded wait of the pass
                   // gave up, 2 when a check of the bounds-checked build
                   // caught an access outside an array (null: not recorded)
  long long src_elems, dst_elems;  // extents of the two arrays in elements of
                                   // each side's type (bounds-checked build)
  const FxPlan* fx;  // fast 6, 7, 8: the axis's host-side plan; the kernels get
                     // a copy
  const BlueTables* blue;  // host-side tables of the chirp-z path (fft_long.cu),
                           // null unless the axis runs it; never read on the device
  int radix[kMaxStages];
};

// Power-of-two lengths with a compile-time-planned kernel (fft_fast.cuh):
// 16 points per thread, n / 16 threads per line.
__host__ __device__ constexpr bool fast_length(int n) {
  return n >= 16 && n <= 4096 && (n & (n - 1)) == 0;
}
// Radix plan of the power-of-two kernel, for E points per thread.  E = 32
// (strided y/z lines of length 512 or 1024): two stages, 32 x (n/32), one
// exchange.  E = 16 (the default), 8 or 4: radix-E stages, then one stage
// of the remaining factor.  E = 8 (lines of at most 256 points) and E = 4
// (at most 128) give short lines more threads, for grids too small to
// fill the GPU at 16 points a thread.
__host__ __device__ constexpr int ilog2c(int n) { return n <= 1 ? 0 : 1 + ilog2c(n / 2); }
__host__ __device__ constexpr int fast_points(int n, bool contiguous) {
  return (!contiguous && (n == 512 || n == 1024)) ? 32 : 16;
}
// Points per thread the power-of-two kernel offers for length n.
__host__ __device__ constexpr bool fast_e_ok(int n, int e) {
  return n >= 16 && n <= 4096 && (n & (n - 1)) == 0 &&
         (e == 16 || (e == 32 && (n == 512 || n == 1024)) || (e == 8 && n <= 256) || (e == 4 && n <= 128));
}
// Lengths with more than one power-of-two plan.
__host__ __device__ constexpr bool fast_has_alt(int n) {
  return n == 512 || n == 1024 || (n >= 16 && n <= 256 && (n & (n - 1)) == 0);
}
__host__ __device__ constexpr int fast_nst(int n, int e) {
  return e == 32 ? 2 : ilog2c(n) / ilog2c(e) + (ilog2c(n) % ilog2c(e) ? 1 : 0);
}
__host__ __device__ constexpr int fast_radix(int n, int e, int s) {
  return e == 32 ? (s == 0 ? 32 : n / 32)
                 : (s < ilog2c(n) / ilog2c(e) ? e : (1 << (ilog2c(n) % ilog2c(e))));
}
// Thread limits of the power-of-two kernel, launched with one CTA per SM
// guaranteed: 16 points a thread at most 64 registers (1024 threads),
// 32 points a thread at most 128 (512 threads).  Smaller tiles of the same
// kernel still run several CTAs per SM.
__host__ __device__ constexpr int fast_max_threads(int e) { return e == 32 ? 512 : 1024; }
// Lengths with a compile-time two-stage plan (fft_mixed.cuh): n = R0 * R1,
// R0 <= R1 <= 32, the most balanced such split, R1 at most 3 R0 (only R0 of
// the R1 threads work in the second stage), of the primes up to 13 (a larger
// prime's butterfly costs its square).
__host__ __device__ constexpr int mixed_r0(int n) {
  int best = 0;
  for (int a = 2; a <= 32; ++a)
    if (n % a == 0 && n / a <= 32 && a <= n / a) best = a;
  return best;
}
__host__ __device__ constexpr bool mixed_length(int n) {
  if (n < 12 || n > 1024 || (n & (n - 1)) == 0 || n > 3 * mixed_r0(n) * mixed_r0(n)) return false;
  for (int p = 2; p <= 13; ++p)
    while (n % p == 0) n /= p;
  return n == 1;
}
// Shared memory of L lines: the exchange matrix with its odd pitch.
__host__ __device__ constexpr size_t mixed_smem_bytes(int r0, int r1, int L) {
  return (size_t)r1 * (size_t)(r0 | 1) * (size_t)L * 8;
}
// the second radices of these lengths (build.py's list)
#define GBFFT_MIXED_R1S(X)                                                                                          \
  X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12) X(13) X(14) X(15) X(16) X(18) X(20) X(21) X(22) X(24) X(25) X(26)  \
  X(27) X(28) X(30) X(32)
template <int R1, int KIND>
cudaError_t launch_mixed_part(bool contiguous, const PassArgs& a, cudaStream_t s);
cudaError_t launch_mixed_f32(int kind, bool contiguous, const PassArgs& a, cudaStream_t s);
// Non-power-of-two lengths with a balanced compile-time plan (fft_gen.cuh,
// fast::GenPlan): E points a thread, n / E threads a line.
__host__ __device__ constexpr bool gen_length(int n) {
  return n == 243 || n == 270 || n == 360 || n == 384 || n == 400;
}
__host__ __device__ constexpr int gen_points(int n) {
  return n == 243 ? 9 : (n == 270 || n == 360) ? 30 : n == 384 ? 24 : n == 400 ? 20 : 0;
}
// the plan's radices, stage by stage (0 after the last)
__host__ __device__ constexpr int gen_radix(int n, int s) {
  return n == 243 ? (s < 2 ? 9 : s == 2 ? 3 : 0)
       : n == 270 ? (s == 0 ? 15 : s == 1 ? 6 : s == 2 ? 3 : 0)
       : n == 360 ? (s == 0 ? 10 : s < 3 ? 6 : 0)
       : n == 384 ? (s < 2 ? 8 : s == 2 ? 6 : 0)
       : n == 400 ? (s < 2 ? 20 : 0) : 0;
}
// thread limit: E <= 16 at most 64 registers (1024 threads, FP32), more
// points at most 128 (512 threads)
__host__ __device__ constexpr int gen_max_threads(int e) { return e <= 16 ? 1024 : 512; }
cudaError_t launch_gen_f32(int kind, bool contiguous, const PassArgs& a, cudaStream_t s);
// Split-precision tensor-core passes (fft_split.cuh): FP32 lines of 256,
// 512, 1024 points, 256-thread CTAs of split_lines_per_cta lines.
bool split_length(int n);
int split_lines_per_cta(int n, bool contiguous);
cudaError_t launch_split_f32(int kind, bool contiguous, const PassArgs& a, cudaStream_t s);
// Lengths whose FP64 lines run in fixed point: up to 2048 points, and 4096,
// whose plan divides by enough on the way.  On longer lines the headroom
// costs more bits than a double's rounding.  rel-L2 against 64 bits over the
// FP64 kernels', 126 lengths, lines of noise, of one modulus, of modes and of 1
// to 256 peaks: c2c and r2c 0.1 to 0.7, c2r 0.15 to 0.92; 4096 points up to 0.9
// but c2r of a few modes, 1.15 (2.5e-16: the first stage's bound is the sum of
// the whole line).
__host__ __device__ constexpr bool fx_length(int n) { return (n >= 2 && n <= 2048) || n == 4096; }

// Shared-memory entries of one power-of-two tile of L lines: the exchange
// buffer, or for c2r the staged half spectra (n/2+1 per real line).
__host__ __device__ constexpr long long fast_smem_entries(int n, int L) {
  // rounded up to an even count: buffers laid end to end stay 16-byte
  // aligned (the c2r staging reads 16-byte pairs)
  return ((long long)(n + 2) * L + (((long long)(n + 2) * L) >> 4) + 2) & ~1ll;
}

cudaError_t launch_fast_f32_c2c(int kind, bool contiguous, const PassArgs& a, cudaStream_t s);
cudaError_t launch_fast_f32_real(int kind, bool contiguous, const PassArgs& a, cudaStream_t s);

// Compile-time plans, one function a kind and layout and group of lengths.
cudaError_t launch_fxc(int kind, bool contiguous, const PassArgs& a, cudaStream_t s);
// Runtime plans of smooth lengths (fft_rt.cuh), FP32 and fixed point.
// threads of a CTA: two CTAs an SM leave 64 registers a thread (FP32), 80
// (fixed point)
__host__ __device__ constexpr int rt_threads(int prec_bytes) { return prec_bytes == 4 ? 512 : 384; }
constexpr int rt_max_radix(int prec_bytes) { return prec_bytes == 4 ? 16 : 10; }
// buffer entries of L lines: a pad entry per 8
__host__ __device__ constexpr size_t rt_entries(int n, int L) { return ((size_t)n + n / 8 + 2) * (size_t)L + 2; }
// one buffer for two stages, two for more (the fixed-point kernel's FP64
// fallback needs two for a single line), and the lines' scale words
__host__ __device__ constexpr size_t rt_smem_bytes(int prec_bytes, int n, int L, int nst) {
  return (nst > 2 || (prec_bytes == 8 && L == 1) ? 2 : 1) * rt_entries(n, L) * (size_t)(2 * prec_bytes) + 32 +
         (prec_bytes == 8 ? (size_t)L * kFxWordBytes : 0);
}
cudaError_t launch_rt_f32(int kind, bool contiguous, const PassArgs& a, cudaStream_t s);
cudaError_t launch_rt_f64(int kind, bool contiguous, const PassArgs& a, cudaStream_t s);
cudaError_t launch_fx(int kind, bool contiguous, const PassArgs& a, cudaStream_t s);

// The x and y passes of one z-plane run by one fused kernel
// (fft_fused.cuh): ax holds the x pass with ax.nlines = complex x lines per
// plane, ay the y pass (ay.nlines = columns, ay.nv = planes).
struct FusedArgs {
  PassArgs ax;
  PassArgs ay;
  long long nplanes;
  int* sync;    // nplanes + 2 ints: ticket, error flag, per-plane counters
  int threads;  // threads per CTA: 256 or 512 (ax.L, ay.L follow from it)
};

// True when a fused x/y kernel exists for these lengths (x first or y
// first, x kind K_C2C / K_R2C / K_C2R).
bool fused_supported(int prec_bytes, int kindx, bool x_first, int nx, int ny);
// Default threads per CTA of the fused kernel (a tile of L = threads / (n / E)
// lines).
constexpr int kFusedThreads = 256;
// Enqueue a fused x/y pass (zeroes f.sync first).
cudaError_t launch_fused(int prec_bytes, int kindx, bool x_first, const FusedArgs& f, cudaStream_t stream);

// ---- batches: every pass of many grids in one persistent launch ----------
constexpr int kBatchThreads = 256;
// Points a thread of the batch kernel's power-of-two plans (lines of 32..256
// points).  16: with 8 (half the points a tile, more tiles resident per SM)
// the 64-grid batch measured 2.45 ms a forward + backward step against 1.94.
__host__ __device__ constexpr int batch_points(int) { return 16; }
struct BatchDesc {
  PassArgs a;       // a.L = tile lines + 1 (shared-memory layout lines)
  int code;         // 2 * kind + (strided ? 1 : 0)
  int dep;          // descriptor that must be complete first, or -1
  long long lines;  // complex lines of the pass (contiguous) or nu * nv (strided)
  long long nu;     // strided: lines along u (x)
};
// Line lengths the batch kernel runs: 32, 48, 64, 96, 128, 192, 256.
bool batch_length(int n);
// Lines one 256-thread tile holds for a length and contiguity.
int batch_tile_lines(int n, bool contiguous);
cudaError_t launch_batch_f32(const BatchDesc* d_desc, const long long* d_prefix, int ndesc, int* d_sync,
                             long long sync_ints, cudaStream_t stream);

// Self-test of the bounded inter-CTA wait: d_words[0] is the counter,
// d_words[1] receives 1 when the wait gave up.
cudaError_t launch_wait_selftest(int* d_words, int need, long long limit, cudaStream_t stream);

// The unfused passes an engine would run for r2c (which = 0) or c2r
// (which = 1) between the given arrays (the engine's pipeline, without
// launching anything).
struct PassInfo {
  PassArgs a;
  int kind;
  bool contiguous;
};
int engine_precision(struct ::gbfft_engine_s* e);
int engine_passes(struct ::gbfft_engine_s* e, int which, const void* in, void* out, PassInfo* out_passes,
                  int max_passes, int* n);

// Shared memory the runtime-planned pass needs for L lines of length n
// (two padded buffers); the power-of-two pass needs half of it.
size_t pass_smem_bytes(int prec_bytes, int n, int L);

// One real-to-real pass along an axis: the window of n points starting at
// point `off` of every line is transformed by kind 1..8 (DCT-I..IV,
// DST-I..IV) through a complex FFT of length M -- of one line's extension
// (dtt.cu), or in fixed point of dtt_fft_length points that carry two real
// lines (one for DCT-IV / DST-IV of an even n; fft_r2r.cuh).
struct DttArgs {
  const void* src;   // real array the window is read from
  void* dst;         // real array it is written to (may be src)
  long long sn;      // element stride between points of a line
  long long sl;      // contiguous: line stride; strided: stride of v
  long long nlines;  // real lines: contiguous all, strided along u (x positions)
  int nv;            // strided: extent of v (grid.y)
  int naxis;         // points on the axis (copied through outside the window)
  int off, n;        // window: first point, length
  int kind;          // 1..8
  int M;             // FFT length
  int nst;           // radix stages of M
  int radix[kMaxStages];
  const void* tw;    // exp(-2 pi i m / M), m < M
  const void* twf;   // FP32, power-of-two or two-stage M: stage-major table of the
                     // compile-time plan, which runs instead of the runtime plan
                     // (null: runtime plan)
  const void* w4;    // exp(-2 pi i m / (4 n)), m < n
  double c0x, c0y;   // exp(-i pi / (4 n))
  const FxPlan* fx;  // FP64: host-side plan of the fixed-point pass, or null; then
  const void* w;     //   the roots of the maps around the FFT, in double
  const void* w_fx;  //   and in Q62
  int pair_vec;      //   strided: the two real lines of a pair are adjacent and
                     //   aligned in both arrays (one access for both)
  int L, tpl;        // transforms a CTA (lines; fixed point: complex lines), threads each
};
// FFT length behind kind 1..8 of an n-point window in fixed point.
__host__ __device__ constexpr int dtt_fft_length(int kind, int n) {
  return kind == 1 ? 2 * (n - 1) : kind == 5 ? 2 * (n + 1) : kind % 4 == 0 && n % 2 == 0 ? n / 2 : n;
}
// Complex lines of a pass: pairs of its real lines, or each alone.
inline long long dtt_complex_lines(const DttArgs& a) {
  return a.kind % 4 == 0 && a.n % 2 == 0 ? a.nlines : (a.nlines + 1) / 2;
}
size_t dtt_smem_bytes(int prec_bytes, int M, int L);
// power-of-two extension lengths with a compile-time plan for the FP32 r2r pass
__host__ __device__ constexpr bool dtt_fast_length(int M) { return M >= 32 && M <= 2048 && (M & (M - 1)) == 0; }
// Extension lengths with the compile-time two-stage plan M = R0 * R1
// (mixed_r0): 126 = 9 * 14 and 510 = 17 * 30, the default windows of every
// kind on axes of 64 and 256 points (FP32).
__host__ __device__ constexpr bool dtt_mixed_length(int M) { return M == 126 || M == 510; }
cudaError_t launch_dtt_pass(int prec_bytes, bool contiguous, const DttArgs& a, cudaStream_t stream);
// ... its fixed-point forms (a.fx), runtime and compile-time plans
cudaError_t launch_fx_r2r(bool contiguous, const DttArgs& a, cudaStream_t stream);
cudaError_t launch_fxc_r2r(bool contiguous, const DttArgs& a, cudaStream_t stream);

// TMA-staged strided c2c passes (fft_tma.cu): FP32 lines of 1024 points
// whose source and destination rows and planes lie multiples of 16 bytes
// apart and start 16-byte aligned, on the axis's own compile-time plan
// (a.tpl = n / 16 or n / 32; the stage-major twiddle table is the axis's).
bool tma_pass_supported(int prec_bytes, int kind, bool contiguous, const PassArgs& a);
cudaError_t launch_tma_pass(const PassArgs& a, cudaStream_t stream);
long long tma_launch_counter();

// Split-precision strided c2c passes of 1024 FP32 points on tcgen05 with
// TMEM accumulators (fft_tc.cu): a.fast == 5, a.tw the n-root table,
// a.status the engine's status word.
bool tc_pass_supported(int prec_bytes, int kind, bool contiguous, const PassArgs& a);
cudaError_t launch_tc_pass(const PassArgs& a, cudaStream_t stream);
long long tc_launch_counter();

// Axis passes whose lines do not fit one shared-memory tile, or whose
// length has a prime factor above kBluePrime (fft_long.cu): one kernel per
// radix stage through `scratch`, which must hold two copies of the pass's
// lines -- of m points each on the chirp-z path (long_pass_scratch_bytes).
// Lines are per row (row_w = 0); a.nst / a.radix are the axis's stages,
// a.tw its n-root table, a.blue the chirp-z tables when set.
size_t long_pass_scratch_bytes(int prec_bytes, bool contiguous, const PassArgs& a);
cudaError_t launch_long_pass(int prec_bytes, int kind, bool contiguous, const PassArgs& a, void* scratch,
                             size_t scratch_bytes, cudaStream_t stream);

// Enqueue one axis pass.  prec_bytes = 4 (float) or 8 (double).
cudaError_t launch_axis_pass(int prec_bytes, int kind, bool contiguous,
                             const PassArgs& a, cudaStream_t stream);

// Enqueue an identity-layout copy of `bytes` bytes (the one-rank transpose).
cudaError_t launch_copy(const void* src, void* dst, size_t bytes,
                        cudaStream_t stream);

// Every device allocation of the library: cudaMalloc, unless a test armed
// gbfft_debug_fail_alloc for this one (then cudaErrorMemoryAllocation,
// nothing allocated).
cudaError_t dev_malloc(void** p, size_t bytes);
// ... and every free of one (counts the live allocations)
cudaError_t dev_free(void* p);

// Record an error message for gbfft_last_error_string(); returns `code`.
int set_error(int code, const char* msg);

// Count of kernels this library has enqueued (for the benchmark's report).
long long launch_counter();
void add_launches(long long n);

}  // namespace gbfft
