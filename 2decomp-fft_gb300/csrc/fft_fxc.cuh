// Fixed-point axis passes of FP64 lines (fft_fx.cuh) with compile-time plans:
// the arithmetic and the scale of fft_fx.cu for the common lengths, with the
// points in registers and one exchange buffer.
//
// What bounds the runtime-planned kernel is the integer and address
// instructions it issues (390 a point at 512 points, 2.1 a clock and SM with
// 16 warps).  With the length known the slots and strides fold into the
// instructions, the first stage starts from the loaded registers, the last
// one stores from them, and half the shared memory and registers a thread
// leave room for more warps.
#pragma once

#include "fft_fx.cuh"
#include "fft_r2r.cuh"

namespace gbfft {
namespace fx {

using namespace dev;

// n = R0 R1 R2 R3 in that order; TPL threads a line, each with butterflies
// t, t + TPL, ... of a stage.
template <int N_, int TPL_, int R0, int R1 = 1, int R2 = 1, int R3 = 1>
struct Plan {
  static constexpr int N = N_, TPL = TPL_;
  static constexpr int NST = R3 > 1 ? 4 : R2 > 1 ? 3 : R1 > 1 ? 2 : 1;
  __host__ __device__ static constexpr int radix(int s) { return s == 0 ? R0 : s == 1 ? R1 : s == 2 ? R2 : R3; }
  __host__ __device__ static constexpr int ns(int s) {
    int v = 1;
    for (int i = 0; i < s; ++i) v *= radix(i);
    return v;
  }
  __host__ __device__ static constexpr int mb(int s) { return (N / radix(s) + TPL - 1) / TPL; }
  __host__ __device__ static constexpr int points() {
    int e = 0;
    for (int s = 0; s < NST; ++s)
      if (mb(s) * radix(s) > e) e = mb(s) * radix(s);
    return e;
  }
  // powers of two that stage s divides its inputs by (its twiddles do)
  __host__ __device__ static constexpr int sh(int s) { return s == 0 ? 0 : radix(s - 1) >= 8 ? 2 : 1; }
  __host__ __device__ static constexpr int shift(int s) {
    int v = 0;
    for (int i = 0; i <= s; ++i) v += sh(i);
    return v;
  }
  __host__ __device__ static constexpr int lg(int s) {
    int l = 0;
    while ((1 << l) < ns(s + 1)) ++l;
    return l;
  }
  static_assert(R0 * R1 * R2 * R3 == N_, "radices");
};

// Exchange slots: contiguous lines padded by one entry in eight (a quarter
// warp's 16-byte accesses cover the banks once), strided tiles dense (the
// lanes walk the lines).
template <class P, bool CONTIG>
struct Slots {
  static constexpr int kLine = P::N + P::N / 8 + 1;
  int base, L;
  __device__ __forceinline__ int operator()(int n) const { return CONTIG ? base + n + (n >> 3) : n * L + base; }
};

// Global accesses of a thread's points t + n, n known at compile time: one
// multiply-add an address (the row strides are below 2^32 bytes).
template <int KIND, bool CONTIG>
struct Io {
  const LineCtx<double, KIND, CONTIG>& c;
  const char *s0, *s1;
  char *d0, *d1;
  unsigned ss, ds;
  __device__ __forceinline__ explicit Io(const LineCtx<double, KIND, CONTIG>& ctx) : c(ctx) {
    constexpr int SB = KIND == K_R2C ? 8 : 16, DB = KIND == K_C2R ? 8 : 16;
    ss = (unsigned)c.ssn * SB;
    ds = (unsigned)c.dsn * DB;
    s0 = reinterpret_cast<const char*>(c.src) + c.sb0 * SB + (unsigned long long)ss * (unsigned)c.t;
    s1 = reinterpret_cast<const char*>(c.src) + c.sb1 * SB + (unsigned long long)ss * (unsigned)c.t;
    d0 = reinterpret_cast<char*>(c.dst) + c.db0 * DB + (unsigned long long)ds * (unsigned)c.t;
    d1 = reinterpret_cast<char*>(c.dst) + c.db1 * DB + (unsigned long long)ds * (unsigned)c.t;
  }
#ifdef GB_DEBUG_BOUNDS
  __device__ __forceinline__ double2 load(int n) const { return c.gload_raw(c.t + n); }
  __device__ __forceinline__ double2 half(int which, int n) const { return c.half(which, c.t + n); }
  __device__ __forceinline__ void store(int n, double2 v) const { c.gstore_raw(c.t + n, v); }
  __device__ __forceinline__ void put_half(int which, int n, double2 v) const { c.put_half(which, c.t + n, v); }
#else
  __device__ __forceinline__ unsigned long long so(int n) const { return (unsigned long long)(unsigned)n * ss; }
  __device__ __forceinline__ unsigned long long dof(int n) const { return (unsigned long long)(unsigned)n * ds; }
  __device__ __forceinline__ double2 load(int n) const {
    if (!c.valid) return make_double2(0, 0);
    if (KIND == K_C2C || (!CONTIG && c.pvec && c.has1)) return *reinterpret_cast<const double2*>(s0 + so(n));
    return make_double2(*reinterpret_cast<const double*>(s0 + so(n)),
                        c.has1 ? *reinterpret_cast<const double*>(s1 + so(n)) : 0.0);
  }
  __device__ __forceinline__ double2 half(int which, int n) const {
    if (!c.valid || (which && !c.has1)) return make_double2(0, 0);
    return *reinterpret_cast<const double2*>((which ? s1 : s0) + so(n));
  }
  __device__ __forceinline__ void store(int n, double2 v) const {
    if (!c.valid) return;
    if (KIND == K_C2C || (!CONTIG && c.pvec && c.has1)) {
      *reinterpret_cast<double2*>(d0 + dof(n)) = v;
      return;
    }
    *reinterpret_cast<double*>(d0 + dof(n)) = v.x;
    if (c.has1) *reinterpret_cast<double*>(d1 + dof(n)) = v.y;
  }
  __device__ __forceinline__ void put_half(int which, int n, double2 v) const {
    if (c.valid && (!which || c.has1)) *reinterpret_cast<double2*>((which ? d1 : d0) + dof(n)) = v;
  }
#endif
};

// The stages from S on.  KIND K_R2C: the last one leaves its outputs in Sm.
template <class P, int S, bool FROM_SMEM, int KIND, bool CONTIG, class Out, class Bk>
__device__ __forceinline__ void run(const Out& io, int t, I2* Sm, const Slots<P, CONTIG>& slot, const W4* __restrict__ tw,
                                    I2 (&v)[P::points()], const Bk& back, const I2* dc = nullptr) {
  constexpr int R = P::radix(S), NS = P::ns(S), NB = P::N / R, MB = P::mb(S), TPL = P::TPL;
  constexpr bool LAST = S == P::NST - 1;
  if constexpr (FROM_SMEM) {
#pragma unroll
    for (int m = 0; m < MB; ++m) {
      const int b = t + m * TPL;
      if ((NB % TPL != 0 && b >= NB)) break;
#pragma unroll
      for (int r = 0; r < R; ++r) v[m * R + r] = Sm[slot(b + r * NB)];
    }
  }
#pragma unroll
  for (int m = 0; m < MB; ++m) {
    const int b = t + m * TPL;
    if ((NB % TPL != 0 && b >= NB)) break;
    if constexpr (NS > 1) {
      const W4* w = tw + (NS - 1) + b % NS;
      constexpr int SH = P::sh(S);
      v[m * R] = mk(scale_down<SH>(v[m * R].x), scale_down<SH>(v[m * R].y));
#pragma unroll
      for (int r = 1; r < R; ++r) v[m * R + r] = mul_tw<SH>(v[m * R + r], ldw(w + (r - 1) * NS), r);
    }
    if constexpr (LAST && KIND == K_C2R) v[m * R] = add(v[m * R], *dc);
    dft<R>(&v[m * R]);
  }
  if constexpr (LAST && KIND != K_R2C) {
#pragma unroll
    for (int m = 0; m < MB; ++m) {
      const int b = t + m * TPL;
      if ((NB % TPL != 0 && b >= NB)) break;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        double2 z = back.point(v[m * R + r]);
        if (KIND == K_C2C && m == 0 && r == 0 && back.off && t == 0) back.dc(z, P::N);
        io.store(m * TPL + r * NS, z);
      }
    }
  } else {
    if constexpr (FROM_SMEM) __syncthreads();  // every point read before the outputs overwrite them
#pragma unroll
    for (int m = 0; m < MB; ++m) {
      const int b = t + m * TPL;
      if ((NB % TPL != 0 && b >= NB)) break;
      const int k = b % NS, base = (b - k) * R + k;
#pragma unroll
      for (int r = 0; r < R; ++r) Sm[slot(base + r * NS)] = v[m * R + r];
    }
    __syncthreads();
    if constexpr (!LAST) run<P, S + 1, true, KIND, CONTIG>(io, t, Sm, slot, tw, v, back, dc);
  }
}

// CTAs an SM the register budget aims at: 64 registers a thread for at most
// ten points a thread (32 warps; 80 registers and 24 measured 15 % slower),
// 128 for more.
template <class P>
__host__ __device__ constexpr int min_ctas() {
  return 65536 / fxc_max_threads(P::TPL) / (P::points() > 10 ? 128 : 64);
}
template <class P, int KIND, bool CONTIG>
__global__ void __launch_bounds__(fxc_max_threads(P::TPL), min_ctas<P>())
    fxc_pass_kernel(const __grid_constant__ PassArgs a, const W4* __restrict__ tw) {
  constexpr int N = P::N, TPL = P::TPL, E = P::points();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  chained_entry();
  LineCtx<double, KIND, CONTIG> c;
  c.init(a);
  const Io<KIND, CONTIG> io(c);
  const int t = c.t, L = a.L;
  I2* Sm = reinterpret_cast<I2*>(smem_raw);
  Slots<P, CONTIG> slot;
  slot.base = CONTIG ? c.line * Slots<P, CONTIG>::kLine : c.line;
  slot.L = L;
  const Words words(smem_raw + fxc_smem_bytes(N, L), L);
  words.clear(L);
  __syncthreads();

  // 1. load: c2r both half spectra (point j in x[2 i], x[2 i + 1]), else the
  // points of the first stage's butterflies
  constexpr int H = N / 2 + 1, J = KIND == K_C2R ? (H + TPL - 1) / TPL : 1;
  constexpr int R0 = P::radix(0), NB0 = N / R0, MB0 = P::mb(0);
  constexpr int Q = KIND == K_C2R ? 2 * J : MB0 * R0;
  double2 x[Q];
  if constexpr (KIND == K_C2R) {
#pragma unroll
    for (int i = 0; i < J; ++i) {
      const int j = t + i * TPL;
      x[2 * i] = j < H ? io.half(0, i * TPL) : make_double2(0, 0);
      x[2 * i + 1] = j < H ? io.half(1, i * TPL) : make_double2(0, 0);
      if (j == 0) {  // bins 0 apart, their Im ignored
        words.ref[c.line] = make_double2(x[0].x, x[1].x);
        x[0] = x[1] = make_double2(0, 0);
      }
      if (2 * j == N) x[2 * i].y = x[2 * i + 1].y = 0;  // Im of the Nyquist bin is ignored
    }
  } else {
#pragma unroll
    for (int m = 0; m < MB0; ++m) {
      const int b = t + m * TPL;
      const bool in = NB0 % TPL == 0 || b < NB0;
#pragma unroll
      for (int r = 0; r < R0; ++r) x[m * R0 + r] = in ? io.load(m * TPL + r * NB0) : make_double2(0, 0);
    }
  }
  // 2. the line's scale
  PassScale<KIND> sc;
  if (!sc.find(x, words, c.line, t == 0, [&](int i) { return NB0 % TPL == 0 || t + i / R0 * TPL < NB0; })) {
    fallback<KIND, CONTIG>(a, reinterpret_cast<double2*>(smem_raw));
    return;
  }
#pragma unroll
  for (int s = 0; s < P::NST; ++s) sc.stage(P::lg(s), P::shift(s), s == P::NST - 1);
  // r2c adds two values that no twiddle has halved
  if (KIND == K_R2C && P::NST == 1) sc.headroom();
  const int sa = sc.shift_a(), sb = sc.shift_b();
  // backward c2c: conjugated on the way in and out (c2r: out)
  const int flip_in = KIND == K_C2C && c.inverse ? (int)0x80000000 : 0;
  const Back<KIND> back = sc.back(P::shift(P::NST - 1), KIND == K_C2R ? (int)0x80000000 : flip_in);
  // 3. integers, and the stages
  I2 v[E];
  if constexpr (KIND == K_C2R) {
    if (t == 0) sc.set_dc(words, c.line, P::shift(P::NST - 1));
#pragma unroll
    for (int i = 0; i < J; ++i) {
      const int j = t + i * TPL;
      if (j < H) {
        const ll ax = to_fixed(x[2 * i].x, sa), ay = to_fixed(x[2 * i].y, sa);
        const ll bx = to_fixed(x[2 * i + 1].x, sb), by = to_fixed(x[2 * i + 1].y, sb);
        // z = x1 + i x2, conjugated for the inverse-by-conjugation
        Sm[slot(j)] = mk(ax - by, -(ay + bx));
        if (j > 0 && 2 * j < N) Sm[slot(N - j)] = mk(ax + by, ay - bx);
      }
    }
    __syncthreads();
  } else {
#pragma unroll
    for (int i = 0; i < Q; ++i) v[i] = mk(to_fixed(x[i].x, sa), to_fixed(x[i].y, sb, flip_in));
  }
  run<P, 0, KIND == K_C2R, KIND, CONTIG>(io, t, Sm, slot, tw, v, back, reinterpret_cast<const I2*>(&words.ref[c.line]));
  if constexpr (KIND == K_R2C) {
    constexpr int K = (H + TPL - 1) / TPL;
#pragma unroll
    for (int i = 0; i < K; ++i) {
      const int k = t + i * TPL;
      if (k < H) {
        const I2 zk = Sm[slot(k)], zm = Sm[slot(k == 0 ? 0 : N - k)];
        double2 xa = back.half_a(zk, zm), xb = back.half_b(zk, zm);
        if (i == 0 && back.off && t == 0) back.dc(xa, xb, N);
        io.put_half(0, i * TPL, xa);
        io.put_half(1, i * TPL, xb);
      }
    }
  }
}

// A real-to-real pass (fft_r2r.cuh) around a compile-time plan of its FFT.
template <class P, bool CONTIG>
__global__ void __launch_bounds__(fxc_max_threads(P::TPL), min_ctas<P>())
    fxc_r2r_kernel(const __grid_constant__ DttArgs a, const W4* __restrict__ tw) {
  constexpr int N = P::N, TPL = P::TPL, Q = (N + TPL - 1) / TPL;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  chained_entry();
  const int t = CONTIG ? threadIdx.x : threadIdx.y, line = CONTIG ? threadIdx.y : threadIdx.x, L = a.L;
  const r2r::Lines<double, CONTIG> ln(a, (long long)blockIdx.x * L + line, CONTIG ? 0 : (long long)blockIdx.y);
  I2* Sm = reinterpret_cast<I2*>(smem_raw);
  Slots<P, CONTIG> slot;
  slot.base = CONTIG ? line * Slots<P, CONTIG>::kLine : line;
  slot.L = L;
  const Words words(smem_raw + fxc_smem_bytes(N, L), L);
  words.clear(L);
  __syncthreads();
  const int cnt = r2r::elements(a.kind, a.n);
  double2 x[Q];
#pragma unroll
  for (int i = 0; i < Q; ++i) {
    const int j = t + i * TPL;
    x[i] = j < cnt ? ln.element(j) : make_double2(0, 0);
  }
  PairScale sc;
  int* const wm = words.m + 2 * line;
  unsigned* const ws = words.s + 2 * line;
  Found found = sc.find<false, true>(x, wm, ws, ln.single, r2r::keeps_mean(a.kind));
  const bool off = found == Found::flat;
  if (__builtin_expect(off, 0)) {
    take_means(x, words, line, t == 0, [&](int i) { return t + i * TPL < cnt; });
    found = sc.find<false, false>(x, wm, ws, ln.single);
  }
  if (found != Found::yes) {
    r2r::fallback<CONTIG>(a, reinterpret_cast<double2*>(smem_raw));
    return;
  }
  using Map = r2r::Maps<r2r::Fixed, Slots<P, CONTIG>>;
  const Map mp{a.kind, a.n, N, reinterpret_cast<const W4*>(a.w_fx), slot};
  const int g = mp.grow(), pre = mp.pre();
  int ta = -1021 + g, tb = ta;
#pragma unroll
  for (int s = 0; s < P::NST; ++s) {
    const int down = pre + P::shift(s) - (s == P::NST - 1 ? mp.post() : 0);
    ta = max(ta, sc.a.bound(P::lg(s), g) - down);
    tb = max(tb, sc.b.bound(P::lg(s), g) - down);
  }
  const int sa = sc.a.shift(ta), sb = sc.b.shift(tb);
  const int down = pre + P::shift(P::NST - 1) + mp.tail() + Map::doubled(a.kind, a.n) - 62;
  const int adj_a = (sc.a.em + ta + down) << 20, adj_b = (sc.b.em + tb + down) << 20;
#pragma unroll
  for (int i = 0; i < Q; ++i) {
    const int j = t + i * TPL;
    if (j < cnt) mp.place(Sm, j, mk(to_fixed(x[i].x, sa), to_fixed(x[i].y, sb)));
  }
  __syncthreads();
  if (mp.combines()) {
#pragma unroll 1
    for (int k = t; 2 * k <= a.n; k += TPL) mp.combine(Sm, k);
    __syncthreads();
  }
  I2 v[P::points()];
  run<P, 0, true, K_R2C, CONTIG>(ln, t, Sm, slot, tw, v, 0);
#pragma unroll 1
  for (int k = t; k < mp.steps(); k += TPL)
    mp.finish(
        Sm, k, [&](int i, ll ya, ll yb) { ln.store(i, sc.a.out(ya, adj_a), sc.b.out(yb, adj_b)); },
        [&](int i, ll y) { ln.store1(i, sc.a.out(y, adj_a)); });
  if (off && t == 0) ln.add_mean(words.ref[line]);
  ln.pass_through(a.naxis, t, TPL);
}

template <class P, bool CONTIG>
cudaError_t launch_r2r_p(const DttArgs& a, cudaStream_t stream) {
  const size_t smem = fxc_smem_bytes(P::N, a.L);
  if (a.tpl != P::TPL || a.L < 1 || a.L * a.tpl > fxc_max_threads(P::TPL) || smem > kFxMaxSmem)
    return cudaErrorInvalidValue;
  auto kern = fxc_r2r_kernel<P, CONTIG>;
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  const long long lines = dtt_complex_lines(a);
  const dim3 block = CONTIG ? dim3(a.tpl, a.L) : dim3(a.L, a.tpl);
  const dim3 grid((unsigned)((lines + a.L - 1) / a.L), CONTIG ? 1u : (unsigned)a.nv);
  const cudaError_t err = launch_chained(kern, grid, block, smem, stream, a, reinterpret_cast<const W4*>(a.fx->tw));
  add_launches(1);
  return err != cudaSuccess ? err : cudaGetLastError();
}

template <class P, int KIND, bool CONTIG>
cudaError_t launch_p(const PassArgs& a, cudaStream_t stream) {
  const size_t smem = fxc_smem_bytes(P::N, a.L);
  if (a.tpl != P::TPL || a.L < 1 || a.L * a.tpl > fxc_max_threads(P::TPL) || smem > kFxMaxSmem) return cudaErrorInvalidValue;
  auto kern = fxc_pass_kernel<P, KIND, CONTIG>;
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  const dim3 block = CONTIG ? dim3(a.tpl, a.L) : dim3(a.L, a.tpl);
  const dim3 grid((unsigned)((a.nlines + a.L - 1) / a.L), CONTIG ? 1u : (unsigned)a.nv);
  const cudaError_t err = launch_chained(kern, grid, block, smem, stream, a, reinterpret_cast<const W4*>(a.fx->tw));
  add_launches(1);
  return err != cudaSuccess ? err : cudaGetLastError();
}

}  // namespace fx
}  // namespace gbfft
