// Axis passes of FP64 lines in 64-bit fixed point (fft_fx.cuh), any length a
// tile holds.
//
// What bounds an FP64 pass on GB300 is the FP64 pipe (two multiply-adds an SM
// and clock): a 512-point line costs about 17 SM clocks a point there, four
// times what its DRAM traffic takes and more.  In integers the same line
// costs two to three.
//
// A CTA owns L lines, `tpl` threads each:
//   1. every thread loads its points (at most kE, in registers) and the line's
//      largest high word goes to shared memory;
//   2. the line's sum of moduli, in units of 2^-20 of that, follows; the two
//      give the scale at which no stage's output leaves the word;
//   3. the points become integers in shared buffer 0, a mean taken off (c2r:
//      the Hermitian combination of the two half spectra but for their bins 0);
//   4. Stockham stages ping-pong between the two buffers, twiddles from a
//      stage-major Q62 table;
//   5. the result goes back to doubles (r2c: the two half spectra apart),
//      rounded once, to nearest.
// A CTA that meets a NaN, an infinity or a line outside the exponents of
// fx::kMinExp..kMaxExp runs its lines in FP64 instead (fx::fallback), on the
// general kernel's stages: 256^3 r2c + c2r 3.5 ms, in fixed point 0.5 (64^3: 154
// and 28 us).
#include "fft_fx.cuh"
#include "fft_r2r.cuh"

namespace gbfft {

namespace {

using namespace dev;
using fx::I2;
using fx::ll;
using fx::W4;

constexpr int kE = kFxPoints;

// down: the powers of two that a stage's twiddles divide by, 1, or 2 after a
// radix of 8 or more (1 throughout left c2r of 2023 = 17 17 7 points 1.1 times
// the FP64 kernels' error).  dc: what joins every output of the line, or null.
template <int R, class Ctx>
__device__ __forceinline__ void fx_stage(const Ctx& c, const I2* A, I2* B, const W4* __restrict__ tw, int Ns,
                                         unsigned magic, int down, const I2* dc) {
  const int nb = c.N / R;
#pragma unroll 1
  for (int b = c.t; b < nb; b += c.tpl) {
    I2 v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = A[c.sidx(b + r * nb)];
    int k = 0;
    if (Ns > 1) {
      k = b - (int)__umulhi((unsigned)b, magic) * Ns;
      const W4* w = tw + (Ns - 1) + k;
      v[0] = fx::mk(fx::scale_down(v[0].x, down), fx::scale_down(v[0].y, down));
#pragma unroll
      for (int r = 1; r < R; ++r) v[r] = fx::mul_tw(v[r], fx::ldw(w + (r - 1) * Ns), r, down);
    }
    if (dc) v[0] = fx::add(v[0], *dc);
    const int base = (b - k) * R + k;
    if constexpr (R > 5 && R % 2 == 1 && R % 3 != 0) {
      fx::dft_odd<R>(v, [&](int m, I2 x) { B[c.sidx(base + m * Ns)] = x; });
    } else {
      fx::dft<R>(v);
#pragma unroll
      for (int r = 0; r < R; ++r) B[c.sidx(base + r * Ns)] = v[r];
    }
  }
}

// Any other prime: every output a direct sum over R inputs, a quarter of each.
// (Halves left c2r of a single peak less accurate than FP64 where two such
// stages follow each other: 2047 points rel-L2 4.3e-16, FP64 3.1e-16.)
template <class Ctx>
__device__ void fx_stage_generic(const Ctx& c, const I2* A, I2* B, const W4* __restrict__ root, int R, int Ns,
                                 const I2* dc) {
  const int N = c.N, nb = N / R, tstride = N / (Ns * R);
#pragma unroll 1
  for (int o = c.t; o < N; o += c.tpl) {
    const int k = o % Ns, r = (o / Ns) % R, b = o / (Ns * R) * Ns + k;
    const int step = (k * tstride + r * nb) % N;
    I2 acc = dc ? *dc : fx::mk(0, 0);
    int e = 0;
#pragma unroll 1
    for (int j = 0; j < R; ++j) {
      acc = fx::add(acc, fx::mul_tw<2>(A[c.sidx(b + j * nb)], fx::ldw(root + e), j));
      e += step;
      if (e >= N) e -= N;
    }
    B[c.sidx(o)] = acc;
  }
}

// The stages of a plan on the lines in A, ping-ponging with B; returns the
// buffer that holds the result.  dc: see fx_stage, in the last stage.
template <class Ctx>
__device__ __forceinline__ const I2* fx_stages(const Ctx& c, const FxPlan& p, I2* first, I2* second,
                                               const I2* dc = nullptr) {
  const I2* A = first;
  I2* B = second;
  const W4* tw = reinterpret_cast<const W4*>(p.tw);
#pragma unroll 1
  for (int s = 0; s < p.nst; ++s) {
    const int R = p.radix[s], Ns = p.ns[s];
    const unsigned mg = p.magic[s];
    const int down = s > 0 ? p.shift[s] - p.shift[s - 1] : 0;
    const I2* const add = s == p.nst - 1 ? dc : nullptr;
    switch (R) {
      case 2: fx_stage<2>(c, A, B, tw, Ns, mg, down, add); break;
      case 3: fx_stage<3>(c, A, B, tw, Ns, mg, down, add); break;
      case 4: fx_stage<4>(c, A, B, tw, Ns, mg, down, add); break;
      case 5: fx_stage<5>(c, A, B, tw, Ns, mg, down, add); break;
      case 6: fx_stage<6>(c, A, B, tw, Ns, mg, down, add); break;
      case 7: fx_stage<7>(c, A, B, tw, Ns, mg, down, add); break;
      case 8: fx_stage<8>(c, A, B, tw, Ns, mg, down, add); break;
      case 9: fx_stage<9>(c, A, B, tw, Ns, mg, down, add); break;
      case 10: fx_stage<10>(c, A, B, tw, Ns, mg, down, add); break;
      case 11: fx_stage<11>(c, A, B, tw, Ns, mg, down, add); break;
      case 13: fx_stage<13>(c, A, B, tw, Ns, mg, down, add); break;
      case 17: fx_stage<17>(c, A, B, tw, Ns, mg, down, add); break;
      default: fx_stage_generic(c, A, B, reinterpret_cast<const W4*>(p.root), R, Ns, add); break;
    }
    __syncthreads();
    I2* const done = B;
    B = const_cast<I2*>(A);
    A = done;
  }
  return A;
}

template <int KIND, bool CONTIG>
__global__ void __launch_bounds__(kFxMaxThreads) fx_pass_kernel(const __grid_constant__ PassArgs a,
                                                                const __grid_constant__ FxPlan p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  chained_entry();
  LineCtx<double, KIND, CONTIG> c;
  c.init(a);
  const int N = c.N, tpl = c.tpl, t = c.t;
  const int e = N * a.L;
  I2* buf0 = reinterpret_cast<I2*>(smem_raw);
  I2* buf1 = buf0 + (e + (e >> 4) + 1);
  const fx::Words words(smem_raw + fx_smem_bytes(N, a.L), a.L);
  words.clear(a.L);
  __syncthreads();

  // c2r: two half spectra of N / 2 + 1 points, point j of both in v[2 i], v[2 i + 1]
  constexpr int J = KIND == K_C2R ? kE / 2 + 1 : kE;
  constexpr int W = KIND == K_C2R ? 2 : 1;
  const int cnt = KIND == K_C2R ? N / 2 + 1 : N;
  double2 v[J * W];
#pragma unroll
  for (int i = 0; i < J; ++i) {
    const int n = t + i * tpl;
    if constexpr (KIND == K_C2R) {
      v[2 * i] = n < cnt ? c.half(0, n) : make_double2(0, 0);
      v[2 * i + 1] = n < cnt ? c.half(1, n) : make_double2(0, 0);
      if (n == 0) {  // bins 0 apart, their Im ignored
        words.ref[c.line] = make_double2(v[0].x, v[1].x);
        v[0] = v[1] = make_double2(0, 0);
      }
      if (2 * n == N) v[2 * i].y = v[2 * i + 1].y = 0;  // Im of the Nyquist bin is ignored
    } else {
      v[i] = n < cnt ? c.gload_raw(n) : make_double2(0, 0);
    }
  }
  fx::PassScale<KIND> sc;
  if (!sc.find(v, words, c.line, t == 0, [&](int i) { return t + i * tpl < cnt; })) {
    fx::fallback<KIND, CONTIG>(a, reinterpret_cast<double2*>(smem_raw));
    return;
  }
#pragma unroll 1
  for (int s = 0; s < p.nst; ++s) sc.stage(p.lg[s], p.shift[s], s == p.nst - 1);
  // r2c adds two values that no twiddle has halved
  if (KIND == K_R2C && p.shift[p.nst - 1] == 0) sc.headroom();
  const int sa = sc.shift_a(), sb = sc.shift_b();
  // backward: conjugated on the way in (c2r: by its combination) and out
  const int flip = c.inverse ? (int)0x80000000 : 0;
  const fx::Back<KIND> out = sc.back(p.shift[p.nst - 1], flip);

  if constexpr (KIND == K_C2R) {
    if (t == 0) sc.set_dc(words, c.line, p.shift[p.nst - 1]);
#pragma unroll
    for (int i = 0; i < J; ++i) {
      const int j = t + i * tpl;
      if (j < cnt) {
        const ll ax = fx::to_fixed(v[2 * i].x, sa), ay = fx::to_fixed(v[2 * i].y, sa);
        const ll bx = fx::to_fixed(v[2 * i + 1].x, sb), by = fx::to_fixed(v[2 * i + 1].y, sb);
        // z = x1 + i x2, conjugated for the inverse-by-conjugation
        buf0[c.sidx(j)] = fx::mk(ax - by, -(ay + bx));
        if (j > 0 && 2 * j < N) buf0[c.sidx(N - j)] = fx::mk(ax + by, ay - bx);
      }
    }
  } else {
#pragma unroll
    for (int i = 0; i < J; ++i) {
      const int n = t + i * tpl;
      if (n < N) buf0[c.sidx(n)] = fx::mk(fx::to_fixed(v[i].x, sa), fx::to_fixed(v[i].y, sb, flip));
    }
  }
  __syncthreads();

  const I2* A =
      fx_stages(c, p, buf0, buf1, KIND == K_C2R ? reinterpret_cast<const I2*>(&words.ref[c.line]) : nullptr);

  if constexpr (KIND == K_R2C) {
#pragma unroll 1
    for (int k = t; 2 * k <= N; k += tpl) {
      const I2 zk = A[c.sidx(k)], zm = A[c.sidx(k == 0 ? 0 : N - k)];
      double2 xa = out.half_a(zk, zm), xb = out.half_b(zk, zm);
      if (out.off && k == 0) out.dc(xa, xb, N);
      c.put_half(0, k, xa);
      c.put_half(1, k, xb);
    }
  } else {
#pragma unroll 1
    for (int n = t; n < N; n += tpl) {
      double2 z = out.point(A[c.sidx(n)]);
      if (KIND == K_C2C && out.off && n == 0) out.dc(z, N);
      c.gstore_raw(n, z);
    }
  }
}

template <int KIND, bool CONTIG>
cudaError_t launch_k(const PassArgs& a, cudaStream_t stream) {
  const FxPlan& p = *a.fx;
  const size_t smem = fx_smem_bytes(a.n, a.L);
  if (a.L < 1 || a.tpl < 1 || a.L * a.tpl > kFxMaxThreads || a.tpl * kE < a.n || smem > kFxMaxSmem)
    return cudaErrorInvalidValue;
  auto kern = fx_pass_kernel<KIND, CONTIG>;
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  const dim3 block = CONTIG ? dim3(a.tpl, a.L) : dim3(a.L, a.tpl);
  const dim3 grid((unsigned)((a.nlines + a.L - 1) / a.L), CONTIG ? 1u : (unsigned)a.nv);
  const cudaError_t err = launch_chained(kern, grid, block, smem, stream, a, p);
  add_launches(1);
  return err != cudaSuccess ? err : cudaGetLastError();
}

// A real-to-real pass (fft_r2r.cuh) in the same arithmetic.
template <bool CONTIG>
__global__ void __launch_bounds__(kFxMaxThreads) fx_r2r_kernel(const __grid_constant__ DttArgs a,
                                                              const __grid_constant__ FxPlan p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  chained_entry();
  LineCtx<double, K_C2C, CONTIG> c;
  c.N = a.M;
  c.L = a.L;
  c.tpl = a.tpl;
  c.t = CONTIG ? threadIdx.x : threadIdx.y;
  c.line = CONTIG ? threadIdx.y : threadIdx.x;
  const r2r::Lines<double, CONTIG> ln(a, (long long)blockIdx.x * a.L + c.line, CONTIG ? 0 : (long long)blockIdx.y);
  const int e = a.M * a.L, t = c.t, tpl = c.tpl, cnt = r2r::elements(a.kind, a.n);
  I2* buf0 = reinterpret_cast<I2*>(smem_raw);
  I2* buf1 = buf0 + (e + (e >> 4) + 1);
  const fx::Words words(smem_raw + fx_smem_bytes(a.M, a.L), a.L);
  words.clear(a.L);
  __syncthreads();
  double2 x[kE];
#pragma unroll
  for (int i = 0; i < kE; ++i) {
    const int j = t + i * tpl;
    x[i] = j < cnt ? ln.element(j) : make_double2(0, 0);
  }
  fx::PairScale sc;
  int* const wm = words.m + 2 * c.line;
  unsigned* const ws = words.s + 2 * c.line;
  fx::Found found = sc.find<false, true>(x, wm, ws, ln.single, r2r::keeps_mean(a.kind));
  const bool off = found == fx::Found::flat;
  if (__builtin_expect(off, 0)) {
    fx::take_means(x, words, c.line, t == 0, [&](int i) { return t + i * tpl < cnt; });
    found = sc.find<false, false>(x, wm, ws, ln.single);
  }
  if (found != fx::Found::yes) {
    r2r::fallback<CONTIG>(a, reinterpret_cast<double2*>(smem_raw));
    return;
  }
  using Map = r2r::Maps<r2r::Fixed, r2r::CtxSlot<LineCtx<double, K_C2C, CONTIG>>>;
  const Map mp{a.kind, a.n, a.M, reinterpret_cast<const W4*>(a.w_fx), {&c}};
  const int g = mp.grow(), pre = mp.pre(), last = p.nst - 1;
  int ta = -1021 + g, tb = ta;
#pragma unroll 1
  for (int s = 0; s <= last; ++s) {
    const int down = pre + p.shift[s] - (s == last ? mp.post() : 0);
    ta = max(ta, sc.a.bound(p.lg[s], g) - down);
    tb = max(tb, sc.b.bound(p.lg[s], g) - down);
  }
  const int sa = sc.a.shift(ta), sb = sc.b.shift(tb);
  const int down = pre + p.shift[last] + mp.tail() + Map::doubled(a.kind, a.n) - 62;
  const int adj_a = (sc.a.em + ta + down) << 20, adj_b = (sc.b.em + tb + down) << 20;
#pragma unroll
  for (int i = 0; i < kE; ++i) {
    const int j = t + i * tpl;
    if (j < cnt) mp.place(buf0, j, fx::mk(fx::to_fixed(x[i].x, sa), fx::to_fixed(x[i].y, sb)));
  }
  __syncthreads();
  if (mp.combines()) {
#pragma unroll 1
    for (int k = t; 2 * k <= a.n; k += tpl) mp.combine(buf0, k);
    __syncthreads();
  }
  const I2* A = fx_stages(c, p, buf0, buf1);
#pragma unroll 1
  for (int k = t; k < mp.steps(); k += tpl)
    mp.finish(
        A, k, [&](int i, ll ya, ll yb) { ln.store(i, sc.a.out(ya, adj_a), sc.b.out(yb, adj_b)); },
        [&](int i, ll y) { ln.store1(i, sc.a.out(y, adj_a)); });
  if (off && t == 0) ln.add_mean(words.ref[c.line]);
  ln.pass_through(a.naxis, t, tpl);
}

template <bool CONTIG>
cudaError_t launch_r2r_k(const DttArgs& a, cudaStream_t stream) {
  const size_t smem = fx_smem_bytes(a.M, a.L);
  if (a.L < 1 || a.tpl < 1 || a.L * a.tpl > kFxMaxThreads || a.tpl * kE < a.M || smem > kFxMaxSmem)
    return cudaErrorInvalidValue;
  auto kern = fx_r2r_kernel<CONTIG>;
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  const long long lines = dtt_complex_lines(a);
  const dim3 block = CONTIG ? dim3(a.tpl, a.L) : dim3(a.L, a.tpl);
  const dim3 grid((unsigned)((lines + a.L - 1) / a.L), CONTIG ? 1u : (unsigned)a.nv);
  const cudaError_t err = launch_chained(kern, grid, block, smem, stream, a, *a.fx);
  add_launches(1);
  return err != cudaSuccess ? err : cudaGetLastError();
}

}  // namespace

cudaError_t launch_fx_r2r(bool contiguous, const DttArgs& a, cudaStream_t s) {
  return contiguous ? launch_r2r_k<true>(a, s) : launch_r2r_k<false>(a, s);
}

cudaError_t launch_fx(int kind, bool contiguous, const PassArgs& a, cudaStream_t s) {
  if (kind == K_C2C) return contiguous ? launch_k<K_C2C, true>(a, s) : launch_k<K_C2C, false>(a, s);
  if (kind == K_R2C) return contiguous ? launch_k<K_R2C, true>(a, s) : launch_k<K_R2C, false>(a, s);
  if (kind == K_C2R) return contiguous ? launch_k<K_C2R, true>(a, s) : launch_k<K_C2R, false>(a, s);
  return cudaErrorInvalidValue;
}

}  // namespace gbfft
