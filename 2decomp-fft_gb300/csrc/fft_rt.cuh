// Runtime-planned axis passes of smooth lengths, one kernel for FP32 and for
// FP64 in fixed point: radices of at most 16 (fixed point: 10), the first
// stage on the points as they are loaded, the last one stored from its
// registers, twiddles from a stage-major table.
//
// The general runtime kernels (fft_axis.cu, fft_fx.cu) load the lines into
// shared memory, run every prime or power-of-two stage from one buffer to
// another with the divisions and 64-bit addresses of arbitrary lengths, and
// store from there.  They stay for lines with other factors.  What bounds
// them is the instructions and barriers of their stages (225 = 3 3 5 5 there,
// 15 15 here), not memory.
#pragma once

#include "fft_fx.cuh"
#include "fft_io.cuh"

namespace gbfft {
namespace rt {

using namespace dev;

// FP32 on the CUDA cores.  The table twiddles are a high and a low part: on a
// line with a few large modes the rounding errors of a table add up in the
// modes' bins.  (Over 70 random boxes the rel-L2 against 64 bits is 0.96 of
// the general kernel's on average, 0.83 to 1.08 on single ones, where the order
// of the roundings differs; with rounded twiddles 0.98.)
struct F32 {
  using T = float;
  using C = float2;
  using W = float4;  // real, imaginary: high parts, low parts
  static constexpr int kMaxR = 16;
  static constexpr bool kFixed = false;
  static constexpr int kPadShift = 4;
  __device__ __forceinline__ static W root(const W* p) { return __ldg(p); }
  __device__ __forceinline__ static C mul(C a, W w, int) {
    return make_float2(fmaf(a.x, w.x, fmaf(-a.y, w.y, fmaf(-a.y, w.w, a.x * w.z))),
                       fmaf(a.x, w.y, fmaf(a.y, w.x, fmaf(a.y, w.z, a.x * w.w))));
  }
  __device__ __forceinline__ static C first(C a) { return a; }
  template <int R>
  __device__ __forceinline__ static void dft(C* v) { dft_f32<R>(v); }
};
// FP64 in fixed point.
struct Fixed {
  using T = double;
  using C = fx::I2;
  using W = fx::W4;
  static constexpr int kMaxR = 10;
  static constexpr bool kFixed = true;
  static constexpr int kPadShift = 3;
  __device__ __forceinline__ static W root(const W* p) { return fx::ldw(p); }
  __device__ __forceinline__ static C mul(C a, W w, int r) { return fx::mul_tw(a, w, r); }
  __device__ __forceinline__ static C first(C a) { return fx::mk(fx::scale_down(a.x), fx::scale_down(a.y)); }
  template <int R>
  __device__ __forceinline__ static void dft(C* v) { fx::dft<R>(v); }
};

// Calls f(integral_constant<R>) for the runtime radix R.
template <class A, class F>
__device__ __forceinline__ void with_radix(int R, F&& f) {
  switch (R) {
    case 2: f(std::integral_constant<int, 2>{}); break;
    case 3: f(std::integral_constant<int, 3>{}); break;
    case 4: f(std::integral_constant<int, 4>{}); break;
    case 5: f(std::integral_constant<int, 5>{}); break;
    case 6: f(std::integral_constant<int, 6>{}); break;
    case 7: f(std::integral_constant<int, 7>{}); break;
    case 8: f(std::integral_constant<int, 8>{}); break;
    case 9: f(std::integral_constant<int, 9>{}); break;
    case 10: f(std::integral_constant<int, 10>{}); break;
    default:
      if constexpr (!A::kFixed) {
        if (R == 11) f(std::integral_constant<int, 11>{});
        else if (R == 12) f(std::integral_constant<int, 12>{});
        else if (R == 13) f(std::integral_constant<int, 13>{});
        else if (R == 14) f(std::integral_constant<int, 14>{});
        else if (R == 15) f(std::integral_constant<int, 15>{});
        else f(std::integral_constant<int, 16>{});
      }
      break;
  }
}

// Exchange slots of a tile: strided dense (the lanes walk the lines),
// contiguous lines with a pad entry per 128 bytes.
template <class A, bool CONTIG>
struct Slots {
  int base, L;
  __device__ __forceinline__ int operator()(int n) const {
    return CONTIG ? base + n + (n >> A::kPadShift) : n * L + base;
  }
};

// How a result leaves FP32 (fixed point: fx::Back).
struct Turn {
  int flip;
  __device__ __forceinline__ float2 point(float2 v) const {
    return make_float2(v.x, __int_as_float(__float_as_int(v.y) ^ flip));
  }
  __device__ __forceinline__ float2 half_a(float2 zk, float2 zm) const {
    return make_float2((zk.x + zm.x) * 0.5f, (zk.y - zm.y) * 0.5f);
  }
  __device__ __forceinline__ float2 half_b(float2 zk, float2 zm) const {
    return make_float2((zk.y + zm.y) * 0.5f, (zm.x - zk.x) * 0.5f);
  }
};

template <class A, int KIND, bool CONTIG>
__global__ void __launch_bounds__(rt_threads(sizeof(typename A::T)), 2) rt_pass_kernel(const __grid_constant__ PassArgs a,
                                                                const __grid_constant__ FxPlan p) {
  using T = typename A::T;
  using C = typename A::C;
  using W = typename A::W;
  using G = Cx<T>;
  constexpr int MR = A::kMaxR;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  chained_entry();
  LineCtx<T, KIND, CONTIG> c;
  c.init(a);
  const Io<T, KIND, CONTIG> io(c);
  const int N = c.N, tpl = c.tpl, t = c.t, last = p.nst - 1;
  C* buf0 = reinterpret_cast<C*>(smem_raw);
  C* buf1 = buf0 + rt_entries(N, a.L);
  Slots<A, CONTIG> slot;
  slot.L = a.L;
  slot.base = CONTIG ? c.line * (N + (N >> A::kPadShift) + 1) : c.line;
  const W* tw = reinterpret_cast<const W*>(p.tw);
  const int back = KIND == K_C2R || (KIND == K_C2C && c.inverse) ? (int)0x80000000 : 0;
  std::conditional_t<A::kFixed, fx::Back<KIND>, Turn> out;
  out.flip = back;

  // the points of butterfly t of the first stage (c2r: the half spectra,
  // points t, t + tpl, ... of both)
  const int R0 = p.radix[0], nb0 = N / R0, h = N / 2 + 1;
  constexpr int Q = KIND == K_C2R ? 2 * (MR / 2 + 1) : MR;
  G x[Q];
  if constexpr (KIND == K_C2R) {
#pragma unroll
    for (int i = 0; i < Q / 2; ++i) {
      const int j = t + i * tpl;
      x[2 * i] = x[2 * i + 1] = io.zero();
      if (j < h) io.halves(i * tpl, x[2 * i], x[2 * i + 1]);
      if (j == 0 || 2 * j == N) x[2 * i].y = x[2 * i + 1].y = 0;  // Im of the DC and Nyquist bins is ignored
    }
  } else {
#pragma unroll
    for (int r = 0; r < MR; ++r) x[r] = r < R0 && t < nb0 ? io.load(r * nb0) : io.zero();
  }
  C v[MR];
  if constexpr (A::kFixed) {
    const fx::Words words(smem_raw + rt_smem_bytes(8, N, a.L, p.nst), a.L);
    words.clear(a.L);
    if (KIND == K_C2R && t == 0) {  // bins 0 apart
      words.ref[c.line] = make_double2(x[0].x, x[1].x);
      x[0] = x[1] = make_double2(0, 0);
    }
    __syncthreads();
    fx::PassScale<KIND> sc;
    if (!sc.find(x, words, c.line, t == 0, [&](int r) { return r < R0 && t < nb0; })) {
      fx::fallback<KIND, CONTIG>(a, reinterpret_cast<double2*>(smem_raw));
      return;
    }
#pragma unroll 1
    for (int s = 0; s <= last; ++s) sc.stage(p.lg[s], p.shift[s], s == last);
    const int sa = sc.shift_a(), sb = sc.shift_b();
    out = sc.back(p.shift[last], back);
    if constexpr (KIND == K_C2R) {
      if (t == 0) sc.set_dc(words, c.line, p.shift[last]);
#pragma unroll
      for (int i = 0; i < Q / 2; ++i) {
        const int j = t + i * tpl;
        if (j < h) {
          const fx::ll ax = fx::to_fixed(x[2 * i].x, sa), ay = fx::to_fixed(x[2 * i].y, sa);
          const fx::ll bx = fx::to_fixed(x[2 * i + 1].x, sb), by = fx::to_fixed(x[2 * i + 1].y, sb);
          // z = x1 + i x2, conjugated for the inverse-by-conjugation
          buf0[slot(j)] = fx::mk(ax - by, -(ay + bx));
          if (j > 0 && 2 * j < N) buf0[slot(N - j)] = fx::mk(ax + by, ay - bx);
        }
      }
    } else {
#pragma unroll
      for (int r = 0; r < MR; ++r) v[r] = fx::mk(fx::to_fixed(x[r].x, sa), fx::to_fixed(x[r].y, sb, back));
    }
  } else if constexpr (KIND == K_C2R) {
#pragma unroll
    for (int i = 0; i < Q / 2; ++i) {
      const int j = t + i * tpl;
      if (j < h) {
        const G u = x[2 * i], w = x[2 * i + 1];
        buf0[slot(j)] = make_float2(u.x - w.y, -(u.y + w.x));
        if (j > 0 && 2 * j < N) buf0[slot(N - j)] = make_float2(u.x + w.y, u.y - w.x);
      }
    }
  } else {
#pragma unroll
    for (int r = 0; r < MR; ++r) v[r] = make_float2(x[r].x, __int_as_float(__float_as_int(x[r].y) ^ back));
  }

  // stage 0, from the registers (c2r: from buffer 0) into buffer 0
  C* A0 = buf0;
  C* B = buf1;
  if constexpr (KIND == K_C2R) {
    __syncthreads();
#pragma unroll
    for (int r = 0; r < MR; ++r)
      if (r < R0 && t < nb0) v[r] = buf0[slot(t + r * nb0)];
    __syncthreads();
  }
  if (t < nb0) {
    with_radix<A>(R0, [&](auto RC) {
      constexpr int R = decltype(RC)::value;
      A::template dft<R>(v);
#pragma unroll
      for (int r = 0; r < R; ++r) A0[slot(t * R + r)] = v[r];
    });
  }
  __syncthreads();
  // the stages between, from buffer to buffer
  int s = 1;
#pragma unroll 1
  for (; s < last; ++s) {
    const int Ns = p.ns[s];
    const unsigned magic = p.magic[s];
    with_radix<A>(p.radix[s], [&](auto RC) {
      constexpr int R = decltype(RC)::value;
      const int nb = N / R;
#pragma unroll 1
      for (int b = t; b < nb; b += tpl) {
        const int k = b - (int)__umulhi((unsigned)b, magic) * Ns, base = (b - k) * R + k;
        const W* w = tw + (Ns - 1) + k;
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = A0[slot(b + r * nb)];
        v[0] = A::first(v[0]);
#pragma unroll
        for (int r = 1; r < R; ++r) v[r] = A::mul(v[r], A::root(w + (r - 1) * Ns), r);
        A::template dft<R>(v);
#pragma unroll
        for (int r = 0; r < R; ++r) B[slot(base + r * Ns)] = v[r];
      }
    });
    __syncthreads();
    C* const q = A0;
    A0 = B;
    B = q;
  }
  // the last stage: its outputs are points b + r ns
  {
    const int Ns = p.ns[last];
    fx::I2 dc;
    if constexpr (A::kFixed && KIND == K_C2R)
      dc = *reinterpret_cast<const fx::I2*>(&fx::Words(smem_raw + rt_smem_bytes(8, N, a.L, p.nst), a.L).ref[c.line]);
    with_radix<A>(p.radix[last], [&](auto RC) {
      constexpr int R = decltype(RC)::value;
#pragma unroll 1
      for (int b = t; b < Ns; b += tpl) {  // n / R = ns butterflies, k = b
        const W* w = tw + (Ns - 1) + b;
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = A0[slot(b + r * Ns)];
        v[0] = A::first(v[0]);
#pragma unroll
        for (int r = 1; r < R; ++r) v[r] = A::mul(v[r], A::root(w + (r - 1) * Ns), r);
        if constexpr (A::kFixed && KIND == K_C2R) v[0] = fx::add(v[0], dc);
        A::template dft<R>(v);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          // in place for r2c: the thread's own points
          if constexpr (KIND == K_R2C) A0[slot(b + r * Ns)] = v[r];
          else {
            G z = out.point(v[r]);
            if constexpr (A::kFixed && KIND == K_C2C)
              if (r == 0 && out.off && b == 0) out.dc(z, N);
            io.store(b - t + r * Ns, z);
          }
        }
      }
    });
  }
  if constexpr (KIND == K_R2C) {
    __syncthreads();
#pragma unroll 1
    for (int k = t; k < h; k += tpl) {
      const C zk = A0[slot(k)], zm = A0[slot(k == 0 ? 0 : N - k)];
      G xa = out.half_a(zk, zm), xb = out.half_b(zk, zm);
      if constexpr (A::kFixed)
        if (out.off && k == 0) out.dc(xa, xb, N);
      io.put_halves(k - t, xa, xb);
    }
  }
}

template <class A, int KIND, bool CONTIG>
cudaError_t launch_k(const PassArgs& a, cudaStream_t stream) {
  const FxPlan& p = *a.fx;
  const size_t smem = rt_smem_bytes((int)sizeof(typename A::T), a.n, a.L, p.nst);
  if (p.nst < 2 || a.L < 1 || a.L * a.tpl > rt_threads((int)sizeof(typename A::T)) || a.tpl * p.radix[0] < a.n || smem > kFxMaxSmem)
    return cudaErrorInvalidValue;
  auto kern = rt_pass_kernel<A, KIND, CONTIG>;
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

template <class A>
cudaError_t launch(int kind, bool contiguous, const PassArgs& a, cudaStream_t s) {
  if (kind == K_C2C) return contiguous ? launch_k<A, K_C2C, true>(a, s) : launch_k<A, K_C2C, false>(a, s);
  if (kind == K_R2C) return contiguous ? launch_k<A, K_R2C, true>(a, s) : launch_k<A, K_R2C, false>(a, s);
  if (kind == K_C2R) return contiguous ? launch_k<A, K_C2R, true>(a, s) : launch_k<A, K_C2R, false>(a, s);
  return cudaErrorInvalidValue;
}

}  // namespace rt
}  // namespace gbfft
