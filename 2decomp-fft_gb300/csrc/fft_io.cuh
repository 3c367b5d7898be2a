// What the smooth-length kernels share: the global accesses of a thread's
// points, and the FP32 butterflies.
#pragma once

#include "fft_common.cuh"

namespace gbfft {
namespace rt {

using namespace dev;

// Forward DFT of size R in registers (FP32).  R = P Q coprime goes without
// twiddles between (Good's mapping: n = Q n1 + P n2 mod R gives W_R^(n k) =
// W_P^(n1 k) W_Q^(n2 k), and result k sits at (k mod P, k mod Q)).
template <int R>
__device__ __forceinline__ void dft_f32(float2* v) {
  if constexpr (R == 1 || coprime_part(R) == R) {
    dftg<R>(v);
  } else {
    constexpr int P = coprime_part(R), Q = R / P;
    float2 a[R];
    static_for<0, Q>([&](auto I2) {
      constexpr int n2 = decltype(I2)::value;
      float2 t[P];
      static_for<0, P>([&](auto I1) { t[decltype(I1)::value] = v[(Q * decltype(I1)::value + P * n2) % R]; });
      dft_f32<P>(t);
      static_for<0, P>([&](auto K1) { a[n2 * P + decltype(K1)::value] = t[decltype(K1)::value]; });
    });
    static_for<0, P>([&](auto K1) {
      constexpr int k1 = decltype(K1)::value;
      float2 u[Q];
      static_for<0, Q>([&](auto I2) { u[decltype(I2)::value] = a[decltype(I2)::value * P + k1]; });
      dft_f32<Q>(u);
      static_for<0, Q>([&](auto K2) { v[crt(P, Q, k1, decltype(K2)::value)] = u[decltype(K2)::value]; });
    });
  }
}

// Global accesses of a thread's points t + n: one multiply-add an address
// (the row strides are below 2^32 bytes).
template <typename T, int KIND, bool CONTIG, class Ctx = LineCtx<T, KIND, CONTIG>>
struct Io {
  using C = Cx<T>;
  const Ctx& c;
  const char *s0, *s1;
  char *d0, *d1;
  unsigned ss, ds;
  __device__ __forceinline__ explicit Io(const Ctx& ctx) : c(ctx) {
    constexpr int SB = (KIND == K_R2C ? 1 : 2) * sizeof(T), DB = (KIND == K_C2R ? 1 : 2) * sizeof(T);
    ss = (unsigned)c.ssn * SB;
    ds = (unsigned)c.dsn * DB;
    s0 = reinterpret_cast<const char*>(c.src) + c.sb0 * SB + (unsigned long long)ss * (unsigned)c.t;
    s1 = reinterpret_cast<const char*>(c.src) + c.sb1 * SB + (unsigned long long)ss * (unsigned)c.t;
    d0 = reinterpret_cast<char*>(c.dst) + c.db0 * DB + (unsigned long long)ds * (unsigned)c.t;
    d1 = reinterpret_cast<char*>(c.dst) + c.db1 * DB + (unsigned long long)ds * (unsigned)c.t;
  }
  __device__ __forceinline__ static C zero() { return cmk<C>(T(0), T(0)); }
#ifdef GB_DEBUG_BOUNDS
  __device__ __forceinline__ C load(int n) const { return c.gload_raw(c.t + n); }
  __device__ __forceinline__ void halves(int n, C& a, C& b) const {
    a = c.half(0, c.t + n);
    b = c.half(1, c.t + n);
  }
  __device__ __forceinline__ void store(int n, C v) const { c.gstore_raw(c.t + n, v); }
  __device__ __forceinline__ void put_halves(int n, C a, C b) const {
    c.put_half(0, c.t + n, a);
    c.put_half(1, c.t + n, b);
  }
#else
  __device__ __forceinline__ unsigned long long so(int n) const { return (unsigned long long)(unsigned)n * ss; }
  __device__ __forceinline__ unsigned long long dof(int n) const { return (unsigned long long)(unsigned)n * ds; }
  template <typename V>
  __device__ __forceinline__ static V ld(const char* p) {
    return Ctx::ld(reinterpret_cast<const V*>(p));
  }
  // c2c: the point; r2c: both real lines' values
  __device__ __forceinline__ C load(int n) const {
    if (!c.valid) return zero();
    if (KIND == K_C2C || (!CONTIG && c.pvec && c.has1)) return ld<C>(s0 + so(n));
    return cmk<C>(ld<T>(s0 + so(n)), c.has1 ? ld<T>(s1 + so(n)) : T(0));
  }
  // c2r: both half spectra's points
  __device__ __forceinline__ void halves(int n, C& a, C& b) const {
    a = b = zero();
    if (!c.valid) return;
    if constexpr (sizeof(T) == 4) {
      if (c.cvec && c.has1) {
        const float4 q = Ctx::ld4(reinterpret_cast<const float4*>(s0 + so(n)));
        a = make_float2(q.x, q.y);
        b = make_float2(q.z, q.w);
        return;
      }
    }
    a = ld<C>(s0 + so(n));
    if (c.has1) b = ld<C>(s1 + so(n));
  }
  __device__ __forceinline__ void store(int n, C v) const {
    if (!c.valid) return;
    if (KIND == K_C2C || (!CONTIG && c.pvec && c.has1)) {
      *reinterpret_cast<C*>(d0 + dof(n)) = v;
      return;
    }
    *reinterpret_cast<T*>(d0 + dof(n)) = v.x;
    if (c.has1) *reinterpret_cast<T*>(d1 + dof(n)) = v.y;
  }
  __device__ __forceinline__ void put_halves(int n, C a, C b) const {
    if (!c.valid) return;
    if constexpr (sizeof(T) == 4) {
      if (c.cvec && c.has1) {
        *reinterpret_cast<float4*>(d0 + dof(n)) = make_float4(a.x, a.y, b.x, b.y);
        return;
      }
    }
    *reinterpret_cast<C*>(d0 + dof(n)) = a;
    if (c.has1) *reinterpret_cast<C*>(d1 + dof(n)) = b;
  }
#endif
};

}  // namespace rt
}  // namespace gbfft
