// Real-to-real transforms (DCT-I..IV, DST-I..IV) around a complex FFT of
// length M, in fixed point and (for the lines fixed point does not take) FP64.
//
// What bounds these passes: the FFT's work.  The extensions of the plain form
// (dtt.cu) are complex lines of 2n points for n real ones; here a complex line
// of n points does two real lines, a quarter of the points.
//
// A complex line carries two real lines a, b as U = a + i b (all maps below
// are real-linear in a and b, so they act on U), except DCT-IV / DST-IV of an
// even n, where it carries one line.  With W = exp(-2 pi i / (4n)),
// F = FFT_M(z):
//   DCT-I   M = 2(n-1): z the even extension;           a_k + i b_k = F_k
//   DST-I   M = 2(n+1): z the odd extension;            a_k = -Im F_{k+1}, b_k = Re F_{k+1}
//   DCT-II  M = n: z_j = U_{2j}, z_{n-1-j} = U_{2j+1};  with G = F_k + conj F_{n-k} (a),
//                  -i (F_k - conj F_{n-k}) (b), H = W^k G: Y_k = Re H, Y_{n-k} = -Im H
//   DCT-III M = n: z_k = W^k (conj U_k + i conj U_{n-k}) (k = 0: conj U_0);
//                  a = Re F, b = -Im F, in DCT-II's order of z
//   DCT-IV  n odd, M = n: odd p = 2j+1 is +-(n + 4i) (mod 8n; n + 4i -> n + 4(i+n)
//                  changes the sign), z_i = +-(-1)^i U_j, and with 2k+1 -> l:
//                  Y_k = +-(-1)^l Re(exp(-i pi n/4) G), G as above at m = 2l mod n
//           n even, M = n/2, one line: z_j = (x_{2j} + i x_{n-1-2j}) w_j, c_k = F_k w_k,
//                  w_j = exp(-2 pi i (8j+1) / (16n)): Y_{2k} = 2 Re c_k, Y_{n-1-2k} = -2 Im c_k
//   DST-II(x)_k  = DCT-II((-1)^j x_j)_{n-1-k}
//   DST-III(x)_k = (-1)^k DCT-III(x_{n-1-j})_k, DST-IV(x)_k = (-1)^k DCT-IV(x_{n-1-j})_k
#pragma once

#include "fft_fx.cuh"

namespace gbfft {
namespace r2r {

using namespace dev;

// Arithmetic of a transform: values C, table roots W, real components T.
template <typename R>
struct Float {
  using C = Cx<R>;
  using W = Cx<R>;
  using T = R;
  __device__ __forceinline__ static C mk(T a, T b) { return cmk<C>(a, b); }
  __device__ __forceinline__ static W root(const W* p) { return __ldg(p); }
  __device__ __forceinline__ static C rot(C a, W w, int) { return cmul(a, w); }
  __device__ __forceinline__ static C down(C a) { return a; }  // the scale of a value that is not rotated
  __device__ __forceinline__ static T isqrt2(T a) { return a * T(0.70710678118654752440); }
};
struct Fixed {
  using C = fx::I2;
  using W = fx::W4;
  using T = fx::ll;
  __device__ __forceinline__ static C mk(T a, T b) { return fx::mk(a, b); }
  __device__ __forceinline__ static W root(const W* p) { return fx::ldw(p); }
  __device__ __forceinline__ static C rot(C a, W w, int r) { return fx::mul_tw(a, w, r); }  // halves
  __device__ __forceinline__ static C down(C a) { return fx::mk(fx::scale_down(a.x), fx::scale_down(a.y)); }
  __device__ __forceinline__ static T isqrt2(T a) { return fx::mulk<fx::sincos_q62(1, 8).c>(a); }
};

__device__ __forceinline__ bool single_line(int kind, int n) { return (kind == 4 || kind == 8) && n % 2 == 0; }
// DCT-II's order: point j of the window at slot perm(j)
__device__ __forceinline__ int perm(int j, int n) { return j & 1 ? n - 1 - (j >> 1) : j >> 1; }
// DCT-IV of odd n: 2j+1 -> i in [0, n); the sign of (the wrap and (-1)^i)
__device__ __forceinline__ int odd_map(int j, int n, bool& neg) {
  const int p = 2 * j + 1;
  const int q = ((p - n) & 3) == 0 ? p : -p;
  int i = (q - n) / 4;
  neg = i < 0;
  if (i < 0) i += n;
  neg = neg != ((i & 1) != 0);
  return i;
}

template <class A, class Slot>
struct Maps {
  using C = typename A::C;
  using T = typename A::T;
  using W = typename A::W;
  int kind, n, M;
  const W* w;
  Slot slot;

  __device__ __forceinline__ static C neg(C v) { return A::mk(-v.x, -v.y); }
  __device__ __forceinline__ static C conj(C v) { return A::mk(v.x, -v.y); }

  // element j of the line (one value of both real lines; even DCT-IV: x_{2j}, x_{n-1-2j})
  __device__ __forceinline__ void place(C* S, int j, C v) const {
    switch (kind) {
      case 1:
        S[slot(j)] = v;
        if (j > 0 && j < n - 1) S[slot(M - j)] = v;
        break;
      case 5:
        S[slot(j + 1)] = v;
        S[slot(M - 1 - j)] = neg(v);
        if (j == 0) S[slot(0)] = S[slot(n + 1)] = A::mk(T(0), T(0));
        break;
      case 2:
        S[slot(perm(j, n))] = v;
        break;
      case 6:
        S[slot(perm(j, n))] = j & 1 ? neg(v) : v;
        break;
      case 3:
        S[slot(j)] = v;
        break;
      case 7:
        S[slot(n - 1 - j)] = v;
        break;
      default:
        if (n % 2 == 0) {
          S[slot(j)] = A::rot(v, A::root(w + j), j);
        } else {
          bool ng;
          const int i = odd_map(kind == 4 ? j : n - 1 - j, n, ng);
          S[slot(i)] = ng ? neg(v) : v;
        }
        break;
    }
  }
  __device__ __forceinline__ bool combines() const { return kind == 3 || kind == 7; }
  // DCT-III: z from U in place; the thread owns the pair (k, n - k), k <= n / 2
  __device__ __forceinline__ void combine(C* S, int k) const {
    const C u = S[slot(k)];
    if (k == 0) {
      S[slot(0)] = A::down(conj(u));
      return;
    }
    const C m = S[slot(n - k)];
    S[slot(k)] = A::rot(A::mk(u.x + m.y, m.x - u.y), A::root(w + k), k);
    if (k != n - k) S[slot(n - k)] = A::rot(A::mk(m.x + u.y, u.x - m.y), A::root(w + n - k), k);
  }
  // outputs from F in S: emit(i, y_a, y_b), or emit1(i, y) for one line
  __device__ __forceinline__ int steps() const {
    return kind == 2 || kind == 6 ? n / 2 + 1 : (kind == 4 || kind == 8) && n % 2 == 0 ? n / 2 : n;
  }
  template <class E, class E1>
  __device__ __forceinline__ void finish(const C* S, int k, E&& emit, E1&& emit1) const {
    switch (kind) {
      case 1: {
        const C f = S[slot(k)];
        emit(k, f.x, f.y);
        break;
      }
      case 5: {
        const C f = S[slot(k + 1)];
        emit(k, -f.y, f.x);
        break;
      }
      case 3:
      case 7: {
        const C f = S[slot(perm(k, n))];
        if (kind == 7 && (k & 1)) emit(k, -f.x, f.y);
        else emit(k, f.x, -f.y);
        break;
      }
      case 2:
      case 6: {
        const C f = S[slot(k)], g = S[slot(k == 0 ? 0 : n - k)];
        const W r = A::root(w + k);
        const C ha = A::rot(A::mk(f.x + g.x, f.y - g.y), r, k);
        const C hb = A::rot(A::mk(f.y + g.y, g.x - f.x), r, k);
        emit(kind == 2 ? k : n - 1 - k, ha.x, hb.x);
        if (k > 0 && k != n - k) emit(kind == 2 ? n - k : k - 1, -ha.y, -hb.y);
        break;
      }
      default:
        if (n % 2 == 0) {
          const C c = A::rot(S[slot(k)], A::root(w + k), k);
          emit1(2 * k, c.x);
          emit1(n - 1 - 2 * k, kind == 8 ? c.y : -c.y);
        } else {
          bool ng;
          const int l = odd_map(k, n, ng);
          if (kind == 8 && (k & 1)) ng = !ng;
          const int m = 2 * l < n ? 2 * l : 2 * l - n;
          const C f = S[slot(m)], g = S[slot(m == 0 ? 0 : n - m)];
          // cos, sin of pi n / 4 are +-1 / sqrt 2
          const bool nc = (n & 7) == 3 || (n & 7) == 5, ns = (n & 7) >= 5;
          const T ax = f.x + g.x, ay = f.y - g.y, bx = f.y + g.y, by = g.x - f.x;
          const T ya = A::isqrt2((nc ? -ax : ax) + (ns ? -ay : ay));
          const T yb = A::isqrt2((nc ? -bx : bx) + (ns ? -by : by));
          emit(k, ng ? -ya : ya, ng ? -yb : yb);
        }
        break;
    }
  }
  // even DCT-IV: c_k carries half of Y
  __device__ __forceinline__ static int doubled(int kind, int n) { return single_line(kind, n) ? 1 : 0; }
  // What the fixed-point scale needs: bits by which the maps before the FFT
  // can raise a modulus (grow) or its halvings lower it (pre), and the
  // headroom (post) and halvings (tail) of those behind it.
  __device__ __forceinline__ int grow() const { return kind == 1 || kind == 5 || kind == 3 || kind == 7 ? 1 : 0; }
  __device__ __forceinline__ int pre() const { return kind == 3 || kind == 7 || single_line(kind, n) ? 1 : 0; }
  __device__ __forceinline__ int post() const { return kind == 2 || kind == 6 || (kind % 4 == 0 && n % 2) ? 1 : 0; }
  __device__ __forceinline__ int tail() const { return kind == 2 || kind == 6 || single_line(kind, n) ? 1 : 0; }
};

// Kinds that have a constant line's whole transform in output 0 (DCT-I,
// DCT-II): 2 (n - 1) and 2 n times it.
__device__ __forceinline__ bool keeps_mean(int kind) { return kind == 1 || kind == 2; }

// The real lines behind complex line cl of an r2r pass.
template <typename T, bool CONTIG>
struct Lines {
  const T* src;
  T* dst;
  long long b0, b1, sn;
  int off, n, kind;
  bool valid, has1, single, vec;
  int only = 2;  // 0, 1: that real line alone (the other reads as zero and is not written)

  __device__ __forceinline__ Lines(const DttArgs& a, long long cl, long long v) {
    single = single_line(a.kind, a.n);
    const long long r0 = single ? cl : 2 * cl;
    valid = r0 < a.nlines;
    has1 = !single && r0 + 1 < a.nlines;
    src = reinterpret_cast<const T*>(a.src);
    dst = reinterpret_cast<T*>(a.dst);
    b0 = CONTIG ? r0 * a.sl : r0 + v * a.sl;
    b1 = CONTIG ? b0 + a.sl : b0 + 1;
    sn = a.sn;
    off = a.off;
    n = a.n;
    kind = a.kind;
    vec = !CONTIG && has1 && a.pair_vec;
  }
  // element j as it enters Maps::place
  __device__ __forceinline__ Cx<T> element(int j) const {
    using C = Cx<T>;
    if (!valid) return cmk<C>(T(0), T(0));
    if (single) {
      const T p = src[b0 + (long long)(off + 2 * j) * sn], q = src[b0 + (long long)(off + n - 1 - 2 * j) * sn];
      return kind == 4 ? cmk<C>(p, q) : cmk<C>(q, p);
    }
    const long long at = (long long)(off + j) * sn;
    if (vec) return *reinterpret_cast<const C*>(src + b0 + at);
    return cmk<C>(only != 1 ? src[b0 + at] : T(0), has1 && only != 0 ? src[b1 + at] : T(0));
  }
  __device__ __forceinline__ void store(int i, T ya, T yb) const {
    if (!valid) return;
    const long long at = (long long)(off + i) * sn;
    if (vec) {
      *reinterpret_cast<Cx<T>*>(dst + b0 + at) = cmk<Cx<T>>(ya, yb);
      return;
    }
    if (only != 1) dst[b0 + at] = ya;
    if (has1 && only != 0) dst[b1 + at] = yb;
  }
  __device__ __forceinline__ void store1(int i, T y) const {
    if (valid) dst[b0 + (long long)(off + i) * sn] = y;
  }
  // puts the lines' means back into output 0, which the calling thread has stored
  __device__ __forceinline__ void add_mean(double2 mean) const {
    if (!valid) return;
    const double w = 2 * (kind == 1 ? n - 1 : n);
    const long long at = (long long)off * sn;
    dst[b0 + at] = __fma_rn(w, mean.x, dst[b0 + at]);
    if (has1) dst[b1 + at] = __fma_rn(w, mean.y, dst[b1 + at]);
  }
  // points outside the window, copied through when dst is another array
  __device__ __forceinline__ void pass_through(int naxis, int t, int tpl) const {
    if (!valid || src == dst) return;
    for (int j = t; j < naxis; j += tpl)
      if (j < off || j >= off + n) {
        if (only != 1) dst[b0 + (long long)j * sn] = src[b0 + (long long)j * sn];
        if (has1 && only != 0) dst[b1 + (long long)j * sn] = src[b1 + (long long)j * sn];
      }
  }
};
__device__ __forceinline__ int elements(int kind, int n) { return single_line(kind, n) ? n / 2 : n; }

// Shared-memory slots of a runtime-planned tile (LineCtx's layout).
template <class Ctx>
struct CtxSlot {
  const Ctx* c;
  __device__ __forceinline__ int operator()(int i) const { return c->sidx(i); }
};

// The runtime-planned transform of a CTA's lines in floating point: thread t
// of tpl of line `line`, complex line cl, its real line `only`, buffers of e
// points.
template <typename T, bool CONTIG>
__device__ __forceinline__ void run_lines(const DttArgs& a, Cx<T>* buf0, size_t e, int t, int tpl, int line, int L,
                                          long long cl, long long v, bool active, int only) {
  using C = Cx<T>;
  using Ctx = LineCtx<T, K_C2C, CONTIG>;
  Ctx c;
  c.tw = reinterpret_cast<const C*>(a.tw);
  c.N = a.M;
  c.L = L;
  c.t = active ? t : a.M;  // a thread without a line takes no point
  c.tpl = tpl;
  c.line = active ? line : 0;
  Lines<T, CONTIG> ln(a, cl, v);
  ln.vec = false;
  ln.only = only;
  if (!active || (only == 1 && !ln.has1)) ln.valid = ln.has1 = false;
  Maps<Float<T>, CtxSlot<Ctx>> mp{a.kind, a.n, a.M, reinterpret_cast<const C*>(a.w), {&c}};
  C* A = buf0;
  C* B = buf0 + (e + (e >> 4) + 1);
  const int first = active ? t : a.naxis + a.M;
#pragma unroll 1
  for (int j = first; j < elements(a.kind, a.n); j += tpl) mp.place(A, j, ln.element(j));
  __syncthreads();
  if (mp.combines()) {
#pragma unroll 1
    for (int k = first; 2 * k <= a.n; k += tpl) mp.combine(A, k);
    __syncthreads();
  }
  run_stages_pp<T, K_C2C, CONTIG>(c, a.nst, a.radix, A, B);
  const T two = T(1 + Maps<Float<T>, CtxSlot<Ctx>>::doubled(a.kind, a.n));
#pragma unroll 1
  for (int k = first; k < mp.steps(); k += tpl)
    mp.finish(A, k, [&](int i, T ya, T yb) { ln.store(i, ya, yb); }, [&](int i, T y) { ln.store1(i, two * y); });
  ln.pass_through(a.naxis, first, tpl);
}

// The lines of a fixed-point CTA that fixed point does not take, in FP64, as
// many at a time as two buffers in the CTA's shared memory hold, the two real
// lines of a pair one after the other: a NaN stays in its line.
template <bool CONTIG>
__device__ __noinline__ void fallback(const DttArgs& a, double2* buf) {
  const int threads = blockDim.x * blockDim.y, tid = threadIdx.x + threadIdx.y * blockDim.x;
  const int G = a.L > 1 ? a.L / 2 : 1, tpl = threads / G;
  const int t = CONTIG ? tid % tpl : tid / G, line = CONTIG ? tid / tpl : tid % G;
  const int lines = single_line(a.kind, a.n) ? 1 : 2;
  for (int g = 0; g < a.L; g += G)
    for (int only = 0; only < lines; ++only) {
      run_lines<double, CONTIG>(a, buf, (size_t)a.M * G, t, tpl, line, G, (long long)blockIdx.x * a.L + g + line,
                                CONTIG ? 0 : (long long)blockIdx.y, t < tpl && line < G && g + line < a.L, only);
      __syncthreads();
    }
}

}  // namespace r2r
}  // namespace gbfft
