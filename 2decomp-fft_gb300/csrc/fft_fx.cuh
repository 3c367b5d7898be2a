// 64-bit fixed-point complex arithmetic for FP64 lines.
//
// An SM issues two FP64 multiply-adds a clock but 64 64-bit integer adds and
// 32 32 x 32 -> 64-bit multiply-adds (measured on GB300).  An FFT is adds
// and multiplications by constants of modulus one, and no value of a line's
// transform exceeds the sum of the moduli of its inputs, so a line can be
// transformed in integers that share one power-of-two scale, chosen from
// that sum: 64 bits for numbers that hold 53.  The scale is the line's own
// (never a neighbour's; of two real lines that share a complex one, each its
// own), so a small line next to a large one keeps all its digits.
//
// Headroom: of 62 bits, those by which the largest of a stage's sums can exceed
// the line's largest value once the twiddles' divisions are taken off: at most
// the maximum over the stages of lg(points summed) - (halvings so far), 3 to 7
// for the compile-time plans of up to 2048 points, 8 at 4096, 9 for the worst
// supported length (1912 = 8 x 239; direct sums).
//
// What this keeps: against the line's norm the error is 0.1 to 0.9 of the FP64
// kernels', whatever the values (figures at fx_length).  A part of a line far
// below its largest value has an error of 2^-53 to 2^-59 of that value.  In
// FP64 it can have less, if the large part cancels exactly there, which takes
// numbers of few digits.  The two common cases are handled: a mean (PassScale,
// take_means) and c2r's bin 0.  Other patterns that cancel exactly (+c -c +c
// -c, say) leave the small rest of such a line the error above, as FP64 does
// for numbers of full length.
//
// Formats: a value is a signed 64-bit integer v, |v| < 2^62.  Table twiddles
// are Q62 (w 2^62) and multiplying by one divides by 2, after a stage of radix
// 8 or more by 4 (compile-time plans and the general kernel; the radices of
// fft_rt.cuh are small), which is cheaper (a value grows by sqrt(R) in a stage
// of radix R on noise and by nothing on a line with one large point; dividing
// by more than the growth loses bits); constants of the butterflies are Q64
// and keep the scale.  Every product is rounded to nearest at 2^-64 of its
// factors' range; the low 32 x 32 product (below half a unit) is left out.
#pragma once

#include "fft_common.cuh"
#include "fft_pp.cuh"

namespace gbfft {
namespace fx {

using ll = long long;

struct alignas(16) I2 {
  ll x, y;
};
// Q62 root: real and imaginary parts as balanced 32-bit halves (both signed,
// neither -2^31, value = hi 2^32 + lo)
struct alignas(16) W4 {
  int xl, xh, yl, yh;
};

__device__ __forceinline__ I2 mk(ll a, ll b) {
  I2 r;
  r.x = a;
  r.y = b;
  return r;
}
__device__ __forceinline__ I2 add(I2 a, I2 b) { return mk(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ I2 sub(I2 a, I2 b) { return mk(a.x - b.x, a.y - b.y); }
// a * b + c, 32 x 32 -> 64 bits.  Spelt out: from (ll)a * b the
// compiler made unsigned products and sign corrections (76 of 313
// instructions a point of a 256-point pass).
__device__ __forceinline__ ll madw(int a, int b, ll c) {
  ll d;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
  return d;
}
// balanced halves: v = hi(v) 2^32 + lo(v), both signed
__host__ __device__ __forceinline__ constexpr int hi(ll v) {
  return (int)(v >> 32) + (int)((unsigned)(unsigned long long)v >> 31);  // one shift-add
}
__host__ __device__ __forceinline__ constexpr int lo(ll v) { return (int)(unsigned)(unsigned long long)v; }
constexpr ll kHalf = 0x80000000ll;  // rounds a sum of middle products

// ---- compile-time roots in Q62 --------------------------------------------
// cos and sin of 2 pi m / d: the angle reduced exactly to [0, pi/4] on the
// rational, then Taylor series in 128-bit integer arithmetic.
constexpr unsigned long long kTwoPiQ61 = 14488038916154245685ull;  // 2 pi 2^61
constexpr ll mulq62(ll a, ll b) { return (ll)(((__int128)a * b + ((__int128)1 << 61)) >> 62); }
struct SC {
  ll s, c;
};
constexpr SC sincos_q62(long long m, long long d) {
  m %= d;
  if (m < 0) m += d;
  bool ns = false, nc = false, swap = false;
  if (2 * m > d) {
    m = d - m;
    ns = true;
  }
  if (4 * m > d) {
    m = d - 2 * m;
    d = 2 * d;
    nc = !nc;
  }
  if (8 * m > d) {
    m = d - 4 * m;
    d = 4 * d;
    swap = true;
  }
  const ll one = 1ll << 62;
  const ll x = (ll)(((unsigned __int128)kTwoPiQ61 * 2 * (unsigned __int128)m + (unsigned __int128)(d / 2)) /
                    (unsigned __int128)d);
  const ll x2 = mulq62(x, x);
  ll ts = x, s = x, tc = one, c = one;
  for (int k = 1; k < 14; ++k) {
    tc = -mulq62(tc, x2) / ((2 * k - 1) * (2 * k));
    c += tc;
    ts = -mulq62(ts, x2) / ((2 * k) * (2 * k + 1));
    s += ts;
  }
  if (swap) {
    const ll t = s;
    s = c;
    c = t;
  }
  return {ns ? -s : s, nc ? -c : c};
}
// A constant of [-1, 1] in Q62 as base + frac: base in {-1, 0, 1}, |frac| at
// most one half, as Q64.
constexpr int k_base(ll q) { return q >= (1ll << 61) ? 1 : q < -(1ll << 61) ? -1 : 0; }
constexpr ll k_frac(ll q) { return (q - k_base(q) * (1ll << 62)) * 4; }

// x times a constant (Q62 template argument), at x's scale.
template <ll Q>
__device__ __forceinline__ ll mulk(ll x) {
  constexpr ll F = k_frac(Q);
  constexpr int B = k_base(Q);
  const ll m = madw(lo(x), hi(F), madw(hi(x), lo(F), kHalf));
  const ll h = madw(hi(x), hi(F), m >> 32);
  return B > 0 ? h + x : B < 0 ? h - x : h;
}
// x * KX + y * KY.  The middle products of two terms fit 64 bits: with moduli
// that sum to at most 2^62 the high halves give at most sqrt(2) 2^61 there,
// the low ones |frac x| + |frac y| (at most 0.634 for the two parts of a
// root) times 2^63.
template <ll QX, ll QY>
__device__ __forceinline__ ll lin2(ll x, ll y) {
  constexpr ll FX = k_frac(QX), FY = k_frac(QY);
  constexpr int BX = k_base(QX), BY = k_base(QY);
  ll m = madw(lo(x), hi(FX), madw(hi(x), lo(FX), kHalf));
  m = madw(lo(y), hi(FY), madw(hi(y), lo(FY), m));
  ll h = madw(hi(y), hi(FY), madw(hi(x), hi(FX), m >> 32));
  h = BX > 0 ? h + x : BX < 0 ? h - x : h;
  return BY > 0 ? h + y : BY < 0 ? h - y : h;
}
// a * exp(-2 pi i M / R)
template <int R, int M>
__device__ __forceinline__ I2 mul_root(I2 a) {
  constexpr int m = ((M % R) + R) % R;
  if constexpr (m == 0) {
    return a;
  } else if constexpr (4 * m == R) {
    return mk(a.y, -a.x);
  } else if constexpr (2 * m == R) {
    return mk(-a.x, -a.y);
  } else if constexpr (4 * m == 3 * R) {
    return mk(-a.y, a.x);
  } else if constexpr ((8 * m) % R == 0) {
    // (+-1 +- i) / sqrt 2: one real constant for each component
    constexpr ll q = sincos_q62(1, 8).c;
    constexpr int o = 8 * m / R;  // 1, 3, 5, 7 eighths of a turn
    if constexpr (o == 1) return mk(mulk<q>(a.x + a.y), mulk<q>(a.y - a.x));
    else if constexpr (o == 3) return mk(mulk<q>(a.y - a.x), mulk<-q>(a.x + a.y));
    else if constexpr (o == 5) return mk(mulk<-q>(a.x + a.y), mulk<q>(a.x - a.y));
    else return mk(mulk<q>(a.x - a.y), mulk<q>(a.x + a.y));
  } else {
    constexpr SC w = sincos_q62(m, R);
    return mk(lin2<w.c, w.s>(a.x, a.y), lin2<-w.s, w.c>(a.x, a.y));
  }
}
__device__ __forceinline__ W4 ldw(const W4* p) {
  const int4 q = __ldg(reinterpret_cast<const int4*>(p));
  W4 w;
  w.xl = q.x;
  w.xh = q.y;
  w.yl = q.z;
  w.yh = q.w;
  return w;
}
// a * w / 2^SH (SH 1 or 2) for a table root: the middle products shifted by
// 30 + SH, the high ones doubled for SH = 1.  Exact ties (the
// twiddle 1 makes them) round up or down by the parity of r's bits, the
// imaginary part the other way: one direction for all would add up in bin 0,
// alternating ones in another.
template <int SH = 1>
__device__ __forceinline__ I2 mul_tw(I2 a, W4 w, int r) {
  static_assert(SH == 1 || SH == 2, "scale");
  const int xh = hi(a.x), xl = lo(a.x), yh = hi(a.y), yl = lo(a.y);
  const int xd = xh * (3 - SH), yd = yh * (3 - SH);
  const int odd = (0x6996 >> (r & 15)) & 1;
  const ll ur = kHalf / (3 - SH) - odd, ui = kHalf / (3 - SH) - 1 + odd;
  const int nh = -w.yh, nl = -w.yl;
  const ll mr = madw(yl, nh, madw(yh, nl, madw(xl, w.xh, madw(xh, w.xl, ur))));
  const ll mi = madw(yl, w.xh, madw(yh, w.xl, madw(xl, w.yh, madw(xh, w.yl, ui))));
  return mk(madw(yd, nh, madw(xd, w.xh, mr >> (30 + SH))), madw(yd, w.xh, madw(xd, w.yh, mi >> (30 + SH))));
}
// v / 2^SH, rounded to nearest even: the scale of a value that meets the
// twiddle 1 (a bias common to all of them would add up in one bin)
template <int SH = 1>
__device__ __forceinline__ ll scale_down(ll v) {
  return (v + (SH - 1) + ((v >> SH) & 1)) >> SH;
}
// The same two for a scale known at run time (1 or 2).
__device__ __forceinline__ I2 mul_tw(I2 a, W4 w, int r, int sh) {
  const int xh = hi(a.x), xl = lo(a.x), yh = hi(a.y), yl = lo(a.y);
  const int xd = xh << (2 - sh), yd = yh << (2 - sh);
  const int odd = (0x6996 >> (r & 15)) & 1;
  const ll ur = (kHalf >> (2 - sh)) - odd, ui = (kHalf >> (2 - sh)) - 1 + odd;
  const int nh = -w.yh, nl = -w.yl;
  const ll mr = madw(yl, nh, madw(yh, nl, madw(xl, w.xh, madw(xh, w.xl, ur))));
  const ll mi = madw(yl, w.xh, madw(yh, w.xl, madw(xl, w.yh, madw(xh, w.yl, ui))));
  return mk(madw(yd, nh, madw(xd, w.xh, mr >> (30 + sh))), madw(yd, w.xh, madw(xd, w.yh, mi >> (30 + sh))));
}
__device__ __forceinline__ ll scale_down(ll v, int sh) { return (v + (sh - 1) + ((v >> sh) & 1)) >> sh; }

// ---- butterflies (forward, natural order in and out) -----------------------
__device__ __forceinline__ void dft4v(I2& a0, I2& a1, I2& a2, I2& a3) {
  const I2 t0 = add(a0, a2), t1 = sub(a0, a2), t2 = add(a1, a3), d = sub(a1, a3);
  a0 = add(t0, t2);
  a2 = sub(t0, t2);
  a1 = mk(t1.x + d.y, t1.y - d.x);
  a3 = mk(t1.x - d.y, t1.y + d.x);
}
__device__ __forceinline__ void dft3p(I2* v) {
  constexpr ll q = sincos_q62(1, 3).s;
  const I2 t = add(v[1], v[2]), d = sub(v[1], v[2]);
  const I2 m = mk(v[0].x - ((t.x + 1) >> 1), v[0].y - (t.y >> 1));
  const ll sx = mulk<q>(d.x), sy = mulk<q>(d.y);
  v[0] = add(v[0], t);
  v[1] = mk(m.x + sy, m.y - sx);
  v[2] = mk(m.x - sy, m.y + sx);
}
// DFT5 on two constants a component: m1, m2 = (a0 - (t1 + t2) / 4) +- sqrt5/4
// (t1 - t2), and the sine pair.
__device__ __forceinline__ void dft5p(I2* v) {
  constexpr ll s1 = sincos_q62(1, 5).s, s2 = sincos_q62(2, 5).s;
  constexpr ll c5 = (sincos_q62(1, 5).c - sincos_q62(2, 5).c) / 2;  // sqrt 5 / 4
  const I2 t1 = add(v[1], v[4]), t2 = add(v[2], v[3]), t3 = sub(v[1], v[4]), t4 = sub(v[2], v[3]);
  const I2 a0 = v[0], ts = add(t1, t2), td = sub(t1, t2);
  const I2 b = mk(a0.x - ((ts.x + 2) >> 2), a0.y - ((ts.y + 2) >> 2));
  const I2 e = mk(mulk<c5>(td.x), mulk<c5>(td.y));
  const I2 m1 = add(b, e), m2 = sub(b, e);
  const I2 n1 = mk(lin2<s1, s2>(t3.x, t4.x), lin2<s1, s2>(t3.y, t4.y));
  const I2 n2 = mk(lin2<s2, -s1>(t3.x, t4.x), lin2<s2, -s1>(t3.y, t4.y));
  v[0] = add(a0, ts);
  v[1] = mk(m1.x + n1.y, m1.y - n1.x);
  v[4] = mk(m1.x - n1.y, m1.y + n1.x);
  v[2] = mk(m2.x + n2.y, m2.y - n2.x);
  v[3] = mk(m2.x - n2.y, m2.y + n2.x);
}
// A sum of constant multiples.  Its middle products are carried before they
// could leave 64 bits: two terms fit while their fracs sum to at most 0.7.
struct Acc {
  ll h, m;
  __device__ __forceinline__ Acc(ll start) : h(start), m(kHalf) {}
  template <ll Q>
  __device__ __forceinline__ void term(ll x) {
    constexpr ll F = k_frac(Q);
    constexpr int B = k_base(Q);
    m = madw(lo(x), hi(F), madw(hi(x), lo(F), m));
    h = madw(hi(x), hi(F), h);
    if (B > 0) h += x;
    if (B < 0) h -= x;
  }
  __device__ __forceinline__ void carry() {
    h += m >> 32;
    m &= 0xffffffffll;
  }
  __device__ __forceinline__ ll value() const { return h + (m >> 32); }
};
constexpr double k_abs(ll f) { return (f < 0 ? -(double)f : (double)f) / 18446744073709551616.0; }
// Whether output m's sum over j is carried after term j: always after every
// second one, and after the first of a pair whose fracs are too large.
template <int R, int M>
constexpr bool carry_after(int j) {
  if (j % 2 == 0) return true;
  const SC a = sincos_q62((j * M) % R, R), b = sincos_q62(((j + 1) * M) % R, R);
  return k_abs(k_frac(a.c)) + k_abs(k_frac(b.c)) > 0.7 || k_abs(k_frac(a.s)) + k_abs(k_frac(b.s)) > 0.7;
}
// Odd prime R from the symmetric pairs (as dev::dft_odd).  Outputs go to
// out(m, value) as they come, so that no second array of R values is live.
template <int R, class Out>
__device__ __forceinline__ void dft_odd(const I2* v, Out&& out) {
  constexpr int H = (R - 1) / 2;
  I2 t[H], u[H];
  const I2 a0 = v[0];
  I2 s0 = a0;
  dev::static_for<0, H>([&](auto J) {
    constexpr int j = decltype(J)::value + 1;
    t[j - 1] = add(v[j], v[R - j]);
    u[j - 1] = sub(v[j], v[R - j]);
    s0 = add(s0, t[j - 1]);
  });
  out(0, s0);
  dev::static_for<1, H + 1>([&](auto Mi) {
    constexpr int m = decltype(Mi)::value;
    Acc rx(a0.x), ry(a0.y), ix(0), iy(0);
    dev::static_for<1, H + 1>([&](auto J) {
      constexpr int j = decltype(J)::value;
      constexpr SC w = sincos_q62((j * m) % R, R);
      rx.template term<w.c>(t[j - 1].x);
      ry.template term<w.c>(t[j - 1].y);
      ix.template term<w.s>(u[j - 1].x);
      iy.template term<w.s>(u[j - 1].y);
      if (carry_after<R, m>(j) && j < H) {
        rx.carry();
        ry.carry();
        ix.carry();
        iy.carry();
      }
    });
    const ll a = rx.value(), b = ry.value(), c = ix.value(), d = iy.value();
    out(m, mk(a + d, b - c));
    out(R - m, mk(a - d, b + c));
  });
}
template <int R>
__device__ __forceinline__ void dft(I2* v);
// R = P Q: DFT_P over n1 of n = Q n1 + n2, W_R^(n2 k1), DFT_Q over n2
template <int R, int P>
__device__ __forceinline__ void dft_pq(I2* v) {
  constexpr int Q = R / P;
  I2 a[R];
  dev::static_for<0, Q>([&](auto I) {
    constexpr int n2 = decltype(I)::value;
    I2 t[P];
    dev::static_for<0, P>([&](auto J) { t[decltype(J)::value] = v[Q * decltype(J)::value + n2]; });
    dft<P>(t);
    dev::static_for<0, P>([&](auto K) {
      constexpr int k1 = decltype(K)::value;
      a[n2 * P + k1] = mul_root<R, n2 * k1>(t[k1]);
    });
  });
  dev::static_for<0, P>([&](auto K) {
    constexpr int k1 = decltype(K)::value;
    I2 u[Q];
    dev::static_for<0, Q>([&](auto I) { u[decltype(I)::value] = a[decltype(I)::value * P + k1]; });
    dft<Q>(u);
    dev::static_for<0, Q>([&](auto I) { v[k1 + P * decltype(I)::value] = u[decltype(I)::value]; });
  });
}
// R = P Q coprime, without twiddles (as dev::dftg)
template <int R, int P>
__device__ __forceinline__ void dft_coprime(I2* v) {
  constexpr int Q = R / P;
  I2 a[R];
  dev::static_for<0, Q>([&](auto I) {
    constexpr int n2 = decltype(I)::value;
    I2 t[P];
    dev::static_for<0, P>([&](auto J) { t[decltype(J)::value] = v[(Q * decltype(J)::value + P * n2) % R]; });
    dft<P>(t);
    dev::static_for<0, P>([&](auto K) { a[n2 * P + decltype(K)::value] = t[decltype(K)::value]; });
  });
  dev::static_for<0, P>([&](auto K) {
    constexpr int k1 = decltype(K)::value;
    I2 u[Q];
    dev::static_for<0, Q>([&](auto I) { u[decltype(I)::value] = a[decltype(I)::value * P + k1]; });
    dft<Q>(u);
    dev::static_for<0, Q>([&](auto I) { v[dev::crt(P, Q, k1, decltype(I)::value)] = u[decltype(I)::value]; });
  });
}
template <int R>
__device__ __forceinline__ void dft(I2* v) {
  if constexpr (R == 1) {
  } else if constexpr (R == 2) {
    const I2 a = v[0];
    v[0] = add(a, v[1]);
    v[1] = sub(a, v[1]);
  } else if constexpr (R == 3) {
    dft3p(v);
  } else if constexpr (R == 4) {
    dft4v(v[0], v[1], v[2], v[3]);
  } else if constexpr (R == 5) {
    dft5p(v);
  } else if constexpr (dev::coprime_part(R) != R) {
    dft_coprime<R, dev::coprime_part(R)>(v);
  } else if constexpr (R % 4 == 0) {
    dft_pq<R, 4>(v);
  } else if constexpr (R % 3 == 0) {
    dft_pq<R, 3>(v);
  } else {
    dft_odd<R>(v, [&](int m, I2 x) { v[m] = x; });
  }
}

// ---- between doubles and a line's integers ---------------------------------
// m: the largest magnitude's high word of a line; em = m >> 20 its biased
// exponent.  A finite line whose exponent lies in [kMinExp, kMaxExp] runs in
// integers: its results then neither overflow nor leave the normal range (the
// unit of a result lies at most 64 powers of two below the line's largest
// value, and a sum of 8192 moduli 14 above it).
constexpr int kMinExp = 80, kMaxExp = 1990;

__device__ __forceinline__ int abs_hi(double v) { return __double2hiint(v) & 0x7fffffff; }
__device__ __forceinline__ int max_hi(double2 v) { return max(fx::abs_hi(v.x), fx::abs_hi(v.y)); }
__device__ __forceinline__ int any_lo(double2 v) { return __double2loint(v.x) | __double2loint(v.y); }
// A value's share of the line's sum of moduli, over 2^(em - 1023), from the
// larger component's high word h: 20 mantissa bits as a float (an upward
// margin of 2^-17 a value covers the rest).
__device__ __forceinline__ float share(int h, int base) { return __int_as_float(max(h - base, 0) << 3); }
__device__ __forceinline__ int share_base(int em) { return (em - 127) << 20; }
__device__ __forceinline__ unsigned share_units(float sum, int count) {
  return (unsigned)(sum * 131072.0f) + (unsigned)count + 1;  // units of 2^(em - 1040)
}
// an integer as a double times 2^(adj >> 20), exponent and sign added to its
// high word unless that is zero (the result is normal or zero; `flip` =
// 0x80000000 negates)
__device__ __forceinline__ double to_double(ll v, int adj, int flip = 0) {
  const double d = __ll2double_rn(v);
  const unsigned h = (unsigned)__double2hiint(d);
  return __hiloint2double((int)(h + min(h, 1u) * ((unsigned)adj + (unsigned)flip)), __double2loint(d));
}

// A tile's scale words, in the kFxWordBytes a line at the end of its shared
// memory: a reference value, and for each of a line's one or two scales the
// largest high word, the sum of moduli and a mark.
struct Words {
  double2* ref;
  int *m, *far;
  unsigned* s;
  __device__ __forceinline__ Words(unsigned char* end, int L)
      : ref(reinterpret_cast<double2*>(end - (size_t)L * kFxWordBytes)),
        m(reinterpret_cast<int*>(ref + L)),
        far(m + 2 * L),
        s(reinterpret_cast<unsigned*>(far + 2 * L)) {}
  // zero but for the references
  __device__ __forceinline__ void clear(int L) const {
    for (int i = threadIdx.x + threadIdx.y * blockDim.x; i < 6 * L; i += blockDim.x * blockDim.y) m[i] = 0;
  }
};

// What a CTA's lines need, the same for all its threads.
enum class Found {
  yes,   // nothing
  fp64,  // a line must run in FP64
  flat   // a thread's values are all near its line's largest (FLAT: looked for)
};
template <bool FLAT>
__device__ __forceinline__ Found cta_found(int bad, int flat) {
  if (!__syncthreads_or(bad | flat)) return Found::yes;
  return FLAT && !__syncthreads_or(bad) ? Found::flat : Found::fp64;
}
constexpr int kNear = 1 << 18;  // of high words: 2^-3 to 2^-2 of a value
// Whether a thread's moduli, of high words up to `most` and, zeros passed over
// (places past a line's points hold them), from least + 1 on, are all near the
// line's largest, m.
__device__ __forceinline__ int near_all(int most, unsigned least, int m) {
  const int from = max(m - kNear, 1 << 20);
  return most >= from && least >= (unsigned)from - 1;
}

// The scale of a line, from the values its threads hold.
struct Scale {
  int m, em, es;  // largest high word, its exponent, exponent of the sum of moduli (over 2^em)
  // The line's scale words start at zero.
  template <bool FLAT, int Q>
  __device__ __forceinline__ Found find(const double2 (&x)[Q], int* smax, unsigned* ssum) {
    int most = 0;
    unsigned least = ~0u;
#pragma unroll
    for (int i = 0; i < Q; ++i) {
      most = max(most, max_hi(x[i]));
      least = min(least, (unsigned)max_hi(x[i]) - 1);
    }
    m = most;
    atomicMax(smax, m);
    __syncthreads();
    m = *smax;
    em = m >> 20;
    float sum = 0;
#pragma unroll
    for (int i = 0; i < Q; ++i) sum += share(max_hi(x[i]), share_base(em));
    atomicAdd(ssum, share_units(sum, Q));
    int bad = m != 0 && (em < kMinExp || em > kMaxExp);
    if (m == 0) {  // all zero, or subnormals below 2^-1042
#pragma unroll
      for (int i = 0; i < Q; ++i) bad |= any_lo(x[i]);
    }
    const Found f = cta_found<FLAT>(bad, FLAT && near_all(most, least, m));
    if (f != Found::yes) return f;
    const unsigned s = *ssum;
    es = 32 - __clz((int)(s + (s >> 1))) - 1040;  // a modulus is at most sqrt 2 times the larger component
    return f;
  }
  // Exponent (less em) that bounds the modulus of a sum of at most 2^lg
  // values, each raised by at most 2^grow: the sum of all, or 2^lg times the
  // largest.
  __device__ __forceinline__ int bound(int lg, int grow) const { return min(es, lg - 1021) + grow; }
  // The moduli may reach 2^62 where exponent `top` bounds them: the right
  // shift of a mantissa, less its exponent.  A zero line shifts all out.
  __device__ __forceinline__ int shift(int top) const { return m == 0 ? 4096 : 1021 + top + em; }
  // A result of a line that shares its transform: a zero line's is zero
  // whatever the other's rounding left there.
  __device__ __forceinline__ double out(ll v, int adj) const { return m == 0 ? 0.0 : to_double(v, adj); }
};

// The scales of the two real lines a, b that a complex line a + i b carries,
// each its own (their transforms separate exactly, so a small line next to a
// large one keeps its digits); of one line alone (`single`), the same twice.
struct PairScale {
  Scale a, b;
  // smax, ssum: two words each, at zero.  HALVES: x[2 i], x[2 i + 1] are
  // points of the lines' half spectra but for their bins 0, which lie in *dc;
  // else x[i] holds a point of a and b.
  template <bool HALVES, bool FLAT, int Q>
  __device__ __forceinline__ Found find(const double2 (&x)[Q], int* smax, unsigned* ssum, bool single = false,
                                        bool flat = true, const double2* dc = nullptr) {
    constexpr int S = HALVES ? 2 : 1;
    auto ha = [&](int i) { return HALVES ? max_hi(x[i]) : abs_hi(x[i].x); };
    auto hb = [&](int i) { return HALVES ? max_hi(x[i + 1]) : abs_hi(x[i].y); };
    int ma = 0, mb = 0;
    unsigned la = ~0u, lb = ~0u;
#pragma unroll
    for (int i = 0; i < Q; i += S) {
      ma = max(ma, ha(i));
      mb = max(mb, hb(i));
      la = min(la, (unsigned)ha(i) - 1);
      lb = min(lb, (unsigned)hb(i) - 1);
    }
    if (single) ma = mb = max(ma, mb);
    atomicMax(smax, ma);
    atomicMax(smax + 1, mb);
    __syncthreads();
    a.m = smax[0];
    b.m = smax[1];
    const double2 d = HALVES ? *dc : make_double2(0, 0);
    if (HALVES && a.m == 0) a.m = abs_hi(d.x);
    if (HALVES && b.m == 0) b.m = abs_hi(d.y);
    a.em = a.m >> 20;
    b.em = b.m >> 20;
    float sa = 0, sb = 0;
    const int ba = share_base(a.em), bb = share_base(b.em);
#pragma unroll
    for (int i = 0; i < Q; i += S) {
      sa += share(ha(i), ba);
      sb += share(hb(i), bb);
    }
    if (single) sa = sb = sa + sb;
    atomicAdd(ssum, share_units(sa, 2 * Q));
    atomicAdd(ssum + 1, share_units(sb, 2 * Q));
    int bad = outside(a) | outside(b);
    if constexpr (HALVES) bad |= max_hi(d) >> 20 > kMaxExp;
    if (a.m == 0 || b.m == 0) {  // all zero, or subnormals below 2^-1042
#pragma unroll
      for (int i = 0; i < Q; i += S) {
        if (a.m == 0) bad |= HALVES ? any_lo(x[i]) : __double2loint(x[i].x);
        if (b.m == 0) bad |= HALVES ? any_lo(x[i + 1]) : __double2loint(x[i].y);
      }
      if (a.m == 0) bad |= __double2loint(d.x);
      if (b.m == 0) bad |= __double2loint(d.y);
    }
    const Found f = cta_found<FLAT>(bad, FLAT && flat && (near_all(ma, la, a.m) | near_all(mb, lb, b.m)));
    if (f != Found::yes) return f;
    // a complex point's modulus is at most sqrt 2 times its larger component;
    // one bit for the other line: the moduli of a + i b sum to at most both
    const unsigned ta = ssum[0], tb = ssum[1];
    if constexpr (HALVES) {
      a.es = with_dc(ta, a.em, abs_hi(d.x));
      b.es = with_dc(tb, b.em, abs_hi(d.y));
    } else {
      a.es = 33 - __clz((int)ta) - 1040;
      b.es = 33 - __clz((int)tb) - 1040;
    }
    return f;
  }
  // ... of a half spectrum whose other bins sum to s units and bin 0 has high word h
  __device__ __forceinline__ static int with_dc(unsigned s, int em, int h) {
    const int over = (h >> 20) - em;
    if (over <= 10) s += share_units(share(h, share_base(em)), 1);
    const int es = 33 - __clz((int)(s + (s >> 1))) - 1040;
    return over <= 10 ? es : max(es, over - 1021) + 1;
  }
  __device__ __forceinline__ static int outside(const Scale& s) {
    return s.m != 0 && (s.em < kMinExp || s.em > kMaxExp);
  }
};

// x as an integer, rounded: 61 mantissa bits shifted right by sh - e (not
// negative).  One bit more is kept until the sign is in: w and ~w become
// w + 1 and -w, whose halves are x and -x rounded.  (Cutting the bits off
// instead shrinks every value the same way, which adds up where a line's
// values meet in one output.)  `flip` = 0x80000000 negates.
__device__ __forceinline__ ll to_fixed(double x, int sh, int flip = 0) {
  const int h = __double2hiint(x);
  const unsigned l = (unsigned)__double2loint(x);
  int s = sh - ((h & 0x7fffffff) >> 20);
  s = s < 63 ? s : 63;
  const int sg = (h ^ flip) >> 31;
  const unsigned mh = (__funnelshift_l(l, (unsigned)h, 9) & 0x1fffffffu) | 0x20000000u;
  const ll m = (ll)(((unsigned long long)(mh ^ (unsigned)sg) << 32) | ((l << 9) ^ (unsigned)sg));
  return ((m >> s) + 1) >> 1;
}
// Takes the mean off a thread's points of a line: its first value, in the
// components (c2c: real and imaginary part; else: lines) whose values all lie
// near that, zero in the others.
//
// On its own scale a mean would leave the rest of the line with the bits
// below it, where an FP64 transform of numbers of few digits cancels it
// exactly (101325 + 100 g of FP32 origin, 512 points, rel-L2 of all but bin 0:
// 1.4e-14, FP64 1.7e-16).  Within kNear the differences are exact, and a mean
// that stands out less costs no more bits than fixed point has to spare.  Only
// CTAs of which a thread saw nothing but near values come here, and scale
// their lines anew.  Thread `first` holds point 0 in x[0]; mine(i): the thread
// has a point in x[i]; the scale words are left cleared and the mean in w.ref.
template <int Q, class Mine>
__device__ __forceinline__ void take_means(double2 (&x)[Q], const Words& w, int line, bool first, Mine&& mine) {
  if (first) w.ref[line] = x[0];
  __syncthreads();
  const double2 r = w.ref[line];
  const int hx = __double2hiint(r.x), hy = __double2hiint(r.y);
  unsigned dx = 0, dy = 0;  // distances, kNear added
#pragma unroll
  for (int i = 0; i < Q; ++i)
    if (mine(i)) {
      dx = max(dx, (unsigned)(__double2hiint(x[i].x) - hx + kNear));
      dy = max(dy, (unsigned)(__double2hiint(x[i].y) - hy + kNear));
    }
  if (dx > 2 * kNear || abs_hi(r.x) < 1 << 20) w.far[2 * line] = 1;
  if (dy > 2 * kNear || abs_hi(r.y) < 1 << 20) w.far[2 * line + 1] = 1;
  __syncthreads();
  const double2 mean = make_double2(w.far[2 * line] ? 0.0 : r.x, w.far[2 * line + 1] ? 0.0 : r.y);
#pragma unroll
  for (int i = 0; i < Q; ++i)
    if (mine(i)) x[i] = make_double2(x[i].x - mean.x, x[i].y - mean.y);
  if (first) {
    w.ref[line] = mean;
    w.m[2 * line] = w.m[2 * line + 1] = 0;
    w.s[2 * line] = w.s[2 * line + 1] = 0;
  }
  __syncthreads();
}

// From the integers of a pass's complex line back to doubles: the exponent of
// each line's unit, in a high word, and the sign of the imaginary part.  A
// zero line that shares its transform is zero whatever the other's rounding
// left there.
template <int KIND>
struct Back {
  int adj_a, adj_b, flip;
  bool za, zb;
  bool off;             // the lines went without their
  const double2* mean;  // mean, which their n-point transform has in bin 0
  __device__ __forceinline__ void dc(double2& v, int n) const {
    v = make_double2(__fma_rn((double)n, mean->x, v.x), __fma_rn((double)n, mean->y, v.y));
  }
  __device__ __forceinline__ void dc(double2& va, double2& vb, int n) const {
    va.x = __fma_rn((double)n, mean->x, va.x);
    vb.x = __fma_rn((double)n, mean->y, vb.x);
  }
  // c2c, c2r: a point (c2r: of both lines)
  __device__ __forceinline__ double2 point(I2 v) const {
    return make_double2(za ? 0.0 : to_double(v.x, adj_a), zb ? 0.0 : to_double(v.y, adj_b, flip));
  }
  // r2c: points of the two half spectra, X1 = (Z_k + conj Z_{n-k}) / 2,
  // X2 = (Z_k - conj Z_{n-k}) / 2i, from Z_k and Z_{n-k}
  __device__ __forceinline__ double2 half_a(I2 zk, I2 zm) const { return half(zk.x + zm.x, zk.y - zm.y, adj_a, za); }
  __device__ __forceinline__ double2 half_b(I2 zk, I2 zm) const { return half(zk.y + zm.y, zm.x - zk.x, adj_b, zb); }
  __device__ __forceinline__ static double2 half(ll x, ll y, int adj, bool zero) {
    const int h = adj - (1 << 20);
    return zero ? make_double2(0.0, 0.0) : make_double2(to_double(x, h), to_double(y, h));
  }
};

// The scale of a pass's complex line and the way back from it: one scale for
// c2c, one for each of the two real lines of r2c and c2r.
//
// c2r: the half spectra go without their bins 0, which are real and join every
// output when the last stage adds them to its butterflies' inputs 0.  Bin 0
// of a field with a mean is far above the others; as one of them it would be
// what the early stages' sums are bounded by.
template <int KIND>
struct PassScale {
  static constexpr int X = KIND == K_C2R ? 1 : 0;  // a point combines two values
  PairScale p;  // c2c: p.a alone
  int ta = -1021 + X, tb = -1021 + X;
  bool off = false;
  const double2* mean;
  // False (for the whole CTA): a line must run in FP64.  w: cleared (c2r: the
  // bins 0 in its references); thread `first` of a line holds its point 0 in
  // x[0], mine(i): the thread has a point in x[i].
  template <int Q, class Mine>
  __device__ __forceinline__ bool find(double2 (&x)[Q], const Words& w, int line, bool first, Mine&& mine) {
    mean = &w.ref[line];
    int* m = w.m + 2 * line;
    unsigned* s = w.s + 2 * line;
    auto look = [&](auto flat) {
      constexpr bool FLAT = decltype(flat)::value;
      if constexpr (KIND == K_C2C) return p.a.find<FLAT>(x, m, s);
      else return p.find<KIND == K_C2R, FLAT>(x, m, s, false, true, mean);
    };
    Found f = look(std::integral_constant<bool, KIND != K_C2R>{});
    if (KIND != K_C2R && __builtin_expect(f == Found::flat, 0)) {
      take_means(x, w, line, first, mine);
      off = true;
      f = look(std::false_type{});
    }
    return f == Found::yes;
  }
  // stage of at most 2^lg summed inputs, divided by 2^shift so far; the last
  // one of c2r has bin 0 too
  __device__ __forceinline__ void stage(int lg, int shift, bool last) {
    if (KIND == K_C2R && last) lg = 4096;
    ta = max(ta, p.a.bound(lg, X) - shift);
    if constexpr (KIND != K_C2C) tb = max(tb, p.b.bound(lg, X) - shift);
  }
  // c2r: the bins 0 as what the last stage adds (conjugated, as its line is),
  // in the line's reference; thread `first` of a line, before a barrier
  __device__ __forceinline__ void set_dc(const Words& w, int line, int shift) const {
    const double2 d = w.ref[line];
    *reinterpret_cast<I2*>(&w.ref[line]) =
        mk(to_fixed(d.x, shift_a() + shift), to_fixed(d.y, shift_b() + shift, (int)0x80000000));
  }
  __device__ __forceinline__ void headroom() {
    ++ta;
    ++tb;
  }
  // right shifts of to_fixed for the two lines (c2c: components)
  __device__ __forceinline__ int shift_a() const { return p.a.shift(ta); }
  __device__ __forceinline__ int shift_b() const { return KIND == K_C2C ? p.a.shift(ta) : p.b.shift(tb); }
  __device__ __forceinline__ Back<KIND> back(int shift, int flip) const {
    Back<KIND> r;
    r.adj_a = (p.a.em - 62 + ta + shift) << 20;
    r.adj_b = KIND == K_C2C ? r.adj_a : (p.b.em - 62 + tb + shift) << 20;
    r.flip = flip;
    r.za = KIND != K_C2C && p.a.m == 0;
    r.zb = KIND != K_C2C && p.b.m == 0;
    r.off = off;
    r.mean = mean;
    return r;
  }
};

// The lines of a CTA that fixed point does not take, in FP64: as many lines
// at a time as two buffers of the CTA's shared memory hold.
template <int KIND, bool CONTIG>
__device__ __noinline__ void fallback(const PassArgs& a, double2* buf) {
  const int threads = blockDim.x * blockDim.y, tid = threadIdx.x + threadIdx.y * blockDim.x;
  const int G = a.L > 1 ? a.L / 2 : 1, tpl = threads / G;
  const int t = CONTIG ? tid % tpl : tid / G, line = CONTIG ? tid / tpl : tid % G;
  for (int g = 0; g < a.L; g += G) {
    dev::LineCtx<double, KIND, CONTIG> c;
    const long long cl = (long long)blockIdx.x * a.L + g + line;
    c.init_at(a, t, line, cl, CONTIG ? 0 : (long long)blockIdx.y, a.nlines);
    c.L = G;
    c.tpl = tpl;
    if (g + line >= a.L) c.valid = false;
    // threads left over by the division take no point
    if (t >= tpl || line >= G) {
      c.t = a.n;
      c.line = 0;
      c.valid = false;
    }
    dev::run_pp_lines<double, KIND, CONTIG>(c, a, buf, (size_t)a.n * G);
    __syncthreads();
  }
}

}  // namespace fx
}  // namespace gbfft
