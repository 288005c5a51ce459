// Fourier transforms of FP64 lines in 64-bit fixed point.
//
// The FP64 pipe of this part executes two operations a clock per SM, its
// integer pipes 16 32x32->64 multiply-adds and 64 or more 32-bit additions a
// clock (measured).  A butterfly is mostly additions, so a line transform
// whose values are 64-bit integers with one power-of-two scale per line takes
// about a seventh of the time of the same transform in FP64 instructions; and
// its 61 bits below the line's bound round less than FP64's 53 (the error of
// every line length against long double is measured by tests/fft_fix_check.cu).
//
// A line of L = N1 N2 complex values is transformed in two passes of N1- and
// N2-point transforms held in registers:
//   pass 1: thread b < N2 transforms the points b + N2 a (a < N1) and
//           multiplies output a' by w_L^(b a');
//   pass 2: thread a < N1 transforms the N2 values of row a; output b' is
//           point a + N1 b' of the line's transform.
// Lines are 3/2-dealiased: L = A B with A a multiple of 3.  The backward
// transform runs with N1 = A, where the zero padding (the middle third of
// the line) is the middle third of every thread's points; the forward
// transform with N2 = A, where the discarded middle third of the spectrum is
// that of every thread's outputs.
//
// Scale.  Every component of every intermediate value of pass 1 is at most
// the sum of |re| + |im| over the N1 points of its thread (bound B1, the
// largest such sum of the line), every one of pass 2 at most the sum S over
// the whole line.  The twiddle product returns a quarter of its value (the
// high 32 bits of a 2^62-scaled product come for free), so integers of 2^e x
// with e = min(61 - lg B1, 63 - lg S) never leave 62 bits.  The bounds are
// integer sums (order independent), so a transform's bits depend on its line
// only.
//
// Values: a line whose magnitudes are all below 2^-895 comes out zero; a line
// with an infinity, a NaN or a magnitude from 2^1009 comes out NaN throughout
// (an FP64 transform spreads NaN and infinities over most of the line).
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <type_traits>
#include <utility>
#include <vector>

namespace owt {

struct __align__(16) fxc {
  long long x, y;
};
// exp(-2 pi i k / L) = c - i s, c and s times 2^62 as high * 2^32 + low with a
// signed low word (never -2^31, so that both words can be negated)
struct __align__(16) FxTw {
  int c1, c0, s1, s0;
};

#define OWT_HD __host__ __device__ __forceinline__

OWT_HD long long fx_wide(int a, int b) { return (long long)a * (long long)b; }
// a = h 2^32 + l with l signed
OWT_HD void fx_split(long long a, int &h, int &l) {
  l = (int)a;
  h = (int)(a >> 32) - (l >> 31);
}
OWT_HD fxc fx_add(fxc a, fxc b) { return fxc{a.x + b.x, a.y + b.y}; }
OWT_HD fxc fx_sub(fxc a, fxc b) { return fxc{a.x - b.x, a.y - b.y}; }

// A real constant c as k 2^-64 + r, r = round(c) in {-1, 0, 1}.
struct FxConst {
  long long k;
  int r;
};
constexpr FxConst kFxSin60 = {-2471395088767036514ll, 1};   // sin 60
constexpr FxConst kFxRoot8 = {-5402926248376769404ll, 1};   // sqrt(1/2)
constexpr FxConst kFxRoot5q = {-8134700645620564469ll, 1};  // sqrt(5)/4
constexpr FxConst kFxSin72 = {-902847917979075853ll, 1};
constexpr FxConst kFxSin36 = {-7604019954369499282ll, 1};
constexpr FxConst kFxCos40 = {-4315718282406409839ll, 1};
constexpr FxConst kFxSin40 = {-6589405544070453923ll, 1};
constexpr FxConst kFxCos80 = {3203243492287910726ll, 0};
constexpr FxConst kFxSin80 = {-280247492088382768ll, 1};
constexpr FxConst kFxCos160 = {1112474790118499113ll, -1};
constexpr FxConst kFxSin160 = {6309158051982071155ll, 0};
constexpr FxConst kFxCos22 = {-1404174782535421627ll, 1};  // 22.5 degrees
constexpr FxConst kFxSin22 = {7059263338087549767ll, 0};

// a c, rounded: three 32x32->64 products (the low x low one is below half a
// unit and left out), the fraction of c in 2^-64, its integer part as +-a.
template <long long K, int R>
OWT_HD long long fx_mulk(long long a) {
  constexpr int k0 = (int)K;
  constexpr int k1 = (int)((K - (long long)k0) >> 32);
  int h, l;
  fx_split(a, h, l);
  const long long cr = fx_wide(l, k1) + (fx_wide(h, k0) + 0x80000000ll);
  long long t = fx_wide(h, k1);
  if (R == 1) t += a;
  if (R == -1) t -= a;
  return t + (cr >> 32);
}
#define OWT_FX_MULK(a, C) fx_mulk<C.k, C.r>(a)

// x (c - i s) / 4 (forward) or x (c + i s) / 4 (backward), rounded
template <bool BACKWARD>
OWT_HD fxc fx_twiddle(fxc x, FxTw w) {
  int xh, xl, yh, yl;
  fx_split(x.x, xh, xl);
  fx_split(x.y, yh, yl);
  const int s1 = BACKWARD ? -w.s1 : w.s1, s0 = BACKWARD ? -w.s0 : w.s0;
  const int n1 = -s1, n0 = -s0;
  const long long half = 0x80000000ll;
  const long long cr = fx_wide(xl, w.c1) + (fx_wide(xh, w.c0) + (fx_wide(yl, s1) + (fx_wide(yh, s0) + half)));
  const long long ci = fx_wide(yl, w.c1) + (fx_wide(yh, w.c0) + (fx_wide(xl, n1) + (fx_wide(xh, n0) + half)));
  return fxc{fx_wide(xh, w.c1) + fx_wide(yh, s1) + (cr >> 32), fx_wide(yh, w.c1) + fx_wide(xh, n1) + (ci >> 32)};
}
OWT_HD fxc fx_quarter(fxc x) { return fxc{(x.x + 2) >> 2, (x.y + 2) >> 2}; }

// multiply by -sign i: forward -i, backward +i
template <bool BACKWARD>
OWT_HD fxc fx_rot(fxc d) {
  return BACKWARD ? fxc{-d.y, d.x} : fxc{d.y, -d.x};
}

// x w_N^E for N = 8, 9, 16 (w_N = exp(-2 pi i/N) forward, its conjugate backward)
template <int E, int N, bool BACKWARD>
OWT_HD fxc fx_twc(fxc x) {
  constexpr int e = E % N;
  if constexpr (e == 0) {
    return x;
  } else if constexpr (2 * e == N) {
    return fxc{-x.x, -x.y};
  } else if constexpr (4 * e == N) {
    return fx_rot<BACKWARD>(x);
  } else if constexpr (8 * e == N) {  // 45 degrees
    const fxc r = fx_rot<BACKWARD>(x);
    return fxc{OWT_FX_MULK(x.x + r.x, kFxRoot8), OWT_FX_MULK(x.y + r.y, kFxRoot8)};
  } else if constexpr (8 * e == 3 * N) {  // 135 degrees
    const fxc r = fx_rot<BACKWARD>(x);
    return fxc{OWT_FX_MULK(r.x - x.x, kFxRoot8), OWT_FX_MULK(r.y - x.y, kFxRoot8)};
  } else {
    // x cos + (rotated x) sin, both with a sign folded in
    const fxc r = fx_rot<BACKWARD>(x);
    if constexpr (16 * e == N) {
      return fxc{OWT_FX_MULK(x.x, kFxCos22) + OWT_FX_MULK(r.x, kFxSin22),
                 OWT_FX_MULK(x.y, kFxCos22) + OWT_FX_MULK(r.y, kFxSin22)};
    } else if constexpr (16 * e == 3 * N) {
      return fxc{OWT_FX_MULK(x.x, kFxSin22) + OWT_FX_MULK(r.x, kFxCos22),
                 OWT_FX_MULK(x.y, kFxSin22) + OWT_FX_MULK(r.y, kFxCos22)};
    } else if constexpr (16 * e == 9 * N) {
      return fxc{-(OWT_FX_MULK(x.x, kFxCos22) + OWT_FX_MULK(r.x, kFxSin22)),
                 -(OWT_FX_MULK(x.y, kFxCos22) + OWT_FX_MULK(r.y, kFxSin22))};
    } else if constexpr (9 * e == N) {
      return fxc{OWT_FX_MULK(x.x, kFxCos40) + OWT_FX_MULK(r.x, kFxSin40),
                 OWT_FX_MULK(x.y, kFxCos40) + OWT_FX_MULK(r.y, kFxSin40)};
    } else if constexpr (9 * e == 2 * N) {
      return fxc{OWT_FX_MULK(x.x, kFxCos80) + OWT_FX_MULK(r.x, kFxSin80),
                 OWT_FX_MULK(x.y, kFxCos80) + OWT_FX_MULK(r.y, kFxSin80)};
    } else {
      static_assert(9 * e == 4 * N, "fx_twc: angle not tabulated");
      return fxc{OWT_FX_MULK(x.x, kFxCos160) + OWT_FX_MULK(r.x, kFxSin160),
                 OWT_FX_MULK(x.y, kFxCos160) + OWT_FX_MULK(r.y, kFxSin160)};
    }
  }
}

template <int B, int E, class F>
OWT_HD void fx_for(F &&f) {
  if constexpr (B < E) {
    f(std::integral_constant<int, B>{});
    fx_for<B + 1, E>(f);
  }
}

// N-point transform in place (unnormalised): 2, 3, 4, 5 written out; 8, 9, 16
// by decimation in time with the constants above; products of coprime
// factors by the Good-Thomas map n = N2 n1 + N1 n2, k = k1 mod N1, k2 mod N2
// (no twiddles): 6, 10, 12, 15, 18, 20, 24.
template <int N> struct FxCoprime { static constexpr int n1 = 0; };
template <> struct FxCoprime<6> { static constexpr int n1 = 2; };
template <> struct FxCoprime<10> { static constexpr int n1 = 2; };
template <> struct FxCoprime<12> { static constexpr int n1 = 4; };
template <> struct FxCoprime<15> { static constexpr int n1 = 3; };
template <> struct FxCoprime<18> { static constexpr int n1 = 2; };
template <> struct FxCoprime<20> { static constexpr int n1 = 4; };
template <> struct FxCoprime<24> { static constexpr int n1 = 8; };

constexpr int fx_crt(int k1, int n1, int k2, int n2) {
  for (int k = k1; k < n1 * n2; k += n1)
    if (k % n2 == k2) return k;
  return -1;
}

template <int N, bool BACKWARD>
OWT_HD void fx_dft(fxc *x) {
  if constexpr (N == 2) {
    const fxc a = x[0], b = x[1];
    x[0] = fx_add(a, b);
    x[1] = fx_sub(a, b);
  } else if constexpr (N == 3) {
    const fxc t = fx_add(x[1], x[2]), d = fx_sub(x[1], x[2]);
    const fxc m = fxc{x[0].x - (t.x >> 1), x[0].y - (t.y >> 1)};
    const fxc u = fx_rot<BACKWARD>(fxc{OWT_FX_MULK(d.x, kFxSin60), OWT_FX_MULK(d.y, kFxSin60)});
    x[0] = fx_add(x[0], t);
    x[1] = fx_add(m, u);
    x[2] = fx_sub(m, u);
  } else if constexpr (N == 4) {
    const fxc t0 = fx_add(x[0], x[2]), t1 = fx_sub(x[0], x[2]), t2 = fx_add(x[1], x[3]);
    const fxc t3 = fx_rot<BACKWARD>(fx_sub(x[1], x[3]));
    x[0] = fx_add(t0, t2);
    x[1] = fx_add(t1, t3);
    x[2] = fx_sub(t0, t2);
    x[3] = fx_sub(t1, t3);
  } else if constexpr (N == 5) {
    const fxc t1 = fx_add(x[1], x[4]), t2 = fx_add(x[2], x[3]);
    const fxc d1 = fx_rot<BACKWARD>(fx_sub(x[1], x[4])), d2 = fx_rot<BACKWARD>(fx_sub(x[2], x[3]));
    const fxc t = fx_add(t1, t2), e = fx_sub(t1, t2);
    const fxc m = fxc{x[0].x - (t.x >> 2), x[0].y - (t.y >> 2)};
    const fxc q = fxc{OWT_FX_MULK(e.x, kFxRoot5q), OWT_FX_MULK(e.y, kFxRoot5q)};
    const fxc a1 = fx_add(m, q), a2 = fx_sub(m, q);
    const fxc b1 = fxc{OWT_FX_MULK(d1.x, kFxSin72) + OWT_FX_MULK(d2.x, kFxSin36),
                       OWT_FX_MULK(d1.y, kFxSin72) + OWT_FX_MULK(d2.y, kFxSin36)};
    const fxc b2 = fxc{OWT_FX_MULK(d1.x, kFxSin36) - OWT_FX_MULK(d2.x, kFxSin72),
                       OWT_FX_MULK(d1.y, kFxSin36) - OWT_FX_MULK(d2.y, kFxSin72)};
    x[0] = fx_add(x[0], t);
    x[1] = fx_add(a1, b1);
    x[4] = fx_sub(a1, b1);
    x[2] = fx_add(a2, b2);
    x[3] = fx_sub(a2, b2);
  } else if constexpr (FxCoprime<N>::n1 != 0) {
    constexpr int N1 = FxCoprime<N>::n1, N2 = N / N1;
    fxc y[N1][N2];
    fx_for<0, N2>([&](auto c2) {
      constexpr int n2 = decltype(c2)::value;
      fxc z[N1];
      fx_for<0, N1>([&](auto c1) { z[decltype(c1)::value] = x[(N2 * decltype(c1)::value + N1 * n2) % N]; });
      fx_dft<N1, BACKWARD>(z);
      fx_for<0, N1>([&](auto c1) { y[decltype(c1)::value][n2] = z[decltype(c1)::value]; });
    });
    fx_for<0, N1>([&](auto c1) {
      constexpr int k1 = decltype(c1)::value;
      fx_dft<N2, BACKWARD>(y[k1]);
      fx_for<0, N2>([&](auto c2) {
        constexpr int k2 = decltype(c2)::value;
        constexpr int k = fx_crt(k1, N1, k2, N2);
        x[k] = y[k1][k2];
      });
    });
  } else {
    static_assert(N == 8 || N == 9 || N == 16, "fx_dft: length");
    constexpr int R = N == 9 ? 3 : N == 8 ? 2 : 4, M = N / R;
    fxc y[R][M];
    fx_for<0, R>([&](auto cr) {
      constexpr int r = decltype(cr)::value;
      fx_for<0, M>([&](auto cm) { y[r][decltype(cm)::value] = x[r + R * decltype(cm)::value]; });
      fx_dft<M, BACKWARD>(y[r]);
    });
    fx_for<0, M>([&](auto ck) {
      constexpr int k1 = decltype(ck)::value;
      fxc z[R];
      fx_for<0, R>([&](auto cr) {
        constexpr int r = decltype(cr)::value;
        z[r] = fx_twc<r * k1, N, BACKWARD>(y[r][k1]);
      });
      fx_dft<R, BACKWARD>(z);
      fx_for<0, R>([&](auto cr) { x[k1 + M * decltype(cr)::value] = z[decltype(cr)::value]; });
    });
  }
}

// ---------------------------------------------------------------------------
// FP64 <-> fixed point, by the IEEE-754 layout (integer instructions: the
// conversion instructions run on the FP64 pipe).
// ---------------------------------------------------------------------------
OWT_HD int fx_hi(long long bits) { return (int)(bits >> 32); }

// Bound of a set of doubles: its largest exponent field m and the sum of its
// magnitudes in units of 2^(m - 1043) (21-bit significands, each rounded up).
struct FxBound {
  int m;
  unsigned s;
};
template <int N>
OWT_HD FxBound fx_bound(const fxc *x) {  // x holds the bits of doubles
  int mh = 0;
  fx_for<0, N>([&](auto c) {
    const int a = fx_hi(x[decltype(c)::value].x) & 0x7fffffff, b = fx_hi(x[decltype(c)::value].y) & 0x7fffffff;
    mh = mh > a ? mh : a;
    mh = mh > b ? mh : b;
  });
  FxBound r{mh >> 20, 0u};
  auto add = [&](int hi) {
    const unsigned mant = ((unsigned)hi & 0xfffffu) | 0x100000u;
    const int sh = r.m - ((hi >> 20) & 0x7ff);
    r.s += (mant >> (sh < 31 ? sh : 31)) + 1u;
  };
  fx_for<0, N>([&](auto c) {
    add(fx_hi(x[decltype(c)::value].x));
    add(fx_hi(x[decltype(c)::value].y));
  });
  return r;
}

// Scale of a line from the bounds of its pass-1 threads.
struct FxScale {
  int rsh;      // a significand left-aligned at bit 62 with exponent field f goes right by rsh + 1 - f
  int e;        // integers are 2^e x; after pass 2 of the transform 2^(e - 2) x
  bool finite;  // false: an infinity, a NaN or a magnitude from 2^1009

};
// b(t), t < n: the bounds
template <class B>
OWT_HD FxScale fx_scale(int n, B b) {
  int m = 0;
  for (int t = 0; t < n; ++t) {
    const int v = b(t).m;
    m = m > v ? m : v;
  }
  unsigned s = 0, s1 = 0;
  for (int t = 0; t < n; ++t) {
    const FxBound q = b(t);
    const int sh = m - q.m;
    const unsigned v = (q.s >> (sh < 31 ? sh : 31)) + 1u;
    s += v;
    s1 = s1 > v ? s1 : v;
  }
#ifdef __CUDA_ARCH__
  const int lgs = 32 - __clz((int)s), lg1 = 32 - __clz((int)s1);
#else
  const int lgs = 32 - __builtin_clz(s), lg1 = 32 - __builtin_clz(s1);
#endif
  FxScale r;
  const int k1 = 61 - lg1, k2 = 63 - lgs;
  r.e = (k1 < k2 ? k1 : k2) + 1043 - m;
  // m in [128, 2032): the output exponents of fx_to_double stay within the
  // format and a zero element (field 0) is shifted out; other lines are
  // taken as zeros here
  r.finite = m < 2032;
  const bool live = m >= 128 && r.finite;
  r.rsh = live ? 62 + 1023 - r.e - 1 : 4096;
  if (!live) r.e = 0;
  return r;
}

// the double with these bits, times 2^e, to the nearest integer (ties away
// from zero); the line's scale keeps it within 62 bits.  Denormals give 0.
OWT_HD long long fx_from_bits(long long bits, const FxScale &s) {
  const int hi = fx_hi(bits);
  const long long m = ((bits & 0xfffffffffffffll) | 0x10000000000000ll) << 10;
  int sh = s.rsh - ((hi >> 20) & 0x7ff);
  sh = sh < 63 ? sh : 63;
  const long long v = (long long)((((unsigned long long)m >> sh) + 1ull) >> 1);
  const long long sg = (long long)(hi >> 31);
  return (v ^ sg) - sg;
}

// 2^k; 0 or infinity beyond the normal range
OWT_HD double fx_pow2(int k) {
  const int f = k < -1022 ? 0 : k > 1023 ? 0x7ff : k + 1023;
#ifdef __CUDA_ARCH__
  return __hiloint2double(f << 20, 0);
#else
  const long long b = (long long)f << 52;
  double d;
  __builtin_memcpy(&d, &b, 8);
  return d;
#endif
}
// Output factor of a line's integers after pass 2: value = n fx_factor(s);
// NaN for a line that is not finite.
OWT_HD double fx_factor(const FxScale &s) {
  const double nan = __builtin_nan("");
  return s.finite ? fx_pow2(2 - s.e) : nan;
}
// The same by the exponent field: one conversion and integer instructions.
struct FxOut {
  int dhi;       // 2 - e in the exponent field's place
  unsigned nan;  // 0, or the high word of a NaN
};
OWT_HD FxOut fx_out(const FxScale &s) { return s.finite ? FxOut{(2 - s.e) * (1 << 20), 0u} : FxOut{0, 0x7ff80000u}; }
#ifdef __CUDACC__
__device__ __forceinline__ double fx_to_double(long long n, FxOut o) {
  const double d = __ll2double_rn(n);
  const int hi = __double2hiint(d);
  return __hiloint2double((int)((unsigned)(hi ? hi + o.dhi : 0) | o.nan), __double2loint(d));
}
#endif

// ---------------------------------------------------------------------------
// Products of lines in physical space and the transform back, all in integers.
// A packed line holds one field on two neighbouring (y, z) lines: its integers
// after a transform are 2^k x with k = e - 2 and at most 62 bits.  Each field
// is shifted left to its own largest value, below 2^62; the high 64 bits of
// u o are then 2^(k_u + k_o - 64) times the real product, below 2^60.  (Two
// fields in one line would share a scale: w beside o_x, hundreds of times
// larger, lost its low bits, and the products' error rose to 1.45 times that
// of FP64 where o_x has a mean.)
// ---------------------------------------------------------------------------
OWT_HD long long fx_product(int ah, int al, int bh, int bl) {  // words of fx_split
  const long long cr = fx_wide(al, bh) + (fx_wide(ah, bl) + 0x80000000ll);
  return fx_wide(ah, bh) + (cr >> 32);
}
OWT_HD long long fx_shift_right(long long x, int d) {  // rounded, 0 <= d <= 62
  return (x + ((1ll << d) >> 1)) >> d;
}
// |high word| of a value or of the larger component, for a line's largest
OWT_HD unsigned fx_mag(long long v) {
  const int hi = fx_hi(v);
  return (unsigned)(hi ^ (hi >> 31));
}
OWT_HD unsigned fx_mag(fxc v) {  // (an OR has the same highest bit as the maximum)
  return fx_mag(v.x) | fx_mag(v.y);
}
OWT_HD int fx_bits_of(unsigned v) {  // position of the highest set bit, from 1; 0 for 0
#ifdef __CUDA_ARCH__
  return 32 - __clz((int)v);
#else
  return v ? 32 - __builtin_clz(v) : 0;
#endif
}
// k of a line after its transform; a line of zeros does not limit the scale
// of the products it enters.
OWT_HD int fx_k(const FxScale &s) { return s.rsh == 4096 ? 1 << 14 : s.e - 2; }
OWT_HD int fx_min(int a, int b) { return a < b ? a : b; }
// Left shifts of the fields u, v, w, ox, oy, oz, right shifts of the products
// and the scales k of lx = v oz - w oy, ly = w ox - u oz, lz = u oy - v ox.
struct FxProducts {
  int s[6];
  int v_oz, w_oy, w_ox, u_oz, u_oy, v_ox;
  int k[3];
};
// k, mag: the six lines' scales and largest magnitudes (fx_mag)
OWT_HD FxProducts fx_products(const int (&k)[6], const unsigned (&mag)[6]) {
  FxProducts p;
  int n[6];
  for (int f = 0; f < 6; ++f) {
    p.s[f] = 30 - fx_bits_of(mag[f]);
    n[f] = k[f] + p.s[f];
  }
  const int cx = fx_min(n[1] + n[5], n[2] + n[4]);
  const int cy = fx_min(n[2] + n[3], n[0] + n[5]);
  const int cz = fx_min(n[0] + n[4], n[1] + n[3]);
  p.v_oz = fx_min(n[1] + n[5] - cx, 62);
  p.w_oy = fx_min(n[2] + n[4] - cx, 62);
  p.w_ox = fx_min(n[2] + n[3] - cy, 62);
  p.u_oz = fx_min(n[0] + n[5] - cy, 62);
  p.u_oy = fx_min(n[0] + n[4] - cz, 62);
  p.v_ox = fx_min(n[1] + n[3] - cz, 62);
  p.k[0] = cx - 64;
  p.k[1] = cy - 64;
  p.k[2] = cz - 64;
  return p;
}
// The Lamb vector at one point: f the six fields in, l out.
OWT_HD void fx_lamb(const long long (&f)[6], const FxProducts &p, long long (&l)[3]) {
  int h[6], w[6];
  for (int i = 0; i < 6; ++i) fx_split(f[i] << p.s[i], h[i], w[i]);
  l[0] = fx_shift_right(fx_product(h[1], w[1], h[5], w[5]), p.v_oz) -
         fx_shift_right(fx_product(h[2], w[2], h[4], w[4]), p.w_oy);
  l[1] = fx_shift_right(fx_product(h[2], w[2], h[3], w[3]), p.w_ox) -
         fx_shift_right(fx_product(h[0], w[0], h[5], w[5]), p.u_oz);
  l[2] = fx_shift_right(fx_product(h[0], w[0], h[4], w[4]), p.u_oy) -
         fx_shift_right(fx_product(h[1], w[1], h[3], w[3]), p.v_ox);
}
// Bound of a thread's integers (below 2^62) in units of 2^38.
template <int N>
OWT_HD unsigned fx_bound_int(const fxc *x) {
  unsigned s = 0;
  auto add = [&](long long v) {
    const int hi = fx_hi(v);
    s += ((unsigned)(hi ^ (hi >> 31)) >> 6) + 1u;
  };
  fx_for<0, N>([&](auto c) {
    add(x[decltype(c)::value].x);
    add(x[decltype(c)::value].y);
  });
  return s;
}
// The line's scale for integers that are 2^k x, and the shift that gives it.
template <class B>
OWT_HD FxScale fx_scale_int(int n, B b, int k, bool finite, int &shift) {
  unsigned s = 0, s1 = 0;
  for (int t = 0; t < n; ++t) {
    const unsigned v = b(t);
    s += (v >> 5) + 1u;
    s1 = s1 > v ? s1 : v;
  }
#ifdef __CUDA_ARCH__
  const int lgs = 32 - __clz((int)s), lg1 = 32 - __clz((int)s1);
#else
  const int lgs = 32 - __builtin_clz(s), lg1 = 32 - __builtin_clz(s1);
#endif
  shift = fx_min(23 - lg1, 20 - lgs);
  FxScale r;
  r.rsh = 0;
  r.e = k + shift;
  r.finite = finite;
  return r;
}
OWT_HD long long fx_rescale(long long x, int left, int right) { return fx_shift_right(x, right) << left; }

// ---------------------------------------------------------------------------
// Lengths.  L = A B with A and B from the radices below, A a multiple of 3
// and the larger of the two as small as possible; the class is the register
// budget of its kernels.  Lengths without such a split (more than 576 points,
// or an odd power of three times 27, 25 times 15 or more) stay with the FP64
// kernels.
// ---------------------------------------------------------------------------
constexpr int kFxRadices[] = {2, 3, 4, 5, 6, 8, 9, 10, 12, 15, 16, 18, 20, 24};
constexpr int kFxClasses = 3;  // radices up to 12, 18, 24
struct FxPlan {
  int8_t A = 0, B = 0, T = 0, cls = -1;  // T: threads a line, the larger radix
};
inline FxPlan fx_plan(int L) {
  FxPlan p;
  for (int hi : kFxRadices)
    for (int lo : kFxRadices)
      if (hi >= lo && hi * lo == L) {
        p.A = (int8_t)(hi % 3 == 0 ? hi : lo);
        p.B = (int8_t)(L / p.A);
        p.T = (int8_t)hi;
        p.cls = (int8_t)(hi <= 12 ? 0 : hi <= 18 ? 1 : 2);
        return p;
      }
  return p;
}

// f(std::integral_constant<int, n>) for the radix n of a plan of class CLS.
template <int CLS, class F>
OWT_HD void fx_radix(int n, F &&f) {
#define OWT_FX_CASE(N) \
  case N:              \
    f(std::integral_constant<int, N>{}); \
    break;
  if constexpr (CLS == 0) {
    switch (n) {
      OWT_FX_CASE(2)
      OWT_FX_CASE(3)
      OWT_FX_CASE(4)
      OWT_FX_CASE(5)
      OWT_FX_CASE(6)
      OWT_FX_CASE(8)
      OWT_FX_CASE(9)
      OWT_FX_CASE(10)
      OWT_FX_CASE(12)
    }
  } else if constexpr (CLS == 1) {
    switch (n) {
      OWT_FX_CASE(5)
      OWT_FX_CASE(9)
      OWT_FX_CASE(10)
      OWT_FX_CASE(12)
      OWT_FX_CASE(15)
      OWT_FX_CASE(16)
      OWT_FX_CASE(18)
    }
  } else {
    switch (n) {
      OWT_FX_CASE(15)
      OWT_FX_CASE(16)
      OWT_FX_CASE(18)
      OWT_FX_CASE(20)
      OWT_FX_CASE(24)
    }
  }
#undef OWT_FX_CASE
}

// Entry k of a line length's twiddles, exp(-2 pi i k / L).
inline FxTw fx_tw_entry(int k, int L) {
  const long double th = 2.0L * 3.14159265358979323846264338327950288L * (long double)k / (long double)L;
  auto words = [](long double v, int &h, int &l) {
    long long q = llroundl(v * 4611686018427387904.0L);  // 2^62
    l = (int)(uint32_t)(uint64_t)q;
    if (l == INT32_MIN) l = -INT32_MAX;
    h = (int)((q - (long long)l) >> 32);
  };
  FxTw w;
  words(cosl(th), w.c1, w.c0);
  words(sinl(th), w.s1, w.s0);
  return w;
}
// The twiddle table of a plan: w_L^(a b) at a B + b (a < A, b < B) for the
// backward transforms, then at L + b A + a for the forward ones (pass-1 output
// slowest, thread fastest in both).  Angles beyond an eighth of the circle
// (where 4 divides L) come by symmetry: cosl and sinl in 128 bits are software
// on some hosts.
inline std::vector<FxTw> fx_twiddles(const FxPlan &p) {
  const int L = p.A * p.B;
  std::vector<FxTw> w((size_t)L), t((size_t)2 * L);
  const int direct = L % 4 == 0 ? L / 8 : L % 2 == 0 ? L / 4 : L / 2;  // the others follow by symmetry
  for (int k = 0; k <= direct; ++k) w[k] = fx_tw_entry(k, L);
  auto entry = [&](auto &self, int k) -> FxTw {
    if (k <= direct) return w[k];
    if (2 * k > L) {
      const FxTw e = self(self, L - k);
      return FxTw{e.c1, e.c0, -e.s1, -e.s0};
    }
    if (4 * k > L) {
      const FxTw e = self(self, L / 2 - k);
      return FxTw{-e.c1, -e.c0, e.s1, e.s0};
    }
    const FxTw e = self(self, L / 4 - k);
    return FxTw{e.s1, e.s0, e.c1, e.c0};
  };
  for (int a = 0; a < p.A; ++a)
    for (int b = 0; b < p.B; ++b) t[(size_t)a * p.B + b] = t[(size_t)L + (size_t)b * p.A + a] = entry(entry, a * b);
  return t;
}

}  // namespace owt
