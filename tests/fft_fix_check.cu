// Host check of the fixed-point line transforms (csrc/fft_fix.cuh): every
// length with a plan, both signs, four kinds of lines, against a direct
// transform in long double.  The relative L2 error must not exceed that of a
// mixed-radix FP64 transform (radices 4, 2, 3, 5, correctly rounded twiddles)
// on the same lines.  Then the ends of the range: scaled lines give the same
// digits, zero and tiny lines zeros, lines with an infinity, a NaN or a
// magnitude from 2^1009 NaN.
#include <cmath>
#include <complex>
#include <cstdio>
#include <cstring>
#include <limits>
#include <random>
#include <vector>

#include "fft_fix.cuh"

using namespace owt;
using cd = std::complex<double>;
using cl = std::complex<long double>;
static const long double kTwoPi = 2.0L * 3.14159265358979323846264338327950288L;

template <int CLS, bool BACKWARD>
static void line_of_class(const FxPlan p, const std::vector<cd> &in, std::vector<cd> &out) {
  const int A = BACKWARD ? p.A : p.B, B = BACKWARD ? p.B : p.A, L = A * B;
  std::vector<FxBound> bd(B);
  std::vector<fxc> S(L);
  auto load = [&](int b, int a) {
    fxc v;
    const double re = in[b + B * a].real(), im = in[b + B * a].imag();
    std::memcpy(&v.x, &re, 8);
    std::memcpy(&v.y, &im, 8);
    return v;
  };
  FxScale sc{};
  for (int pass = 0; pass < 2; ++pass) {
    if (pass == 1) sc = fx_scale(B, [&](int t) { return bd[t]; });
    for (int b = 0; b < B; ++b)
      fx_radix<CLS>(A, [&](auto n) {
        constexpr int N = decltype(n)::value;
        fxc x[N];
        for (int a = 0; a < N; ++a) x[a] = load(b, a);
        if (pass == 0) {
          bd[b] = fx_bound<N>(x);
          return;
        }
        for (int a = 0; a < N; ++a) x[a] = fxc{fx_from_bits(x[a].x, sc), fx_from_bits(x[a].y, sc)};
        fx_dft<N, BACKWARD>(x);
        S[b] = fx_quarter(x[0]);
        for (int a = 1; a < N; ++a) S[a * B + b] = fx_twiddle<BACKWARD>(x[a], fx_tw_entry(a * b, L));
      });
  }
  const double f = fx_factor(sc);
  for (int a = 0; a < A; ++a)
    fx_radix<CLS>(B, [&](auto n) {
      constexpr int N = decltype(n)::value;
      fxc y[N];
      for (int b = 0; b < N; ++b) y[b] = S[a * B + b];
      fx_dft<N, BACKWARD>(y);
      for (int b = 0; b < N; ++b) out[a + A * b] = cd((double)y[b].x * f, (double)y[b].y * f);
    });
}

template <bool BACKWARD>
static void fix_line(const std::vector<cd> &in, std::vector<cd> &out) {
  const FxPlan p = fx_plan((int)in.size());
  out.resize(in.size());
  if (p.cls == 0) line_of_class<0, BACKWARD>(p, in, out);
  else if (p.cls == 1) line_of_class<1, BACKWARD>(p, in, out);
  else line_of_class<2, BACKWARD>(p, in, out);
}

static std::vector<cl> g_w;  // exp(2 pi i k / L)
static void fp64_line(const cd *x, int n, int stride, cd *o, int sign, int L) {
  if (n == 1) {
    o[0] = x[0];
    return;
  }
  const int R = n % 4 == 0 ? 4 : n % 2 == 0 ? 2 : n % 3 == 0 ? 3 : 5, m = n / R;
  std::vector<cd> y(n);
  for (int r = 0; r < R; ++r) fp64_line(x + r * stride, m, stride * R, &y[r * m], sign, L);
  const cd I(0.0, sign);
  for (int k = 0; k < m; ++k) {
    cd z[5];
    for (int r = 0; r < R; ++r) {
      const cl w = g_w[(size_t)(r * k) * (L / n) % L];
      z[r] = r * k ? y[r * m + k] * cd((double)w.real(), sign * (double)w.imag()) : y[r * m + k];
    }
    if (R == 2) {
      o[k] = z[0] + z[1];
      o[k + m] = z[0] - z[1];
    } else if (R == 4) {
      const cd a = z[0] + z[2], b = z[0] - z[2], c = z[1] + z[3], d = (z[1] - z[3]) * I;
      o[k] = a + c;
      o[k + m] = b + d;
      o[k + 2 * m] = a - c;
      o[k + 3 * m] = b - d;
    } else if (R == 3) {
      const cd t = z[1] + z[2], d = (z[1] - z[2]) * (I * 0.86602540378443864676), q = z[0] - 0.5 * t;
      o[k] = z[0] + t;
      o[k + m] = q + d;
      o[k + 2 * m] = q - d;
    } else {
      const double c1 = 0.30901699437494742410, c2 = -0.80901699437494742410;
      const double s1 = 0.95105651629515357212, s2 = 0.58778525229247312917;
      const cd t1 = z[1] + z[4], t2 = z[2] + z[3], d1 = (z[1] - z[4]) * I, d2 = (z[2] - z[3]) * I;
      const cd a1 = z[0] + c1 * t1 + c2 * t2, a2 = z[0] + c2 * t1 + c1 * t2;
      const cd b1 = s1 * d1 + s2 * d2, b2 = s2 * d1 - s1 * d2;
      o[k] = z[0] + (t1 + t2);
      o[k + m] = a1 + b1;
      o[k + 4 * m] = a1 - b1;
      o[k + 2 * m] = a2 + b2;
      o[k + 3 * m] = a2 - b2;
    }
  }
}

int main() {
  std::mt19937_64 gen(20);
  std::normal_distribution<double> nd;
  int lengths = 0, bad = 0;
  double worst = 0.0;
  for (int L = 6; L <= 576; L += 3) {
    if (fx_plan(L).cls < 0) continue;
    ++lengths;
    g_w.resize(L);
    for (int k = 0; k < L; ++k) g_w[k] = cl(std::cos(kTwoPi * k / L), std::sin(kTwoPi * k / L));
    // white; decaying and padded, as a velocity's line; white and padded; one dominant mode
    for (int kind = 0; kind < 4; ++kind)
      for (int sign = -1; sign <= 1; sign += 2) {
        long double ef = 0, ed = 0;
        for (int rep = 0; rep < (L < 64 ? 12 : 3); ++rep) {
          std::vector<cd> x(L), f, o(L);
          for (int k = 0; k < L; ++k) {
            const int kk = k <= L / 2 ? k : L - k;
            const double amp = (kind == 1 || kind == 2) && kk > L / 3 ? 0.0 : kind == 1 ? 1.0 / (1 + kk * kk)
                               : kind == 3 && k == 0                  ? 1000.0
                                                                      : 1.0;
            x[k] = amp * cd(nd(gen), nd(gen));
          }
          if (sign > 0) fix_line<true>(x, f);
          else fix_line<false>(x, f);
          fp64_line(x.data(), L, 1, o.data(), sign, L);
          for (int k = 0; k < L; ++k) {
            cl s = 0;
            for (int j = 0; j < L; ++j) s += cl(x[j]) * (sign > 0 ? g_w[(j * k) % L] : std::conj(g_w[(j * k) % L]));
            ef += std::norm(cl(f[k]) - s);
            ed += std::norm(cl(o[k]) - s);
          }
        }
        const double ratio = (double)std::sqrt(ef / ed);
        worst = std::max(worst, ratio);
        if (!(ratio <= 1.0)) {
          ++bad;
          std::printf("length %d kind %d sign %d: error %.2f times that of FP64\n", L, kind, sign, ratio);
        }
      }
    // the ends of the range
    std::vector<cd> x(L), f0, f1;
    for (cd &v : x) v = cd(nd(gen), nd(gen));
    fix_line<true>(x, f0);
    for (int e : {900, -850}) {
      std::vector<cd> s(L);
      for (int k = 0; k < L; ++k) s[k] = cd(std::ldexp(x[k].real(), e), std::ldexp(x[k].imag(), e));
      fix_line<true>(s, f1);
      for (int k = 0; k < L; ++k)
        bad += std::ldexp(f1[k].real(), -e) != f0[k].real() || std::ldexp(f1[k].imag(), -e) != f0[k].imag();
    }
    for (double v : {0.0, -0.0, 1e-300, 4.9e-324}) {
      std::vector<cd> s(L, cd(v, -v));
      fix_line<false>(s, f1);
      for (const cd &q : f1) bad += q != cd(0.0, 0.0);
    }
    for (double v : {std::numeric_limits<double>::infinity(), std::numeric_limits<double>::quiet_NaN(), 1e307}) {
      std::vector<cd> s = x;
      s[L / 2] = cd(0.0, -v);
      fix_line<true>(s, f1);
      for (const cd &q : f1) bad += !std::isnan(q.real()) || !std::isnan(q.imag());
    }
  }
  std::printf("%d lengths, largest error %.2f times that of FP64, %d failures\n", lengths, worst, bad);
  return bad || lengths != 38 ? 1 : 0;
}
