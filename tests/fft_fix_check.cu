// Host check of the fixed-point line transforms (csrc/fft_fix.cuh): every
// length with a plan, both signs, four kinds of lines, against a direct
// transform in long double.  The relative L2 error must not exceed that of a
// mixed-radix FP64 transform (radices 4, 2, 3, 5, correctly rounded twiddles)
// on the same lines.  The products of six lines and their transform back are
// held to the same bound against FP64 products of FP64 transforms.  Then the
// ends of the range: scaled lines give the same
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

// One line's transform on load(point), as a block's threads run it; INT: the
// input is integers 2^k x.
template <bool BACKWARD, bool INT, class Load>
static FxScale transform(int L, Load load, int k, std::vector<fxc> &out) {
  const FxPlan p = fx_plan(L);
  const int A = BACKWARD ? p.A : p.B, B = BACKWARD ? p.B : p.A;
  std::vector<FxBound> bd(B);
  std::vector<fxc> S(L);
  out.resize(L);
  FxScale sc{};
  int shift = 0;
  auto run = [&](auto cls) {
    constexpr int CLS = decltype(cls)::value;
    for (int pass = 0; pass < 2; ++pass) {
      if (pass == 1) {
        if (INT) sc = fx_scale_int(B, [&](int t) { return bd[t].s; }, k, true, shift);
        else sc = fx_scale(B, [&](int t) { return bd[t]; });
      }
      for (int b = 0; b < B; ++b)
        fx_radix<CLS>(A, [&](auto n) {
          constexpr int N = decltype(n)::value;
          fxc x[N];
          for (int a = 0; a < N; ++a) x[a] = load(b + B * a);
          if (pass == 0) {
            if (INT) bd[b].s = fx_bound_int<N>(x);
            else bd[b] = fx_bound<N>(x);
            return;
          }
          const int left = std::max(shift, 0), right = std::max(-shift, 0);
          for (int a = 0; a < N; ++a)
            x[a] = INT ? fxc{fx_rescale(x[a].x, left, right), fx_rescale(x[a].y, left, right)}
                       : fxc{fx_from_bits(x[a].x, sc), fx_from_bits(x[a].y, sc)};
          fx_dft<N, BACKWARD>(x);
          S[b] = fx_quarter(x[0]);
          for (int a = 1; a < N; ++a) S[a * B + b] = fx_twiddle<BACKWARD>(x[a], fx_tw_entry(a * b, L));
        });
    }
    for (int a = 0; a < A; ++a)
      fx_radix<CLS>(B, [&](auto n) {
        constexpr int N = decltype(n)::value;
        fxc y[N];
        for (int b = 0; b < N; ++b) y[b] = S[a * B + b];
        fx_dft<N, BACKWARD>(y);
        for (int b = 0; b < N; ++b) out[a + A * b] = y[b];
      });
  };
  if (p.cls == 0) run(std::integral_constant<int, 0>{});
  else if (p.cls == 1) run(std::integral_constant<int, 1>{});
  else run(std::integral_constant<int, 2>{});
  return sc;
}

static fxc bits(cd z) {
  fxc v;
  const double re = z.real(), im = z.imag();
  std::memcpy(&v.x, &re, 8);
  std::memcpy(&v.y, &im, 8);
  return v;
}

template <bool BACKWARD>
static void fix_line(const std::vector<cd> &in, std::vector<cd> &out) {
  std::vector<fxc> n;
  const FxScale sc = transform<BACKWARD, false>((int)in.size(), [&](int i) { return bits(in[i]); }, 0, n);
  const double f = fx_factor(sc);
  out.resize(in.size());
  for (size_t i = 0; i < in.size(); ++i) out[i] = cd((double)n[i].x * f, (double)n[i].y * f);
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

// The Lamb vector's lines: six fields on two neighbouring lines from their
// spectra (a field's two lines per complex transform), u x omega, a component's
// two lines per transform back, against long double.  Returns the largest error
// over that of the same in FP64 with the FP64 kernels' packing: u + i v,
// w + i o_x, o_y + i o_z, l_x + i l_y of one line.
static double product_ratio(int L, const double amp[6], double decay, double mean, double mean_ox, std::mt19937_64 &gen) {
  std::normal_distribution<double> nd;
  const int H = L / 3;
  long double ef[3] = {}, ed[3] = {};
  std::vector<cd> f[2][6];
  std::vector<long double> ph[2][6];
  for (int rep = 0; rep < 2; ++rep) {
    for (int l = 0; l < 2; ++l) {
      for (int i = 0; i < 6; ++i) {
        f[l][i].resize(H);
        for (int k = 0; k < H; ++k) {
          f[l][i][k] = amp[i] * std::pow(1.0 + k, -decay) * cd(nd(gen), nd(gen));
          if (k == 0) f[l][i][k] = f[l][i][k].real();
        }
      }
      f[l][0][0] += mean;
      f[l][3][0] += mean_ox;
      for (int i = 0; i < 6; ++i) {
        ph[l][i].resize(L);
        for (int x = 0; x < L; ++x) {
          cl v = f[l][i][0].real();
          for (int k = 1; k < H; ++k) v += 2.0L * std::real(cl(f[l][i][k]) * g_w[(size_t)k * x % L]);
          ph[l][i][x] = v.real();
        }
      }
    }
    auto packed = [&](const std::vector<cd> &p, const std::vector<cd> &q) {
      std::vector<cd> z(L);
      for (int m = 0; m < L; ++m) {
        cd a, b;
        if (m < H) a = p[m], b = q[m];
        else if (m > L - H) a = std::conj(p[L - m]), b = std::conj(q[L - m]);
        z[m] = a + cd(0, 1) * b;
      }
      return z;
    };
    // fixed point
    std::vector<fxc> n[6], out[3];
    int k[6];
    unsigned mag[6] = {};
    for (int i = 0; i < 6; ++i) {
      const std::vector<cd> z = packed(f[0][i], f[1][i]);
      k[i] = fx_k(transform<true, false>(L, [&](int j) { return bits(z[j]); }, 0, n[i]));
      for (const fxc &v : n[i]) mag[i] |= fx_mag(v);
    }
    const FxProducts c = fx_products(k, mag);
    std::vector<fxc> p[3];
    for (int r = 0; r < 3; ++r) p[r].resize(L);
    for (int x = 0; x < L; ++x) {
      long long a[6], b[6], la[3], lb[3];
      for (int i = 0; i < 6; ++i) a[i] = n[i][x].x, b[i] = n[i][x].y;
      fx_lamb(a, c, la);
      fx_lamb(b, c, lb);
      for (int r = 0; r < 3; ++r) p[r][x] = fxc{la[r], lb[r]};
    }
    double fac[3];
    for (int r = 0; r < 3; ++r)
      fac[r] = fx_factor(transform<false, true>(L, [&](int j) { return p[r][j]; }, c.k[r], out[r]));
    for (int l = 0; l < 2; ++l) {
      // FP64
      std::vector<cd> d[3], d01(L), d2(L), q01(L), q2(L);
      for (int q = 0; q < 3; ++q) {
        const std::vector<cd> z = packed(f[l][2 * q], f[l][2 * q + 1]);
        d[q].resize(L);
        fp64_line(z.data(), L, 1, d[q].data(), 1, L);
      }
      for (int x = 0; x < L; ++x) {
        const double u = d[0][x].real(), v = d[0][x].imag(), w = d[1][x].real(), ox = d[1][x].imag(),
                     oy = d[2][x].real(), oz = d[2][x].imag();
        const volatile double t[6] = {v * oz, w * oy, w * ox, u * oz, u * oy, v * ox};
        d01[x] = cd(t[0] - t[1], t[2] - t[3]);
        d2[x] = t[4] - t[5];
      }
      fp64_line(d01.data(), L, 1, q01.data(), -1, L);
      fp64_line(d2.data(), L, 1, q2.data(), -1, L);
      const std::vector<long double> *P = ph[l];
      for (int m = 0; m < H; ++m)
        for (int r = 0; r < 3; ++r) {
          cl s = 0;
          for (int x = 0; x < L; ++x) {
            const long double lam = r == 0   ? P[1][x] * P[5][x] - P[2][x] * P[4][x]
                                    : r == 1 ? P[2][x] * P[3][x] - P[0][x] * P[5][x]
                                             : P[0][x] * P[4][x] - P[1][x] * P[3][x];
            s += lam * std::conj(g_w[(size_t)m * x % L]);
          }
          const int mc = m ? L - m : 0;
          const fxc zm = out[r][m], zc = out[r][mc];
          const double w = 0.5 * fac[r];
          const cd a = l ? cd((double)(zm.y + zc.y) * w, (double)(zc.x - zm.x) * w)
                         : cd((double)(zm.x + zc.x) * w, (double)(zm.y - zc.y) * w);
          const cd qm = r < 2 ? q01[m] : q2[m], qc = r < 2 ? q01[mc] : q2[mc];
          const cd b = r == 1 ? cd((qm.imag() + qc.imag()) * 0.5, (qc.real() - qm.real()) * 0.5)
                              : cd((qm.real() + qc.real()) * 0.5, (qm.imag() - qc.imag()) * 0.5);
          ef[r] += std::norm(cl(a) - s);
          ed[r] += std::norm(cl(b) - s);
        }
    }
  }
  double worst = 0.0;
  for (int r = 0; r < 3; ++r) worst = std::max(worst, (double)std::sqrt(ef[r] / ed[r]));
  return worst;
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
  // white fields; a channel's core (mean flow, vorticity 20 times the velocity
  // fluctuations), two decays; next to the wall (shear, v and w small);
  // a mean o_x in the line that w shares
  const double one[6] = {1, 1, 1, 1, 1, 1}, core[6] = {0.1, 0.05, 0.05, 2, 2, 2}, wall[6] = {0.1, 0.001, 1e-5, 50, 50, 80};
  for (int L : {48, 192, 480, 576}) {
    g_w.resize(L);
    for (int k = 0; k < L; ++k) g_w[k] = cl(std::cos(kTwoPi * k / L), std::sin(kTwoPi * k / L));
    const double r[5] = {product_ratio(L, one, 0.0, 0.0, 0.0, gen), product_ratio(L, core, 1.0, 1.3, 0.0, gen),
                         product_ratio(L, core, 2.0, 1.3, 0.0, gen), product_ratio(L, wall, 1.0, 1.3, 0.0, gen),
                         product_ratio(L, core, 2.0, 1.3, 30.0, gen)};
    std::printf("products on lines of %d: error %.2f %.2f %.2f %.2f %.2f times that of FP64\n", L, r[0], r[1], r[2], r[3], r[4]);
    for (double x : r) bad += !(x <= 1.0);
  }
  return bad || lengths != 38 ? 1 : 0;
}
