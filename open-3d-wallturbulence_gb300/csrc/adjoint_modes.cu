// Adjoint of the mode kernel (src/solver.cpp:541-627 backwards, per mode):
// solve_horizontal^T, the transposed solves of the v- and omega_y-systems on
// the forward factors, and the source assembly^T into the three history
// levels.  The v solve also yields d objective / d v_w from the two wall rows.
//
//  k_adj_modes_stream : the mapping and the packed factor streams of
//    modes_stream.cuh, an omega_y and a v warp per 16 unique modes and sign of
//    kz.  The transposed sweeps need the same entries in the opposite order:
//    U^T reads the backward sweep's stream from its end, L^T the forward
//    sweep's.  The two systems' parts read and write disjoint data and need no
//    barrier.
//  k_adj_modes : the full band, for the dense solves.
//
// Right-hand sides, forward-swept values and solutions share one scratch row
// per unknown; the source's adjoint is gathered node by node from the last node
// down (adj_v_sources, adj_g_sources) instead of added to memory per row.
// Bound by FP64 issue like the forward kernel.  128x129x128, on the band
// storage -> here: 2.43 -> 1.14 ms.
#include <cuda_runtime.h>

#include "adjoint_kernels.h"
#include "modes_stream.cuh"

namespace owt {

namespace {

// levels l of the histories' weights: alpha (velocities), beta (sources)
constexpr double kAl0 = 3.0, kAl1 = -1.5, kAl2 = 1.0 / 3.0, kBe0 = 3.0, kBe1 = -3.0, kBe2 = 1.0;

struct AdjMode {
  bool horiz;
  // i ax z has the component c = sax times the other component of z, ...
  double sax, saz, skx, skz, k2;
  size_t e0, eo, row;  // this and the other component of row 0; between rows
};
__device__ __forceinline__ AdjMode adj_mode(const AdjModeArgs &a, const StrLane &L) {
  AdjMode c;
  const int k = L.m / a.NXH;
  const double kx = a.kx[L.m - k * a.NXH], kz = a.kz[k];
  c.k2 = fma(kx, kx, kz * kz);
  c.horiz = !(c.k2 < 1.e-8);
  const double ik2 = c.horiz ? 1.0 / c.k2 : 0.0, sgn = L.comp ? -1.0 : 1.0;
  c.sax = sgn * (kx * ik2);
  c.saz = sgn * (kz * ik2);
  c.skx = sgn * kx;
  c.skz = sgn * kz;
  c.e0 = 2 * (size_t)L.m + L.comp;
  c.eo = 2 * (size_t)L.m + 1 - L.comp;
  c.row = 2 * (size_t)a.M;
  return c;
}
__device__ __forceinline__ const double *comps(const double2 *f) { return reinterpret_cast<const double *>(f); }
__device__ __forceinline__ double *comps(double2 *f) { return reinterpret_cast<double *>(f); }

// Adjoints of the v solve's unknowns: v, and D1 v through DY1 v = c11 d1,
// DY2 v = c21 d1 + c22 d2, with the adjoint (forward: u = i ax DY1v - i az g,
// w = i ax g + i az DY1v, om_x = i/k2 (kx DY1g + kz DY2v) - i kz v,
// om_z = i/k2 (kz DY1g - kx DY2v) + i kx v).  put(c, value) for every column.
template <class Put>
__device__ __forceinline__ void adj_v_inputs(const AdjModeArgs &a, const AdjMode &c, Put put) {
  const int NY = a.NY;
  const double *in[7] = {comps(a.vb) + c.e0,  comps(a.v[0]) + c.e0, comps(a.q[0]) + c.e0, comps(a.ub) + c.eo,
                         comps(a.wb) + c.eo, comps(a.oxb) + c.eo,  comps(a.ozb) + c.eo};
  double x[7];
#pragma unroll
  for (int i = 0; i < 7; ++i) x[i] = in[i][0];
#pragma unroll 2
  for (int j = 0; j < NY; ++j) {
    double f[7];
    const size_t at = (size_t)(j + 1 < NY ? j + 1 : NY - 1) * c.row;
#pragma unroll
    for (int i = 0; i < 7; ++i) {
      f[i] = x[i];
      x[i] = in[i][at];
    }
    double v = f[1] + f[0], q = f[2], dv = 0.0;
    if (c.horiz) {
      dv = fma(c.sax, f[3], c.saz * f[4]);
      q += fma(c.saz, f[5], -(c.sax * f[6]));
      v += fma(c.skx, f[6], -(c.skz * f[5]));
    }
    put(vcol(0, j, NY), v);
    put(vcol(1, j, NY), a.inv_h * fma(a.c11[j], dv, a.c21[j] * q));
    put(vcol(2, j, NY), __dmul_rn(a.inv_h2 * a.c22[j], q));
    put(vcol(3, j, NY), 0.0);
    if (j < 2 || j >= NY - 2) put(vcol(4, j, NY), 0.0);
  }
}

// Adjoints of the omega_y solve's unknowns (g = icg (s + nu c21 d1 + nu c22 d2)
// inside) and the part of source_g's that comes from g itself: put, put_s.
template <class Put, class PutS>
__device__ __forceinline__ void adj_g_inputs(const AdjModeArgs &a, const AdjMode &c, double icg, Put put, PutS put_s) {
  const int NY = a.NY;
  const double *in[6] = {comps(a.gb) + c.e0, comps(a.g[0]) + c.e0, comps(a.ub) + c.eo,
                         comps(a.wb) + c.eo, comps(a.oxb) + c.eo,  comps(a.ozb) + c.eo};
  double x[6];
#pragma unroll
  for (int i = 0; i < 6; ++i) x[i] = in[i][0];
#pragma unroll 2
  for (int j = 0; j < NY; ++j) {
    double f[6];
    const size_t at = (size_t)(j + 1 < NY ? j + 1 : NY - 1) * c.row;
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      f[i] = x[i];
      x[i] = in[i][at];
    }
    double g = f[1] + f[0], dg = 0.0;
    if (c.horiz) {
      g += fma(c.sax, f[3], -(c.saz * f[2]));
      dg = fma(c.sax, f[4], c.saz * f[5]);
    }
    const bool inside = j != 0 && j != NY - 1;
    const double gi = inside ? __dmul_rn(icg, g) : 0.0;
    put(2 * j, a.inv_h * fma(a.c11[j], dg, a.nu * a.c21[j] * gi));
    put(2 * j + 1, __dmul_rn(a.inv_h2 * a.nu * a.c22[j], gi));
    put_s(j, gi);
  }
}

// level 1 += c0 s, level 2 += c1 s, level 0 = c2 s at node j; x1, x2: levels 1, 2
__device__ __forceinline__ void adj_update(double2 *const *f, size_t e, double x1, double x2, double s, double c0, double c1,
                                           double c2) {
  comps(f[1])[e] = fma(c0, s, x1);
  comps(f[2])[e] = fma(c1, s, x2);
  comps(f[0])[e] = c2 * s;
}

// source_v's adjoint from the solution z(p) through the rows' tables (row
// scale rs(e) of listed row e), then into Hv, v and DY2 v; the wall rows'
// gradient.  source_v = sum beta Hv_l - k^2/dt sum alpha v_l + sum alpha q_l/dt
// on nodes 2 .. NY - 3; the tables reference no other node.
template <class Z, class Rs>
__device__ __forceinline__ void adj_v_sources(const AdjModeArgs &a, const StrLane &L, const AdjMode &c, Z z, Rs rs) {
  const int NY = a.NY;
  for (int p = 0; p < a.n_v; ++p) {
    const int tag = a.rhs_node_v[p];
    if (tag != kRhsWallBottom && tag != kRhsWallTop) continue;
    const double r = __dmul_rn(z(p), a.rs_v[(size_t)p * a.U + L.u]);
    double *gr = comps(a.grad) + (tag == kRhsWallBottom ? c.e0 : c.row + c.e0);
    if (L.active) *gr += r;
  }
  int e = a.vptr[NY] - 1;
  double zn = e >= 0 ? z(a.vrows[e].p) : 0.0, rn = e >= 0 ? rs(e) : 0.0;  // the next listed row's
  double acc[3] = {0.0, 0.0, 0.0};                                        // nodes j - 2 .. j
  double2 *const *const f[3] = {a.hv, a.v, a.q};
  double x[6];
#pragma unroll
  for (int i = 0; i < 6; ++i) x[i] = comps(f[i / 2][1 + i % 2])[(size_t)(NY - 1) * c.row + c.e0];
  const double idt = a.inv_dt, mk2 = -c.k2 * idt;
#pragma unroll 2
  for (int j = NY - 1; j >= 0; --j) {
    double y[6];
    const size_t at = (size_t)(j > 0 ? j - 1 : 0) * c.row + c.e0;
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      y[i] = x[i];
      if (j > 0) x[i] = comps(f[i / 2][1 + i % 2])[at];
    }
    for (const int first = a.vptr[j]; e >= first; --e) {
      const StrRow &w = a.vrows[e];
      const double r = __dmul_rn(zn, rn);
      if (e > 0) {
        zn = z(a.vrows[e - 1].p);
        rn = rs(e - 1);
      }
#pragma unroll
      for (int i = 0; i < 3; ++i) acc[i] = fma(w.w[2 + i], r, acc[i]);
    }
    const double s = acc[2];
    if (L.active) {
      const size_t o = (size_t)j * c.row + c.e0;
      adj_update(a.hv, o, y[0], y[1], s, kBe0, kBe1, kBe2);
      adj_update(a.v, o, y[2], y[3], mk2 * s, kAl0, kAl1, kAl2);
      adj_update(a.q, o, y[4], y[5], idt * s, kAl0, kAl1, kAl2);
    }
    acc[2] = acc[1];
    acc[1] = acc[0];
    acc[0] = 0.0;
  }
}

// source_g's adjoint: s0(j) and the rows' part, into Hg and g.
template <class Z, class Rs, class S0>
__device__ __forceinline__ void adj_g_sources(const AdjModeArgs &a, const StrLane &L, const AdjMode &c, Z z, Rs rs, S0 s0) {
  const int NY = a.NY;
  int e = a.gptr[NY] - 1;
  double zn = e >= 0 ? z(a.grows[e].p) : 0.0, rn = e >= 0 ? rs(e) : 0.0;
  double acc[5];  // nodes j - 4 .. j
#pragma unroll
  for (int i = 0; i < 5; ++i) acc[i] = NY - 5 + i >= 0 ? s0(NY - 5 + i) : 0.0;
  double2 *const *const f[2] = {a.hg, a.g};
  double x[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) x[i] = comps(f[i / 2][1 + i % 2])[(size_t)(NY - 1) * c.row + c.e0];
  const double idt = a.inv_dt;
#pragma unroll 2
  for (int j = NY - 1; j >= 0; --j) {
    double y[4];
    const size_t at = (size_t)(j > 0 ? j - 1 : 0) * c.row + c.e0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      y[i] = x[i];
      if (j > 0) x[i] = comps(f[i / 2][1 + i % 2])[at];
    }
    const double sn = j >= 5 ? s0(j - 5) : 0.0;
    for (const int first = a.gptr[j]; e >= first; --e) {
      const StrRow &w = a.grows[e];
      const double r = __dmul_rn(zn, rn);
      if (e > 0) {
        zn = z(a.grows[e - 1].p);
        rn = rs(e - 1);
      }
#pragma unroll
      for (int i = 0; i < 5; ++i)
        if (i != 2 || nonzero(w.w[2])) acc[i] = fma(w.w[i], r, acc[i]);
    }
    const double s = acc[4];
    if (L.active) {
      const size_t o = (size_t)j * c.row + c.e0;
      adj_update(a.hg, o, y[0], y[1], s, kBe0, kBe1, kBe2);
      adj_update(a.g, o, y[2], y[3], idt * s, kAl0, kAl1, kAl2);
    }
#pragma unroll
    for (int i = 4; i > 0; --i) acc[i] = acc[i - 1];
    acc[0] = sn;
  }
}

// U^T y = b, columns 0 .. n - 1, on the backward sweep's stream: y_c = (b_c -
// sum_t U(c - t, c) y_(c-t)) / U(c, c).  rows as str_forward.
template <class S>
__device__ __forceinline__ void str_transposed_u(const double *stream, int n, double *ring, int lane, double *rows) {
  using Y = StrLayout<S>;
  constexpr int KV = S::KV;
  // values before an interior quad that its masks reach
  constexpr auto reach = [](int s) {  // column 3 - s of the quad
    int t = 0;
    for (int b = 1; b <= KV; ++b)
      if ((Y::mask_b(s) >> b) & 1ull) t = b;
    return t - (3 - s);
  };
  constexpr int R01 = reach(0) > reach(1) ? reach(0) : reach(1), R23 = reach(2) > reach(3) ? reach(2) : reach(3);
  constexpr int R = R01 > R23 ? R01 : R23, WI = R > 4 ? R : 4;
  const int lo = Y::lo(n), nq = Y::quads(n), q = lane >> 1;
  StrFeedBack<Y::slot> feed(stream + Y::bwd_size(n), ring, lane);
  const int units = lo + Y::hi(n) + nq;
  auto fetch = [&](int i) {
    if (i >= lo && i < lo + nq) feed.template fetch<Y::IB>();
    else if (i < units) feed.template fetch<Y::EB>();
    else feed.template fetch<0>();
  };
  fetch(0);
  fetch(1);
  auto row = [&](int p) { return p < n ? rows[32 * p] : 0.0; };
  double h[KV];  // y_(c - 1), y_(c - 2), ...
#pragma unroll
  for (int t = 0; t < KV; ++t) h[t] = 0.0;
  double in[4];
#pragma unroll
  for (int t = 0; t < 4; ++t) in[t] = row(t);
  int c = 0, unit = 0;
  auto edge = [&](int count) {
#pragma unroll 1
    for (int e = 0; e < count; ++e, ++c, ++unit) {
      const double *f = feed.ready();
      fetch(unit + 2);
      f += q;
      double acc = in[0];
#pragma unroll
      for (int t = 0; t < 3; ++t) in[t] = in[t + 1];
      in[3] = row(c + 4);
#pragma unroll
      for (int t = 1; t <= KV; ++t) fms(acc, f[t * 16], h[t - 1]);
      acc *= f[0];
      rows[32 * c] = acc;
#pragma unroll
      for (int t = KV - 1; t > 0; --t) h[t] = h[t - 1];
      h[0] = acc;
    }
  };
  edge(lo);
  if (nq > 0) {
#pragma unroll 1
    for (int e = 0; e < nq; ++e, c += 4, ++unit) {
      const double *f = feed.ready();
      fetch(unit + 2);
      f += q;
      double y[4];
      fx_for<0, 4>([&](auto kc) {
        constexpr int k = decltype(kc)::value, s = 3 - k;
        constexpr unsigned long long m = Y::mask_b(s);
        double acc = in[k];
        in[k] = row(c + 4 + k);
        fx_for<1, KV + 1>([&](auto tc) {
          constexpr int t = decltype(tc)::value;
          if constexpr ((m >> t) & 1ull) {
            const double l = f[(Y::before_b(s) + bits_below(m, t)) * 16];
            if constexpr (t <= k) fms(acc, l, y[k - t]);
            else fms(acc, l, h[t - k - 1]);
          }
        });
        y[k] = acc * f[Y::before_b(s) * 16];
        rows[32 * (c + k)] = y[k];
      });
#pragma unroll
      for (int t = WI - 1; t >= 4; --t) h[t] = h[t - 4];
#pragma unroll
      for (int t = 0; t < 4; ++t) h[t] = y[3 - t];
    }
#pragma unroll
    for (int t = WI; t < KV; ++t) h[t] = rows[32 * (c - 1 - t)];
    edge(Y::hi(n));
  }
  str_wait<0>();
  __syncwarp();
}

// L^T and the interchanges, columns n - 1 .. 0, on the forward sweep's stream:
// b_c -= sum_i L(c + i, c) b_(c+i), then interchange c undone.  rows: y on
// entry, the solution on return.
template <class S>
__device__ __forceinline__ void str_transposed_l(const double *stream, int n, double *ring, int lane, double *rows) {
  using Y = StrLayout<S>;
  constexpr int KL = S::KL, W = S::WF;
  static_assert(KL < W, "window");
  const int hi = Y::hi(n) + (Y::quads(n) ? 0 : Y::lo(n)), nq = Y::quads(n), q = lane >> 1;
  StrFeedBack<Y::slot> feed(stream + Y::fwd_size(n), ring, lane);
  const int units = Y::lo(n) + Y::hi(n) + nq;
  auto fetch = [&](int i) {
    if (i >= hi && i < hi + nq) feed.template fetch<Y::IF>();
    else if (i < units) feed.template fetch<Y::EF>();
    else feed.template fetch<0>();
  };
  fetch(0);
  fetch(1);
  auto row = [&](int p) { return p >= 0 ? rows[32 * p] : 0.0; };
  double w[W];  // b_c, b_(c+1), ...
#pragma unroll
  for (int t = 0; t < W; ++t) w[t] = 0.0;
  double in[4];
#pragma unroll
  for (int t = 0; t < 4; ++t) in[t] = row(n - 1 - t);
  int c = n - 1, unit = 0;
  auto edge = [&](int count) {
#pragma unroll 1
    for (int e = 0; e < count; ++e, --c, ++unit) {
      const double *f = feed.ready();
      fetch(unit + 2);
      if (c + W < n) rows[32 * (c + W)] = w[W - 1];
#pragma unroll
      for (int t = W - 1; t > 0; --t) w[t] = w[t - 1];
      w[0] = in[0];
#pragma unroll
      for (int t = 0; t < 3; ++t) in[t] = in[t + 1];
      in[3] = row(c - 4);
      const int off = (int)reinterpret_cast<const unsigned *>(f)[q];
      f += 16 + q;
#pragma unroll
      for (int i = 1; i <= KL; ++i) fms(w[0], f[(i - 1) * 16], w[i]);
      if (off) {
#pragma unroll
        for (int i = 1; i <= KL; ++i)
          if (off == i) {
            const double tmp = w[0];
            w[0] = w[i];
            w[i] = tmp;
          }
      }
    }
  };
  edge(hi);
  if (nq > 0) {
#pragma unroll 1
    for (int e = 0; e < nq; ++e, c -= 4, ++unit) {
      const double *f = feed.ready();
      fetch(unit + 2);
      double *o = rows + 32 * (c + 1);  // w[t] is entry c + 1 + t, below n: the upper edge has more columns than W
#pragma unroll
      for (int t = W - 4; t < W; ++t) o[32 * t] = w[t];
#pragma unroll
      for (int t = W - 1; t >= 4; --t) w[t] = w[t - 4];
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        w[3 - t] = in[t];
        in[t] = row(c - 4 - t);
      }
      const unsigned off = reinterpret_cast<const unsigned *>(f)[q];
      f += 16 + q;
      fx_for<0, 4>([&](auto kc) {
        constexpr int s = 3 - decltype(kc)::value;
        constexpr unsigned long long ml = Y::mask_f(s), mp = S::p(Y::type_f(s));
        static_assert((ml >> (W - s)) == 0 && (mp >> (W - s)) == 0, "window too short for the masks");
        fx_for<1, KL + 1>([&](auto ic) {
          constexpr int i = decltype(ic)::value;
          if constexpr ((ml >> i) & 1ull) fms(w[s], f[(Y::before_f(s) + bits_below(ml, i)) * 16], w[s + i]);
        });
        if constexpr (mp != 0) {
          const int of = (off >> (8 * s)) & 0xff;
          fx_for<1, KL + 1>([&](auto ic) {
            constexpr int i = decltype(ic)::value;
            if constexpr ((mp >> i) & 1ull)
              if (of == i) {
                const double tmp = w[s];
                w[s] = w[s + i];
                w[s + i] = tmp;
              }
          });
        }
      });
    }
    edge(Y::lo(n));
  }
#pragma unroll
  for (int t = 0; t < W; ++t)
    if (t < n) rows[32 * t] = w[t];
  str_wait<0>();
  __syncwarp();
}

template <int MINB, class VM>
__global__ void __launch_bounds__(64, MINB) k_adj_modes_stream(const __grid_constant__ AdjModeArgs a) {
  using S = StrV<VM>;
  __shared__ __align__(16) double ring[kStrRingV + kStrRingG];
  const int lane = threadIdx.x & 31, warp = blockIdx.x;
  const StrLane L = str_lane(a, warp, lane);
  if (!__any_sync(0xffffffffu, L.active)) return;
  const AdjMode c = adj_mode(a, L);
  const size_t g = warp >> 1;
  if (threadIdx.x < 32) {
    double *y = str_global(comps(a.yg) + (size_t)warp * a.n_g * 32 + lane);
    double *sg = str_global(comps(a.sgb) + (size_t)warp * a.NY * 32 + lane);
    adj_g_inputs(a, c, a.inv_cg[L.u], [&](int p, double x) { y[32 * p] = x; }, [&](int j, double x) { sg[32 * j] = x; });
    double *r = ring + kStrRingV;
    str_transposed_u<StrG>(a.str.gb + g * StrLayout<StrG>::bwd_size(a.n_g), a.n_g, r, lane, y);
    str_transposed_l<StrG>(a.str.gf + g * StrLayout<StrG>::fwd_size(a.n_g), a.n_g, r, lane, y);
    adj_g_sources(a, L, c, [&](int p) { return y[32 * p]; }, [&](int e) { return a.str.grs[(size_t)e * a.U + L.u]; },
                  [&](int j) { return sg[32 * j]; });
  } else {
    double *y = str_global(comps(a.yv) + (size_t)warp * a.n_v * 32 + lane);
    adj_v_inputs(a, c, [&](int p, double x) { y[32 * p] = x; });
    str_transposed_u<S>(a.str.vb + g * StrLayout<S>::bwd_size(a.n_v), a.n_v, ring, lane, y);
    str_transposed_l<S>(a.str.vf + g * StrLayout<S>::fwd_size(a.n_v), a.n_v, ring, lane, y);
    adj_v_sources(a, L, c, [&](int p) { return y[32 * p]; }, [&](int e) { return a.str.vrs[(size_t)e * a.U + L.u]; });
  }
}

// Over the full band, on the band storage: blocks of two warps serve 16 modes
// (both real components), warp 0 the v-system's part, warp 1 the omega_y-system's.
__global__ void __launch_bounds__(64) k_adj_modes(const __grid_constant__ AdjModeArgs a) {
  const int tid = blockIdx.x * 32 + (threadIdx.x & 31);
  StrLane L;
  L.m = tid >> 1;
  L.comp = tid & 1;
  L.active = L.m < a.M;
  if (!L.active) return;
  const int k = L.m / a.NXH;
  L.u = (k <= a.NZH ? k : a.NZ - k) * a.NXH + L.m - k * a.NXH;
  const AdjMode c = adj_mode(a, L);
  auto E = [&](int j) { return (size_t)j * c.row + c.e0; };
  if (threadIdx.x < 32) {
    double *y = comps(a.yv);
    adj_v_inputs(a, c, [&](int p, double x) { y[E(p)] = x; });
    band_solve_t<kVKL, kVKU>(
        a.ab_v, a.piv_v, a.n_v, a.U, L.u, [&](int p) { return y[E(p)]; }, [&](int p, double x) { y[E(p)] = x; },
        [&](int p) { return y[E(p)]; }, [&](int p, double x) { y[E(p)] = x; });
    adj_v_sources(a, L, c, [&](int p) { return y[E(p)]; },
                  [&](int e) { return a.rs_v[(size_t)a.vrows[e].p * a.U + L.u]; });
  } else {
    double *y = comps(a.yg), *sg = comps(a.sgb);
    adj_g_inputs(a, c, a.inv_cg[L.u], [&](int p, double x) { y[E(p)] = x; }, [&](int j, double x) { sg[E(j)] = x; });
    band_solve_t<6, 6>(
        a.ab_g, a.piv_g, a.n_g, a.U, L.u, [&](int p) { return y[E(p)]; }, [&](int p, double x) { y[E(p)] = x; },
        [&](int p) { return y[E(p)]; }, [&](int p, double x) { y[E(p)] = x; });
    adj_g_sources(a, L, c, [&](int p) { return y[E(p)]; },
                  [&](int e) { return a.rs_gi[(size_t)a.grows[e].p * a.U + L.u]; }, [&](int j) { return sg[E(j)]; });
  }
}

}  // namespace

void launch_adj_modes(const AdjModeArgs &a, int vmode, cudaStream_t st) {
  const int blocks = 2 * str_groups(a.U);
  if (vmode == 1) k_adj_modes_stream<6, VMasks><<<blocks, 64, 0, st>>>(a);
  else if (vmode == 2) k_adj_modes_stream<6, VMasks6><<<blocks, 64, 0, st>>>(a);
  else k_adj_modes<<<(2 * a.M + 31) / 32, 64, 0, st>>>(a);
}

}  // namespace owt
