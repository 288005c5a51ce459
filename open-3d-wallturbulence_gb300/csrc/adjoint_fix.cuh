// The Lamb vector's adjoint (adjoint.cu) with fixed-point line transforms, for
// the line lengths with a plan: the same three kernels, data layouts, weights
// and products as the FP64 ones, on the passes of transforms_fix.cuh.  One
// translation unit per plan class (adjoint_fix0.cu, ...).  The x pass has the
// integer work of the forward one and its FP64 pipe half busy with conversions
// and products: 128x129x128, FP64 kernel -> this, 2.06 -> 0.74 ms (0.93 with
// two fields in a packed line and one line a group).
#pragma once
#include "adjoint_kernels.h"
#include "transforms_fix.cuh"

namespace owt {

// Resident blocks asked of the register allocator for an x group of one pair of
// (y, z) lines (9 backward and 6 forward packed lines), by plan class.
template <int CLS> struct FxAdjCfg;
template <> struct FxAdjCfg<0> { static constexpr int XB = 5; };
template <> struct FxAdjCfg<1> { static constexpr int XB = 3; };
template <> struct FxAdjCfg<2> { static constexpr int XB = 2; };

template <int CLS>
__global__ void __launch_bounds__(FxCfg<CLS>::TX *FxCfg<CLS>::T, FxCfg<CLS>::ZB)
    k_zback_adj_fx(const __grid_constant__ AdjXformArgs a) {
  const XformDims d = a.d;
  const int i = blockIdx.x * FxCfg<CLS>::TX + threadIdx.x % FxCfg<CLS>::TX, j = blockIdx.y, f = blockIdx.z;
  const bool col = i < d.NXH;
  const bool adj = f >= 6;  // fields 6..8: lambda_bar (F^T, the Nyquist row kept), else the step's fields (B)
  const double2 *src = (adj ? a.lb[f - 6] : a.st[f]) + (size_t)j * d.NZ * d.NXH + i;
  const double w = i == 0 ? a.inv_n : 0.5 * a.inv_n;
  double2 *dst = a.zbuf + ((size_t)f * d.NY + j) * d.NZ2 * d.NXH + i;
  fx_z_lines<CLS, true>(
      a.fpz, a.fxz,
      [&](auto, int s) {
        const int kz = s < d.NZH ? s : s > d.NZ || (adj && s == d.NZ) ? s - d.NZH : -1;
        double2 v = make_double2(0.0, 0.0);
        if (col && kz >= 0) {
          v = src[(size_t)kz * d.NXH];
          if (adj) v = make_double2(v.x * w, v.y * w);
        }
        return v;
      },
      [&](auto, int s, fxc v, const FxScale &sc) {
        const FxOut o = fx_out(sc);
        if (col) dst[(size_t)s * d.NXH] = make_double2(fx_to_double(v.x, o), fx_to_double(v.y, o));
      });
}

template <int CLS>
__global__ void __launch_bounds__(FxCfg<CLS>::TX *FxCfg<CLS>::T, FxCfg<CLS>::ZB)
    k_zfwd_adj_fx(const __grid_constant__ AdjXformArgs a) {
  const XformDims d = a.d;
  const int i = blockIdx.x * FxCfg<CLS>::TX + threadIdx.x % FxCfg<CLS>::TX, j = blockIdx.y, f = blockIdx.z;
  const bool col = i < d.NXH;
  const double2 *src = a.lbuf + ((size_t)f * d.NY + j) * d.NZ2 * d.NXH + i;
  double2 *dst = a.out[f] + (size_t)j * d.NZ * d.NXH + i;
  fx_z_lines<CLS, false>(
      a.fpz, a.fxz, [&](auto, int s) { return col ? src[(size_t)s * d.NXH] : make_double2(0.0, 0.0); },
      [&](auto, int s, fxc v, const FxScale &sc) {  // the Nyquist row (slot NZ) is zero
        const int kz = s < d.NZH ? s : s >= d.NZ ? s - d.NZH : -1;
        if (col && kz >= 0) {
          const FxOut o = fx_out(sc);
          dst[(size_t)kz * d.NXH] =
              s == d.NZ ? make_double2(0.0, 0.0) : make_double2(fx_to_double(v.x, o), fx_to_double(v.y, o));
        }
      });
}

template <int CLS>
constexpr size_t fx_adj_xsmem(int A, int B) {
  return 9 * (size_t)fx_xline(A, B) * sizeof(fxc) + (size_t)fx_xtables(A, B) * sizeof(FxTw) +
         9 * ((size_t)FxCfg<CLS>::T * sizeof(FxBound) + sizeof(FxScale));
}

// Persistent; per pair of (y, z) lines: 9 packed backward lines (u v w ox oy oz
// lbx lby lbz, one field on both lines, as the step's x pass), products,
// 6 packed forward lines.  In place: a line's pass reads all it needs before a
// barrier.
template <int CLS>
__global__ void __launch_bounds__(9 * FxCfg<CLS>::T, FxAdjCfg<CLS>::XB)
    k_xlamb_adj_fx(const __grid_constant__ AdjXformArgs a) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const XformDims d = a.d;
  const FxPlan p = a.fpx;
  const int A = p.A, B = p.B, LS = fx_xline(A, B), ntw = fx_xtables(A, B);
  fxc *R = reinterpret_cast<fxc *>(smraw);
  FxTw *tw = reinterpret_cast<FxTw *>(R + 9 * LS);
  FxBound *bd = reinterpret_cast<FxBound *>(tw + ntw);
  FxScale *sc = reinterpret_cast<FxScale *>(bd + 9 * FxCfg<CLS>::T);
  double2 *D = reinterpret_cast<double2 *>(R);
  for (int k = threadIdx.x; k < ntw; k += blockDim.x) tw[k] = a.fxx[k];
  const int q = threadIdx.x / p.T, t = threadIdx.x - q * p.T;
  const size_t fstride = (size_t)d.NY * d.NZ2 * d.NXH;
  const int ngroups = fx_groups(d, 2);
  for (int g = blockIdx.x; g < ngroups; g += gridDim.x) {
    __syncthreads();  // the last group's spectra are read (the first: the table is written)
    const FxPair pr = fx_pair(d, (unsigned)g);
    // 1. backward transforms: line q is field q
    const double2 *Af = a.zbuf + (size_t)q * fstride + pr.line * d.NXH;
    fx_x_pass1<CLS, true>(
        p, t < B, q, t,
        [&](auto upper, int s) {
          return fx_bits(fx_hermitian<decltype(upper)::value>(Af, pr.have, pr.have_b, s, d.NXH, d.NX2));
        },
        R + q * LS, tw, bd, sc);
    __syncthreads();
    fx_x_pass2_back<CLS>(p, t < A, t, R + q * LS, sc + q);
    __syncthreads();
    // 2. u_bar = om x lb, om_bar = lb x u into lines 0..5, in place
    for (int x = threadIdx.x; x < A * B; x += blockDim.x) {
      const double2 u = D[x], v = D[LS + x], w = D[2 * LS + x], ox = D[3 * LS + x], oy = D[4 * LS + x],
                    oz = D[5 * LS + x], bx = D[6 * LS + x], by = D[7 * LS + x], bz = D[8 * LS + x];
      D[x] = make_double2(oy.x * bz.x - oz.x * by.x, oy.y * bz.y - oz.y * by.y);
      D[LS + x] = make_double2(oz.x * bx.x - ox.x * bz.x, oz.y * bx.y - ox.y * bz.y);
      D[2 * LS + x] = make_double2(ox.x * by.x - oy.x * bx.x, ox.y * by.y - oy.y * bx.y);
      D[3 * LS + x] = make_double2(by.x * w.x - bz.x * v.x, by.y * w.y - bz.y * v.y);
      D[4 * LS + x] = make_double2(bz.x * u.x - bx.x * w.x, bz.y * u.y - bx.y * w.y);
      D[5 * LS + x] = make_double2(bx.x * v.x - by.x * u.x, bx.y * v.y - by.y * u.y);
    }
    __syncthreads();
    // 3. forward transforms
    fx_x_pass1<CLS, false>(
        p, q < 6 && t < A, q, t, [&](auto, int s) { return fx_bits(D[q * LS + s]); }, R + q * LS,
        A == B ? tw : tw + A * B, bd, sc);
    __syncthreads();
    fx_x_pass2_fwd<CLS, true>(p, q < 6 && t < B, t, R + q * LS, R + q * LS);
    __syncthreads();
    // 4. unpack the real-pair spectra, keep kx < NXH, weight 1 (kx = 0) or 2
    for (int idx = threadIdx.x; idx < 6 * d.NXH; idx += blockDim.x) {
      const int f = idx / d.NXH, km = idx - f * d.NXH;
      const int mc = (km == 0) ? 0 : d.NX2 - km;
      const double w = (km == 0 ? 0.5 : 1.0) * fx_factor(sc[f]);
      const fxc zm = R[f * LS + km], zc = R[f * LS + mc];
      double2 *o = a.lbuf + (size_t)f * fstride + pr.line * d.NXH + km;
      o[0] = make_double2(__ll2double_rn(zm.x + zc.x) * w, __ll2double_rn(zm.y - zc.y) * w);
      if (pr.have_b) o[d.NXH] = make_double2(__ll2double_rn(zm.y + zc.y) * w, __ll2double_rn(zc.x - zm.x) * w);
    }
  }
}

template <int CLS>
FxAdjKernels fx_adj_kernels_of_class(int L) {
  const FxPlan p = fx_plan(L);
  FxAdjKernels k;
  if (p.cls != CLS) return k;
  k.ok = true;
  k.zback = k_zback_adj_fx<CLS>;
  k.zfwd = k_zfwd_adj_fx<CLS>;
  k.xlamb = k_xlamb_adj_fx<CLS>;
  k.tx = FxCfg<CLS>::TX;
  k.zthreads = FxCfg<CLS>::TX * p.T;
  k.zsmem = fx_zsmem<CLS>(L);
  k.xthreads = 9 * p.T;
  k.xsmem = fx_adj_xsmem<CLS>(p.A, p.B);
  return k;
}

}  // namespace owt
