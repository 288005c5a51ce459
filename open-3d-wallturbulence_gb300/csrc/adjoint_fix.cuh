// The Lamb vector's adjoint (adjoint.cu) with fixed-point line transforms, for
// the line lengths with a plan: the same three kernels, data layouts, weights
// and products as the FP64 ones, on the passes of transforms_fix.cuh.  One
// translation unit per plan class (adjoint_fix0.cu, ...).
#pragma once
#include "adjoint_kernels.h"
#include "transforms_fix.cuh"

namespace owt {

// (y, z) lines per x group (5 backward and 3 forward lines each) and resident
// blocks asked of the register allocator, by plan class.
template <int CLS> struct FxAdjCfg;
template <> struct FxAdjCfg<0> { static constexpr int P = 2, XB = 5; };
template <> struct FxAdjCfg<1> { static constexpr int P = 1, XB = 5; };
template <> struct FxAdjCfg<2> { static constexpr int P = 1, XB = 3; };

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
  constexpr int P = FxAdjCfg<CLS>::P;
  return 6 * P * (size_t)fx_xline(A, B) * sizeof(fxc) + (size_t)fx_xtables(A, B) * sizeof(FxTw) +
         5 * P * ((size_t)FxCfg<CLS>::T * sizeof(FxBound) + sizeof(FxScale));
}

// Persistent; per group of P (y, z) lines: 5P packed backward lines (u,v)
// (w,ox) (oy,oz) (lbx,lby) (lbz,0), products, 3P packed forward lines.
template <int CLS>
__global__ void __launch_bounds__(5 * FxAdjCfg<CLS>::P *FxCfg<CLS>::T, FxAdjCfg<CLS>::XB)
    k_xlamb_adj_fx(const __grid_constant__ AdjXformArgs a) {
  constexpr int P = FxAdjCfg<CLS>::P, NF = 3 * P;
  extern __shared__ __align__(16) unsigned char smraw[];
  const XformDims d = a.d;
  const FxPlan p = a.fpx;
  const int A = p.A, B = p.B, LS = fx_xline(A, B), ntw = fx_xtables(A, B);
  fxc *R = reinterpret_cast<fxc *>(smraw);
  FxTw *tw = reinterpret_cast<FxTw *>(R + 6 * P * LS);
  FxBound *bd = reinterpret_cast<FxBound *>(tw + ntw);
  FxScale *sc = reinterpret_cast<FxScale *>(bd + 5 * P * FxCfg<CLS>::T);
  double2 *D = reinterpret_cast<double2 *>(R);
  for (int k = threadIdx.x; k < ntw; k += blockDim.x) tw[k] = a.fxx[k];
  const int q = threadIdx.x / p.T, t = threadIdx.x - q * p.T;
  const size_t nlines = (size_t)d.NY * d.NZ2, fstride = nlines * d.NXH;
  const int ngroups = (int)((nlines + P - 1) / P);
  for (int g = blockIdx.x; g < ngroups; g += gridDim.x) {
    __syncthreads();  // the last group's spectra are read (the first: the table is written)
    const size_t line0 = (size_t)g * P;
    // 1. backward transforms
    {
      const int pair = q / P, l = q - pair * P;
      const bool have = line0 + l < nlines;
      const double2 *Af = a.zbuf + (size_t)(2 * pair) * fstride + (line0 + l) * d.NXH;
      fx_x_pass1<CLS, true>(
          p, t < B, q, t,
          [&](auto upper, int s) {
            return fx_bits(fx_hermitian<decltype(upper)::value>(Af, fstride, have, s, d.NXH, d.NX2, pair < 4));
          },
          R + q * LS, tw, bd, sc);
    }
    __syncthreads();
    fx_x_pass2_back<CLS>(p, t < A, t, R + q * LS, sc + q);
    __syncthreads();
    // 2. u_bar = om x lb, om_bar = lb x u, packed (ub,vb) (wb,oxb) (oyb,ozb), in place
    for (int idx = threadIdx.x; idx < P * A * B; idx += blockDim.x) {
      const int l = idx / (A * B), x = idx - l * (A * B);
      const double2 uv = D[(0 * P + l) * LS + x], wox = D[(1 * P + l) * LS + x], oyz = D[(2 * P + l) * LS + x];
      const double2 bxy = D[(3 * P + l) * LS + x], bz0 = D[(4 * P + l) * LS + x];
      const double u = uv.x, v = uv.y, w = wox.x, ox = wox.y, oy = oyz.x, oz = oyz.y;
      const double bx = bxy.x, by = bxy.y, bz = bz0.x;
      D[(0 * P + l) * LS + x] = make_double2(oy * bz - oz * by, oz * bx - ox * bz);
      D[(1 * P + l) * LS + x] = make_double2(ox * by - oy * bx, by * w - bz * v);
      D[(2 * P + l) * LS + x] = make_double2(bz * u - bx * w, bx * v - by * u);
    }
    __syncthreads();
    // 3. forward transforms
    fx_x_pass1<CLS, false>(
        p, q < NF && t < A, q, t, [&](auto, int s) { return fx_bits(D[q * LS + s]); }, R + (NF + (q < NF ? q : 0)) * LS,
        A == B ? tw : tw + A * B, bd, sc);
    __syncthreads();
    if (q < NF && t < B) fx_x_pass2_fwd<CLS>(p, t, R + (NF + q) * LS, R + q * LS);
    __syncthreads();
    // 4. unpack the real-pair spectra, keep kx < NXH, weight 1 (kx = 0) or 2
    for (int idx = threadIdx.x; idx < P * d.NXH; idx += blockDim.x) {
      const int l = idx / d.NXH, km = idx - l * d.NXH;
      const size_t line = line0 + l;
      if (line >= nlines) continue;
      const int mc = (km == 0) ? 0 : d.NX2 - km;
#pragma unroll
      for (int pair = 0; pair < 3; ++pair) {
        const double w = (km == 0 ? 0.5 : 1.0) * fx_factor(sc[pair * P + l]);
        const fxc zm = R[(pair * P + l) * LS + km], zc = R[(pair * P + l) * LS + mc];
        a.lbuf[(size_t)(2 * pair) * fstride + line * d.NXH + km] =
            make_double2(__ll2double_rn(zm.x + zc.x) * w, __ll2double_rn(zm.y - zc.y) * w);
        a.lbuf[(size_t)(2 * pair + 1) * fstride + line * d.NXH + km] =
            make_double2(__ll2double_rn(zm.y + zc.y) * w, __ll2double_rn(zc.x - zm.x) * w);
      }
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
  k.xlines = FxAdjCfg<CLS>::P;
  k.xthreads = 5 * FxAdjCfg<CLS>::P * p.T;
  k.xsmem = fx_adj_xsmem<CLS>(p.A, p.B);
  return k;
}

}  // namespace owt
