// Discrete adjoint of the time step (src/solver.cpp:541-627 with wall
// blowing/suction in the v boundary rows), in FP64.
//
// The forward step is, per mode, linear in the state except for the Lamb
// vector.  Its adjoint runs the step's stages backwards with the transposes of
// the same discrete operators:
//
//  k_adj_nl     nonlinear_source^T: lambda_bar from Hv_bar, Hg_bar, with
//               DY1^T = B_1^T A_1^-T diag(c11) (transposed band solve);
//               the adjoint of the mean-Lamb-vector record joins mode (0, 0).
//  k_zback_adj  } Lamb_vec^T.  The forward map is  lambda = F((B u) x (B om))
//  k_xlamb_adj  } with B the dealiased inverse transform (Hermitian extension
//  k_zfwd_adj   } in x, z-Nyquist row dropped) and F the truncating forward
//               transform (normalised, z-Nyquist row kept).  With the real
//               inner product, F^T = (1/N) B' where B' is B with weight 1/2 on
//               kx > 0 and the Nyquist row kept, and B^T = N F' where F' is F
//               with weight 2 on kx > 0 and the Nyquist row dropped.  So
//                 u_bar  = B^T (om_p x lambda_bar_p)
//                 om_bar = B^T (lambda_bar_p x u_p),  lambda_bar_p = F^T lambda_bar
//               with u_p, om_p the step's physical fields recomputed from its
//               spectral fields (the recompute tape).
//  k_adj_mean   solve_mean^T + solve_friction_force^T (one block).
//  k_adj_modes  mode kernel^T (adjoint_modes.cu): solve_horizontal^T, then transposed solves of
//               the augmented v- and omega_y-systems on the forward factors,
//               and the source assembly^T into the three history levels.  The
//               transposed v solve also yields d objective / d v_w from the
//               two wall rows; it skips the entries outside the interior
//               fill masks where the forward's masked solves apply.
#include <cuda_runtime.h>

#include <algorithm>

#include "adjoint_kernels.h"
#include "owt_device.cuh"
#include "setup_host.h"

namespace owt {

// ---------------------------------------------------------------------------
// One thread per real component of a mode, as the nonlinear source (solve.cu):
// one sweep up with U^T, one down with L^T, B_1^T on the last seven solved rows
// and the outputs.  Bound by FP64 issue (18 operations a node and component);
// the operator tables of a block are in shared memory, what a row reads from
// memory is fetched four rows ahead.  128x129x128, one thread a mode, the solve
// and B_1^T through memory -> here: 0.404 -> 0.215 ms.
constexpr int kANLThreads = 64, kANLThreadsLarge = 256;
// per row: U's column from the diagonal (5), L (2), c11, B_1's column (7 rows)
constexpr int kANLRow = 15;
constexpr size_t adj_nl_smem(int NY) { return (size_t)NY * (kANLRow * sizeof(double) + 1) + 8; }
constexpr size_t kANLSmem = 220 * 1024;  // larger tables are read from device memory

template <bool SMEM>
__global__ void __launch_bounds__(kANLThreadsLarge) k_adj_nl(const __grid_constant__ AdjNLArgs a) {
  const int M = a.M, NY = a.NY, n = NY - 1, tid = blockIdx.x * blockDim.x + threadIdx.x;
  extern __shared__ __align__(16) unsigned char smraw[];
  double *tab = reinterpret_cast<double *>(smraw);
  uint8_t *spiv = reinterpret_cast<uint8_t *>(tab + (size_t)NY * kANLRow);
  auto b1t = [&](int j, int r) {  // B_1(j + r, j)
    double b = 0.0;
    for (int e = 0; e < 8; ++e)
      if (a.b1t_col[j * 8 + e] == j + r && nonzero(a.b1t_val[j * 8 + e])) b = a.b1t_val[j * 8 + e];
    return b;
  };
  auto band = [&](int row, int j) { return a.ab1[(size_t)row * NY + j]; };  // LAPACK layout, KV = 4
  if (SMEM) {
    for (int e = threadIdx.x; e < NY * kANLRow; e += blockDim.x) {
      const int j = e / kANLRow, q = e - j * kANLRow;
      tab[e] = q < 5 ? band(4 - q, j) : q < 7 ? band(q, j) : q == 7 ? a.c11[j] : b1t(j, q - 11);
    }
    for (int j = threadIdx.x; j < NY; j += blockDim.x) spiv[j] = a.piv1[j];
    __syncthreads();
  }
  auto up = [&](int j, int t) { return SMEM ? tab[j * kANLRow + t] : band(4 - t, j); };
  auto lo = [&](int j, int t) { return SMEM ? tab[j * kANLRow + 4 + t] : band(4 + t, j); };
  auto c11 = [&](int j) { return SMEM ? tab[j * kANLRow + 7] : a.c11[j]; };
  auto bt = [&](int j, int r) { return SMEM ? tab[j * kANLRow + 11 + r] : b1t(j, r); };
  auto piv = [&](int j) { return SMEM ? (int)spiv[j] : (int)a.piv1[j]; };
  const int m = tid >> 1, comp = tid & 1;
  if (m >= M) return;
  const int k = m / a.NXH, i = m - k * a.NXH;
  const double kx = a.kx[i], kz = a.kz[k];
  const double k2 = fma(kx, kx, kz * kz);
  const double sgn = comp ? 1.0 : -1.0;  // component c of z gives component 1 - c of -+ i z
  const double skx = sgn * kx, skz = sgn * kz;
  const size_t ld = 2 * (size_t)M;
  const double *hv = reinterpret_cast<const double *>(a.hvb) + tid, *hg = reinterpret_cast<const double *>(a.hgb) + tid;
  double *y = reinterpret_cast<double *>(a.ys) + tid;
  double *lx = reinterpret_cast<double *>(a.lxb) + 2 * (size_t)m + 1 - comp;
  double *lz = reinterpret_cast<double *>(a.lzb) + 2 * (size_t)m + 1 - comp;
  double *ly = reinterpret_cast<double *>(a.lyb) + tid;
  auto at = [&](int j) { return (size_t)(j < n ? (j > 0 ? j : 0) : n) * ld; };
  {
    // U^T y = c11 Hv_bar
    double h[4] = {0.0, 0.0, 0.0, 0.0}, nx[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) nx[q] = hv[at(q)];
#pragma unroll 4
    for (int c = 0; c <= n; ++c) {
      double acc = c11(c) * nx[0];
#pragma unroll
      for (int q = 0; q < 3; ++q) nx[q] = nx[q + 1];
      nx[3] = hv[at(c + 4)];
#pragma unroll
      for (int t = 1; t <= 4; ++t) fms(acc, up(c, t), h[t - 1]);
      acc *= up(c, 0);
      y[(size_t)c * ld] = acc;
#pragma unroll
      for (int t = 3; t > 0; --t) h[t] = h[t - 1];
      h[0] = acc;
    }
  }
  // L^T and the interchanges: b0 .. b2 the entries c .. c + 2, of which c + 2 is
  // final after column c; w: the last seven final rows, c + 2 .. c + 8; node
  // c + 5 goes out
  double b0 = 0.0, b1 = 0.0, b2 = 0.0, w[7] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0}, ny[4], ng[4], nv[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    ny[q] = y[at(n - q)];
    ng[q] = hg[at(n - q)];
    nv[q] = hv[at(n - q)];
  }
#pragma unroll 4
  for (int c = n; c >= -5; --c) {
    b2 = b1;
    b1 = b0;
    b0 = 0.0;
    if (c >= 0) {
      b0 = ny[0];
#pragma unroll
      for (int q = 0; q < 3; ++q) ny[q] = ny[q + 1];
      ny[3] = y[at(c - 4)];
      fms(b0, lo(c, 1), b1);
      fms(b0, lo(c, 2), b2);
      const int off = piv(c);
      if (off == 1) {
        const double q = b0; b0 = b1; b1 = q;
      } else if (off == 2) {
        const double q = b0; b0 = b2; b2 = q;
      }
    }
#pragma unroll
    for (int q = 6; q > 0; --q) w[q] = w[q - 1];
    w[0] = b2;
    const int j = c + 5;
    if (j > n) continue;
    // q = B_1^T w, so that the adjoint of f = i kx lx + i kz lz is -q; the rows
    // further than two off reach only the nodes at the walls
    double q = 0.0;
    if (j <= 3) q = bt(j, -3) * w[0];
    q = fma(bt(j, -2), w[1], q);
    q = fma(bt(j, -1), w[2], q);
    if (j == 0 || j == n) q = fma(bt(j, 0), w[3], q);
    q = fma(bt(j, 1), w[4], q);
    q = fma(bt(j, 2), w[5], q);
    if (j >= n - 3) q = fma(bt(j, 3), w[6], q);
    // lx_bar = -i kz Hg_bar + i kx q ; ly_bar = -k^2 Hv_bar ; lz_bar = i kx Hg_bar + i kz q
    double bx = fma(skz, ng[0], -(skx * q)), bz = -fma(skx, ng[0], skz * q);
    if (m == 0) {
      bx += reinterpret_cast<const double *>(a.lxmb)[2 * j + 1 - comp];
      bz += reinterpret_cast<const double *>(a.lzmb)[2 * j + 1 - comp];
    }
    const size_t o = (size_t)j * ld;
    lx[o] = bx;
    ly[o] = -k2 * nv[0];
    lz[o] = bz;
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      ng[r] = ng[r + 1];
      nv[r] = nv[r + 1];
    }
    ng[3] = hg[at(j - 4)];
    nv[3] = hv[at(j - 4)];
  }
}

void launch_adj_nl(const AdjNLArgs &a, cudaStream_t st) {
  const int bs = 2 * a.M >= kSMs * 4 * kANLThreadsLarge ? kANLThreadsLarge : kANLThreads, gs = (2 * a.M + bs - 1) / bs;
  const size_t b = adj_nl_smem(a.NY);
  if (b <= kANLSmem) k_adj_nl<true><<<gs, bs, b, st>>>(a);
  else k_adj_nl<false><<<gs, bs, 0, st>>>(a);
}

// ---------------------------------------------------------------------------
// Lamb vector adjoint.  Tile shapes as the FP64 forward transforms: ATX kx
// lines per z block, AP (y, z) lines per x block.
constexpr int ATX = 6, AP = 2, ANPAIR = 5;

// R5: the lines have a radix-5 stage (the butterfly is compiled in only then).
template <bool R5>
__global__ void __launch_bounds__(1024) k_zback_adj(AdjXformArgs a) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const XformDims d = a.d;
  const int ls = d.NZ2 + 1;
  double2 *bufa = reinterpret_cast<double2 *>(smraw);
  double2 *bufb = bufa + ATX * ls;
  const int i0 = blockIdx.x * ATX, j = blockIdx.y, f = blockIdx.z;
  const int M = d.NZ * d.NXH;
  const bool adj = f >= 6;  // fields 6..8: lambda_bar (F^T), else the step's fields (B)
  const double2 *src = (adj ? a.lb[f - 6] : a.st[f]) + (size_t)j * M;
  for (int idx = threadIdx.x; idx < ATX * ls; idx += blockDim.x) bufa[idx] = make_double2(0.0, 0.0);
  __syncthreads();
  for (int idx = threadIdx.x; idx < d.NZ * ATX; idx += blockDim.x) {
    const int kz = idx / ATX, c = idx - kz * ATX, i = i0 + c;
    if (i < d.NXH && (adj || kz != d.NZH)) {
      const int slot = kz < d.NZH ? kz : kz + d.NZH;
      double2 v = src[(size_t)kz * d.NXH + i];
      if (adj) {
        const double s = i == 0 ? a.inv_n : 0.5 * a.inv_n;
        v.x *= s;
        v.y *= s;
      }
      bufa[c * ls + slot] = v;
    }
  }
  __syncthreads();
  const double2 *r = fft_lines<double, true, R5>(bufa, bufb, ATX, ls, a.pz, a.twz);
  double2 *dst = a.zbuf + ((size_t)f * d.NY + j) * d.NZ2 * d.NXH;
  for (int idx = threadIdx.x; idx < d.NZ2 * ATX; idx += blockDim.x) {
    const int z = idx / ATX, c = idx - z * ATX;
    if (i0 + c < d.NXH) dst[(size_t)z * d.NXH + i0 + c] = r[c * ls + z];
  }
}

template <bool R5>
__global__ void __launch_bounds__(1024) k_xlamb_adj(AdjXformArgs a) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const XformDims d = a.d;
  const int ls = d.NX2 + 1;
  double2 *bufa = reinterpret_cast<double2 *>(smraw);
  double2 *bufb = bufa + ANPAIR * AP * ls;
  const size_t nlines = (size_t)d.NY * d.NZ2;
  const size_t line0 = (size_t)blockIdx.x * AP;
  const size_t fstride = nlines * d.NXH;
  // 1. pack (u,v) (w,ox) (oy,oz) (lbx,lby) (lbz,0) with the Hermitian extension
  for (int idx = threadIdx.x; idx < ANPAIR * AP * d.NX2; idx += blockDim.x) {
    const int q = idx / d.NX2, mm = idx - q * d.NX2;
    const int pair = q / AP, l = q - pair * AP;
    const size_t line = line0 + l;
    double2 z = make_double2(0.0, 0.0);
    if (line < nlines) {
      const double2 *A = a.zbuf + (size_t)(2 * pair) * fstride + line * d.NXH;
      const double2 *B = (2 * pair + 1 < 9) ? A + fstride : nullptr;
      if (mm == 0) {
        z = make_double2(A[0].x, B ? B[0].x : 0.0);
      } else if (mm < d.NXH) {
        const double2 x = A[mm], y = B ? B[mm] : make_double2(0.0, 0.0);
        z = make_double2(x.x - y.y, x.y + y.x);
      } else if (mm > d.NX2 - d.NXH) {
        const int mp = d.NX2 - mm;
        const double2 x = A[mp], y = B ? B[mp] : make_double2(0.0, 0.0);
        z = make_double2(x.x + y.y, y.x - x.y);
      }
    }
    bufa[q * ls + mm] = z;
  }
  __syncthreads();
  double2 *r = fft_lines<double, true, R5>(bufa, bufb, ANPAIR * AP, ls, a.px, a.twx);
  double2 *o = (r == bufa) ? bufb : bufa;
  // 2. u_bar = om x lb, om_bar = lb x u, packed (ub,vb) (wb,oxb) (oyb,ozb)
  for (int idx = threadIdx.x; idx < AP * d.NX2; idx += blockDim.x) {
    const int l = idx / d.NX2, x = idx - l * d.NX2;
    const double2 uv = r[(0 * AP + l) * ls + x], wox = r[(1 * AP + l) * ls + x], oyz = r[(2 * AP + l) * ls + x];
    const double2 bxy = r[(3 * AP + l) * ls + x], bz0 = r[(4 * AP + l) * ls + x];
    const double u = uv.x, v = uv.y, w = wox.x, ox = wox.y, oy = oyz.x, oz = oyz.y;
    const double bx = bxy.x, by = bxy.y, bz = bz0.x;
    o[(0 * AP + l) * ls + x] = make_double2(oy * bz - oz * by, oz * bx - ox * bz);
    o[(1 * AP + l) * ls + x] = make_double2(ox * by - oy * bx, by * w - bz * v);
    o[(2 * AP + l) * ls + x] = make_double2(bz * u - bx * w, bx * v - by * u);
  }
  __syncthreads();
  const double2 *fo = fft_lines<double, false, R5>(o, r, 3 * AP, ls, a.px, a.twx);
  // 3. unpack the real-pair spectra, keep kx < NXH, weight 1 (kx = 0) or 2
  for (int idx = threadIdx.x; idx < AP * d.NXH; idx += blockDim.x) {
    const int l = idx / d.NXH, mm = idx - l * d.NXH;
    const size_t line = line0 + l;
    if (line >= nlines) continue;
    const int mc = (mm == 0) ? 0 : d.NX2 - mm;
    const double hw = mm == 0 ? 0.5 : 1.0;
#pragma unroll
    for (int pair = 0; pair < 3; ++pair) {
      const double2 zm = fo[(pair * AP + l) * ls + mm], zc = fo[(pair * AP + l) * ls + mc];
      a.lbuf[(size_t)(2 * pair) * fstride + line * d.NXH + mm] =
          make_double2((zm.x + zc.x) * hw, (zm.y - zc.y) * hw);
      a.lbuf[(size_t)(2 * pair + 1) * fstride + line * d.NXH + mm] =
          make_double2((zm.y + zc.y) * hw, (zc.x - zm.x) * hw);
    }
  }
}

template <bool R5>
__global__ void __launch_bounds__(1024) k_zfwd_adj(AdjXformArgs a) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const XformDims d = a.d;
  const int ls = d.NZ2 + 1;
  double2 *bufa = reinterpret_cast<double2 *>(smraw);
  double2 *bufb = bufa + ATX * ls;
  const int i0 = blockIdx.x * ATX, j = blockIdx.y, f = blockIdx.z;
  const double2 *src = a.lbuf + ((size_t)f * d.NY + j) * d.NZ2 * d.NXH;
  for (int idx = threadIdx.x; idx < d.NZ2 * ATX; idx += blockDim.x) {
    const int z = idx / ATX, c = idx - z * ATX;
    bufa[c * ls + z] = (i0 + c < d.NXH) ? src[(size_t)z * d.NXH + i0 + c] : make_double2(0.0, 0.0);
  }
  __syncthreads();
  const double2 *r = fft_lines<double, false, R5>(bufa, bufb, ATX, ls, a.pz, a.twz);
  double2 *dst = a.out[f] + (size_t)j * d.NZ * d.NXH;
  for (int idx = threadIdx.x; idx < d.NZ * ATX; idx += blockDim.x) {
    const int kz = idx / ATX, c = idx - kz * ATX;
    if (i0 + c < d.NXH) {
      const int slot = kz < d.NZH ? kz : kz + d.NZH;
      dst[(size_t)kz * d.NXH + i0 + c] = kz == d.NZH ? make_double2(0.0, 0.0) : r[c * ls + slot];
    }
  }
}

static size_t adj_smem_z(const XformDims &d) { return 2 * (size_t)ATX * (d.NZ2 + 1) * sizeof(double2); }
static size_t adj_smem_x(const XformDims &d) { return 2 * (size_t)ANPAIR * AP * (d.NX2 + 1) * sizeof(double2); }
size_t adj_zbuf_values(const XformDims &d) { return 9 * (size_t)d.NY * d.NZ2 * d.NXH; }
size_t adj_lbuf_values(const XformDims &d) { return 6 * (size_t)d.NY * d.NZ2 * d.NXH; }

// The instances for the channel's line lengths: fixed point where the length
// has a plan, else the FP64 kernels above.
struct AdjXformKernels {
  void (*zback)(AdjXformArgs), (*xlamb)(AdjXformArgs), (*zfwd)(AdjXformArgs);
  int tx, xlines, zthreads, xthreads;
  size_t zsmem, xsmem;
  bool persistent;  // the x pass runs the resident blocks, a group a pair of lines
};
static FxAdjKernels fx_adj_kernels(int L) {
  switch (fx_plan(L).cls) {
    case 0: return fx_adj_kernels0(L);
    case 1: return fx_adj_kernels1(L);
    case 2: return fx_adj_kernels2(L);
    default: return FxAdjKernels{};
  }
}
static AdjXformKernels adj_kernels(const XformDims &d, bool stockham) {
  const bool z5 = d.NZ2 % 5 == 0, x5 = d.NX2 % 5 == 0;
  AdjXformKernels k{z5 ? k_zback_adj<true> : k_zback_adj<false>, x5 ? k_xlamb_adj<true> : k_xlamb_adj<false>,
                    z5 ? k_zfwd_adj<true> : k_zfwd_adj<false>, ATX, AP, d.NZ2, d.NX2, adj_smem_z(d), adj_smem_x(d),
                    false};
  if (stockham) return k;
  const FxAdjKernels fz = fx_adj_kernels(d.NZ2), fx = fx_adj_kernels(d.NX2);
  if (fz.ok) {
    k.zback = fz.zback; k.zfwd = fz.zfwd;
    k.tx = fz.tx; k.zthreads = fz.zthreads; k.zsmem = fz.zsmem;
  }
  if (fx.ok) {
    k.xlamb = fx.xlamb;
    k.xthreads = fx.xthreads; k.xsmem = fx.xsmem;
    k.persistent = true;
  }
  return k;
}

cudaError_t adj_lamb_prepare(const XformDims &d) {
  cudaError_t e = cudaSuccess;
  for (int stockham = 0; stockham < 2 && e == cudaSuccess; ++stockham) {
    const AdjXformKernels k = adj_kernels(d, stockham != 0);
    e = raise_smem_limit(k.zback, k.zsmem);
    if (e == cudaSuccess) e = raise_smem_limit(k.zfwd, k.zsmem);
    if (e == cudaSuccess) e = raise_smem_limit(k.xlamb, k.xsmem);
  }
  return e;
}

void launch_adj_lamb(const AdjXformArgs &a, cudaStream_t st) {
  const XformDims &d = a.d;
  const AdjXformKernels k = adj_kernels(d, a.stockham != 0);
  const int gx = (d.NXH + k.tx - 1) / k.tx;
  k.zback<<<dim3(gx, d.NY, 9), k.zthreads, k.zsmem, st>>>(a);
  size_t grid = ((size_t)d.NY * d.NZ2 + k.xlines - 1) / k.xlines;
  if (k.persistent) grid = std::min(fx_groups(d, 2), resident_blocks(k.xlamb, k.xthreads, k.xsmem));
  k.xlamb<<<(unsigned)grid, k.xthreads, k.xsmem, st>>>(a);
  k.zfwd<<<dim3(gx, d.NY, 6), k.zthreads, k.zsmem, st>>>(a);
}

// ---------------------------------------------------------------------------
// Mean mode: U (with fx) and W (with fz).  Forward:
//   s_j = sum_l beta_l (L_l,j + f_l) + sum_l alpha_l U_l,j / dt   (interior j)
//   U = solve(s) by the omega_y-system of mode (0, 0), dU = c11 d1
//   f = -nu/Ly (dU_NY-1 - dU_0).re ;  u(0,0) = U ;  om_z(0,0) = -dU
//   (W: om_x(0,0) = +dW)
//
// One block: the solves are a serial chain, one lane per real component of each
// profile; the factors of mode (0, 0) (strided by the number of unique modes in
// memory) and the vectors are in shared memory, everything else is spread over
// the block.  128x129x128, two threads on device memory -> here: 1.36 -> 0.26 ms.
constexpr int kAMNThreads = 256, kAMNBand = 19;  // band rows of the factors
size_t adj_mean_smem(int NY, int n) {
  return 2 * (size_t)(NY + n) * sizeof(double2) + (size_t)kAMNBand * n * sizeof(double) + n;
}
constexpr size_t kAMNSmem = 200 * 1024;  // larger factors are read from device memory

template <bool SMEM>
__global__ void __launch_bounds__(kAMNThreads) k_adj_mean(const __grid_constant__ AdjMeanArgs a) {
  const int t = threadIdx.x, NY = a.NY, n = a.n_g, M = a.M;
  const double icg = a.inv_cg0, nu = a.nu;
  extern __shared__ __align__(16) unsigned char smraw[];
  double2 *sb = SMEM ? reinterpret_cast<double2 *>(smraw) : a.scratch;  // [2][NY] source adjoints
  double2 *yy = sb + 2 * NY;                                            // [2][n]
  const double *ab = a.ab_g;
  const uint8_t *piv = a.piv_g;
  const int U = SMEM ? 1 : a.U;
  if (SMEM) {
    double *sab = reinterpret_cast<double *>(yy + 2 * n);
    uint8_t *spv = reinterpret_cast<uint8_t *>(sab + (size_t)kAMNBand * n);
    for (int e = t; e < kAMNBand * n; e += blockDim.x) sab[e] = a.ab_g[(size_t)e * a.U];
    for (int e = t; e < n; e += blockDim.x) spv[e] = a.piv_g[(size_t)e * a.U];
    ab = sab;
    piv = spv;
  }
  for (int e = t; e < 2 * NY; e += blockDim.x) {
    const int q = e / NY, j = e - q * NY;
    const double2 x = q == 0 ? a.Ub[0][j] : a.Wb[0][j], f = (q == 0 ? a.ub : a.wb)[(size_t)j * M];
    const double2 ubar = make_double2(x.x + f.x, x.y + f.y);
    const double2 o = (q == 0 ? a.ozb : a.oxb)[(size_t)j * M];
    double2 dbar = q == 0 ? make_double2(-o.x, -o.y) : o;
    const double fbar = q == 0 ? *a.fxb[0] + a.weight : *a.fzb[0];
    if (j == NY - 1) dbar.x += -nu / a.Ly * fbar;
    if (j == 0) dbar.x += nu / a.Ly * fbar;
    const bool in = j != 0 && j != NY - 1;
    const double w1 = in ? nu * a.c21[j] * icg : 0.0, w2 = in ? a.inv_h2 * nu * a.c22[j] * icg : 0.0, c1 = a.c11[j];
    sb[e] = in ? make_double2(icg * ubar.x, icg * ubar.y) : make_double2(0.0, 0.0);
    yy[q * n + 2 * j] = make_double2(a.inv_h * (c1 * dbar.x + w1 * ubar.x), a.inv_h * (c1 * dbar.y + w1 * ubar.y));
    yy[q * n + 2 * j + 1] = make_double2(w2 * ubar.x, w2 * ubar.y);
  }
  __syncthreads();
  if (t < 4) {
    double *y = reinterpret_cast<double *>(yy + (t >> 1) * n) + (t & 1);
    band_solve_t<6, 6>(
        ab, piv, n, U, 0, [&](int c) { return y[2 * c]; }, [&](int p, double v) { y[2 * p] = v; },
        [&](int p) { return y[2 * p]; }, [&](int p, double z) { y[2 * p] = z; });
  }
  __syncthreads();
  // the rows' sources node by node: those whose last node is j .. j + 4
  const double al0 = 3.0, al1 = -1.5, al2 = 1.0 / 3.0, be0 = 3.0, be1 = -3.0, be2 = 1.0;
  const double q0 = al0 * a.inv_dt, q1 = al1 * a.inv_dt, q2 = al2 * a.inv_dt;
  for (int e = t; e < 2 * NY; e += blockDim.x) {
    const int q = e / NY, j = e - q * NY;
    double2 s = sb[e];
    for (int l = min(j + 4, NY - 1); l >= j; --l)
      for (int r = a.gptr[l + 1] - 1; r >= a.gptr[l]; --r) {
        const StrRow &row = a.grows[r];
        const double w = row.w[4 - (l - j)] * (icg * a.rs_g[(size_t)row.p * a.U]);
        const double2 z = yy[q * n + row.p];
        s.x = fma(w, z.x, s.x);
        s.y = fma(w, z.y, s.y);
      }
    sb[e] = s;
    double2 *const *X = q == 0 ? a.Ub : a.Wb, *const *L = q == 0 ? a.Lxb : a.Lzb;
    L[1][j].x += be0 * s.x; L[1][j].y += be0 * s.y;
    L[2][j].x += be1 * s.x; L[2][j].y += be1 * s.y;
    L[0][j] = make_double2(be2 * s.x, be2 * s.y);
    X[1][j].x += q0 * s.x; X[1][j].y += q0 * s.y;
    X[2][j].x += q1 * s.x; X[2][j].y += q1 * s.y;
    X[0][j] = make_double2(q2 * s.x, q2 * s.y);
  }
  __syncthreads();
  if (t < 2) {
    double fsum = 0.0;
    for (int j = 0; j < NY; ++j) fsum += sb[t * NY + j].x;
    double *const *F = t == 0 ? a.fxb : a.fzb;
    *F[1] += be0 * fsum;
    *F[2] += be1 * fsum;
    *F[0] = be2 * fsum;
  }
}

void launch_adj_mean(const AdjMeanArgs &a, cudaStream_t st) {
  const size_t b = adj_mean_smem(a.NY, a.n_g);
  if (b <= kAMNSmem) k_adj_mean<true><<<1, kAMNThreads, b, st>>>(a);
  else k_adj_mean<false><<<1, kAMNThreads, 0, st>>>(a);
}

cudaError_t adj_prepare(int NY, int n_g) {
  cudaError_t e = cudaSuccess;
  if (adj_nl_smem(NY) <= kANLSmem) e = raise_smem_limit(k_adj_nl<true>, adj_nl_smem(NY));
  if (e == cudaSuccess && adj_mean_smem(NY, n_g) <= kAMNSmem)
    e = raise_smem_limit(k_adj_mean<true>, adj_mean_smem(NY, n_g));
  return e;
}

// ---------------------------------------------------------------------------
__global__ void k_objective_add(const double *fx_ring, const long long *step, double weight, double *acc) {
  *acc += weight * fx_ring[ring_head(*step)];
}

void launch_objective_add(const double *fx_ring, const long long *step, double weight, double *acc,
                          cudaStream_t st) {
  k_objective_add<<<1, 1, 0, st>>>(fx_ring, step, weight, acc);
}

}  // namespace owt
