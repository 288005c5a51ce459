// Transform kernels of the FP64 step with 64-bit fixed-point line transforms
// (fft_fix.cuh): the three kernels, data layouts and dealiasing of
// transforms.cu (src/FFT.cpp:49-194, src/solver.cpp:262-304), FP64 in memory,
// for the line lengths with a plan (fx_plan).  One translation unit per plan
// class instantiates them (transforms_fix0.cu, ...), so that the register
// budget of a kernel is that of its largest radix and the units compile in
// parallel.
//
// A line of A B points has T = max(A, B) threads; every thread of a block
// takes part in every barrier, those beyond the number of a pass's transforms
// idle in it.
//
//  k_zback_fx : block (kTX kx columns, y, field), column fastest in the
//               thread index so that rows of kx coalesce; the padded z line
//               is gathered straight into pass-1 registers.
//  k_xlamb_fx : persistent; per group of P (y, z) lines: 3P packed backward
//               lines, products in shared memory (integers too), 3P/2 packed
//               forward lines, the real-pair unpack; the next group's input
//               is prefetched into L2.  A packed line holds one field on two
//               z-neighbours of a plane, so that a field has its own scale.
//  k_zfwd_fx  : as k_zback_fx, forward.
//
// Measured at 384x257x384 (lines of 576 points), FP64 kernels -> these:
// z backward 10.74 -> 1.65 ms, x pass 27.99 -> 6.92 ms, z forward
// 5.27 -> 0.96 ms; at 128x129x128 0.496 -> 0.095, 1.189 -> 0.400 and
// 0.255 -> 0.060 ms.  The z passes are bound by integer issue at half of the
// DRAM rate, the x pass by latency (about 1.6 instructions a clock whatever the
// number of resident blocks; a fifth of the stalls are its barriers).  In the
// x pass FP64 products of converted values took 7.85 and 0.42 ms: a conversion
// is an FP64 instruction, and the FP64 pipe was 43% busy.  Block shapes were
// measured over the classes (three blocks an SM instead of two for the x pass
// of class 2: 12.2 -> 7.9 ms with the zero thirds left out; z blocks of 4 or 16
// columns 5 to 25% slower).
#pragma once
#include <cuda_runtime.h>

#include "batch.cuh"
#include "fft_fix.cuh"
#include "owt_device.cuh"
#include "solve_kernels.h"

namespace owt {

// Block shapes by plan class: kx columns per z block, (y, z) lines per x
// group, and the resident blocks asked of the register allocator.
template <int CLS> struct FxCfg;
template <> struct FxCfg<0> { static constexpr int T = 12, TX = 8, P = 4, ZB = 8, XB = 5; };
template <> struct FxCfg<1> { static constexpr int T = 18, TX = 8, P = 2, ZB = 3, XB = 4; };
template <> struct FxCfg<2> { static constexpr int T = 24, TX = 8, P = 2, ZB = 2, XB = 3; };

__device__ __forceinline__ fxc fx_bits(double2 v) {
  return fxc{__double_as_longlong(v.x), __double_as_longlong(v.y)};
}

__device__ __forceinline__ FxTw fx_ldg(const FxTw *p) {
  const int4 v = __ldg(reinterpret_cast<const int4 *>(p));
  return FxTw{v.x, v.y, v.z, v.w};
}

// The rest of pass 1 once the line's scale is known: x (doubles' bits) to
// integers, N-point transform, output r times twiddle(r) to store(r, value).
// INT: x are integers of that scale already.
template <int N, bool BACKWARD, bool INT, class Twiddle, class Store>
__device__ __forceinline__ void fx_line_pass1(fxc *x, const FxScale &s, Twiddle twiddle, Store store) {
  if constexpr (!INT)
    fx_for<0, N>([&](auto rc) {
      constexpr int r = decltype(rc)::value;
      if constexpr (!BACKWARD || N % 3 != 0 || r < N / 3 || r >= 2 * N / 3)
        x[r] = fxc{fx_from_bits(x[r].x, s), fx_from_bits(x[r].y, s)};
    });
  fx_dft<N, BACKWARD>(x);
  store(0, fx_quarter(x[0]));
  fx_for<1, N>([&](auto rc) {
    constexpr int r = decltype(rc)::value;
    store(r, fx_twiddle<BACKWARD>(x[r], twiddle(r)));
  });
}

// Shared memory of a z block: the transposes of TX lines ([a'][b][column]),
// the bounds and scales of its lines.
template <int CLS>
__host__ __device__ constexpr size_t fx_zsmem(int L) {
  return (size_t)FxCfg<CLS>::TX * (L * sizeof(fxc) + FxCfg<CLS>::T * sizeof(FxBound) + sizeof(FxScale));
}

// One block of line transforms along z.  load(r, s) gives slot s = t + N2 r of
// this thread's column (r a compile-time index), store(r, s, value, scale)
// takes output slot s = t + N1 r.  The middle third of the slots is zero in a
// backward transform's input and unused in a forward transform's output.
template <int CLS, bool BACKWARD, class Load, class Store>
__device__ __forceinline__ void fx_z_lines(const FxPlan p, const FxTw *__restrict__ tw, Load load, Store store) {
  constexpr int TX = FxCfg<CLS>::TX;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int L = p.A * p.B, N1 = BACKWARD ? p.A : p.B, N2 = BACKWARD ? p.B : p.A;
  fxc *S = reinterpret_cast<fxc *>(smraw);
  FxBound *bd = reinterpret_cast<FxBound *>(S + (size_t)TX * L);
  FxScale *sc = reinterpret_cast<FxScale *>(bd + TX * FxCfg<CLS>::T);
  const int c = threadIdx.x % TX, t = threadIdx.x / TX;
  if (!BACKWARD) tw += L;
  fx_radix<CLS>(N1, [&](auto n) {
    constexpr int N = decltype(n)::value;
    fxc x[N];
    fx_for<0, N>([&](auto rc) { x[decltype(rc)::value] = fxc{0, 0}; });
    if (t < N2) {
      fx_for<0, N>([&](auto rc) {
        constexpr int r = decltype(rc)::value;
        if constexpr (!BACKWARD || N % 3 != 0 || r < N / 3 || r >= 2 * N / 3) x[r] = fx_bits(load(rc, t + N2 * r));
      });
      bd[t * TX + c] = fx_bound<N>(x);
    }
    __syncthreads();
    if (t < N2) {
      const FxScale s = fx_scale(N2, [&](int k) { return bd[k * TX + c]; });
      if (t == 0) sc[c] = s;
      fx_line_pass1<N, BACKWARD, false>(x, s, [&](int r) { return fx_ldg(tw + r * N2 + t); },
                                 [&](int r, fxc v) { S[(r * N2 + t) * TX + c] = v; });
    }
  });
  __syncthreads();
  if (t < N1)
    fx_radix<CLS>(N2, [&](auto n) {
      constexpr int N = decltype(n)::value;
      fxc y[N];
      fx_for<0, N>([&](auto rc) { y[decltype(rc)::value] = S[(t * N + decltype(rc)::value) * TX + c]; });
      fx_dft<N, BACKWARD>(y);
      const FxScale s = sc[c];
      fx_for<0, N>([&](auto rc) {
        constexpr int r = decltype(rc)::value;
        if constexpr (BACKWARD || N % 3 != 0 || r < N / 3 || r >= 2 * N / 3) store(rc, t + N1 * r, y[r], s);
      });
    });
}

template <int CLS>
__device__ __forceinline__ void zback_fx_body(const XformArgs &a, const int bx, const int j, const int f) {
  const XformDims d = a.d;
  const int i = bx * FxCfg<CLS>::TX + threadIdx.x % FxCfg<CLS>::TX;
  const bool col = i < d.NXH;
  const double2 *base = a.in[f];
  if (a.ring_mask & (1 << f)) base += (size_t)ring_head(*a.step) * a.fs;
  const double2 *src = base + (size_t)j * d.NZ * d.NXH + i;
  double2 *dst = reinterpret_cast<double2 *>(a.zbuf) + ((size_t)f * d.NY + j) * d.NZ2 * d.NXH + i;
  fx_z_lines<CLS, true>(
      a.fpz, a.fxz,
      [&](auto, int s) {  // slot of the padded line: k < NZH -> k, k > NZH -> k + NZH, the Nyquist row dropped
        const int kz = s < d.NZH ? s : s > d.NZ ? s - d.NZH : -1;
        return col && kz >= 0 ? src[(size_t)kz * d.NXH] : make_double2(0.0, 0.0);
      },
      [&](auto, int s, fxc v, const FxScale &sc) {
        const FxOut o = fx_out(sc);
        if (col) dst[(size_t)s * d.NXH] = make_double2(fx_to_double(v.x, o), fx_to_double(v.y, o));
      });
}

template <int CLS>
__device__ __forceinline__ void zfwd_fx_body(const XformArgs &a, const int bx, const int j, const int f) {
  const XformDims d = a.d;
  const int i = bx * FxCfg<CLS>::TX + threadIdx.x % FxCfg<CLS>::TX;
  const bool col = i < d.NXH;
  const double2 *src = reinterpret_cast<const double2 *>(a.lbuf) + ((size_t)f * d.NY + j) * d.NZ2 * d.NXH + i;
  double2 *dst = a.out[f] + (size_t)j * d.NZ * d.NXH + i;
  fx_z_lines<CLS, false>(
      a.fpz, a.fxz, [&](auto, int s) { return col ? src[(size_t)s * d.NXH] : make_double2(0.0, 0.0); },
      [&](auto, int s, fxc v, const FxScale &sc) {  // keep slots k < NZH (kz k) and NZ + k (kz k + NZH)
        const int kz = s < d.NZH ? s : s >= d.NZ ? s - d.NZH : -1;
        if (col && kz >= 0) {
          const double w = a.inv_nz2 * fx_factor(sc);
          dst[(size_t)kz * d.NXH] = make_double2(__dmul_rn(__ll2double_rn(v.x), w), __dmul_rn(__ll2double_rn(v.y), w));
        }
      });
}

// ---------------------------------------------------------------------------
// x pass
// ---------------------------------------------------------------------------
// Point m = t + N2 r of the packed line of two real lines' spectra A and
// B = A + NXH (hermitian_pair of owt_device.cuh): UPPER (r in the upper third) takes the
// conjugate half, the padding slot 2 NX2/3 included as zero.  have, have_b:
// the lines exist (else zeros).
template <bool UPPER>
__device__ __forceinline__ double2 fx_hermitian(const double2 *__restrict__ A, bool have, bool have_b, int m, int NXH,
                                                int NX2) {
  const int mp = UPPER ? NX2 - m : m;
  double2 x = make_double2(0.0, 0.0), y = x;
  if (have && mp < NXH) {
    x = __ldg(A + mp);
    if (have_b) y = __ldg(A + NXH + mp);
  }
  if (UPPER) return make_double2(x.x + y.y, y.x - x.y);
  if (m == 0) x.y = y.y = 0.0;
  return make_double2(x.x - y.y, x.y + y.x);
}

// Pairs of z-neighbours are numbered plane by plane (the last of a plane with
// an odd number of lines holds one line); groups of the x pass are PAIRS
// consecutive pairs.
struct FxPair {
  bool have, have_b;
  size_t line;  // the first line, y NZ2 + z
};
__device__ __forceinline__ FxPair fx_pair(const XformDims &d, unsigned pair) {
  const unsigned half = (unsigned)(d.NZ2 + 1) / 2, j = pair / half, z = 2 * (pair - j * half);
  const bool have = j < (unsigned)d.NY;
  return FxPair{have, have && (int)z + 1 < d.NZ2, (size_t)j * d.NZ2 + z};
}

// Shared memory: 3P lines of LS values (transposes with odd row stride, or
// the line itself), the twiddle tables (one where A = B), bounds and scales.
__host__ __device__ constexpr int fx_row(int B) { return B | 1; }
__host__ __device__ constexpr int fx_xline(int A, int B) {
  return A * fx_row(B) > B * fx_row(A) ? A * fx_row(B) : B * fx_row(A);
}
__host__ __device__ constexpr int fx_xtables(int A, int B) { return (A == B ? 1 : 2) * A * B; }
template <int CLS>
constexpr size_t fx_xsmem(int A, int B) {
  constexpr int P = FxCfg<CLS>::P;
  return 3 * P * (size_t)fx_xline(A, B) * sizeof(fxc) + (size_t)fx_xtables(A, B) * sizeof(FxTw) +
         3 * P * ((size_t)FxCfg<CLS>::T * sizeof(FxBound) + sizeof(FxScale) + sizeof(unsigned));
}

// Pass 1 of line q's transform on input in(r, s) (s = t + N2 r), its
// transposes to R[r RS + t] of its line; the line's scale to sc[q].  act: the
// thread has a transform in this pass.  All threads call it.  INT: the input
// is the integers of products, at the scale and finiteness pk, ok of the line.
template <int CLS, bool BACKWARD, bool INT = false, class In>
__device__ __forceinline__ void fx_x_pass1(const FxPlan p, bool act, int q, int t, In in, fxc *R, const FxTw *tw,
                                           FxBound *bd, FxScale *sc, int pk = 0, bool ok = true) {
  const int N1 = BACKWARD ? p.A : p.B, N2 = BACKWARD ? p.B : p.A, RS = fx_row(N2);
  bd += q * p.T;
  fx_radix<CLS>(N1, [&](auto n) {
    constexpr int N = decltype(n)::value;
    fxc x[N];
    // (set on both paths: left undefined where !act, they would be kept in
    // local memory around the loop over groups)
    fx_for<0, N>([&](auto rc) { x[decltype(rc)::value] = fxc{0, 0}; });
    if (act) {
      fx_for<0, N>([&](auto rc) {
        constexpr int r = decltype(rc)::value;
        if constexpr (!BACKWARD || N % 3 != 0 || r < N / 3 || r >= 2 * N / 3)
          x[r] = in(std::integral_constant<bool, (r >= 2 * N / 3)>{}, t + N2 * r);
      });
      if constexpr (INT) bd[t].s = fx_bound_int<N>(x);
      else bd[t] = fx_bound<N>(x);
    }
    __syncthreads();
    if (act) {
      FxScale s;
      if constexpr (INT) {
        int shift;
        s = fx_scale_int(N2, [&](int k) { return bd[k].s; }, pk, ok, shift);
        const int left = max(shift, 0), right = max(-shift, 0);
        fx_for<0, N>([&](auto rc) {
          fxc &v = x[decltype(rc)::value];
          v = fxc{fx_rescale(v.x, left, right), fx_rescale(v.y, left, right)};
        });
      } else {
        s = fx_scale(N2, [&](int k) { return bd[k]; });
      }
      if (t == 0) sc[q] = s;
      fx_line_pass1<N, BACKWARD, INT>(x, s, [&](int r) { return tw[r * N2 + t]; },
                                      [&](int r, fxc v) { R[r * RS + t] = v; });
    }
  });
}

// Backward pass 2 of line q: point t + A r, in place (R: the line), as FP64 or
// (INT) as integers of scale fx_k(*sc) with the highest bit of fx_mag into mag
// (zero on entry).
template <int CLS, bool INT = false>
__device__ __forceinline__ void fx_x_pass2_back(const FxPlan p, bool act, int t, fxc *R, const FxScale *sc,
                                                unsigned *mag = nullptr) {
  const int A = p.A;
  fx_radix<CLS>(p.B, [&](auto n) {
    constexpr int N = decltype(n)::value, RS = fx_row(N);
    fxc y[N];
    fx_for<0, N>([&](auto rc) { y[decltype(rc)::value] = fxc{0, 0}; });
    if (act) {
      fx_for<0, N>([&](auto rc) { y[decltype(rc)::value] = R[t * RS + decltype(rc)::value]; });
      fx_dft<N, true>(y);
      if constexpr (INT) {
        unsigned m = 0;
        fx_for<0, N>([&](auto rc) { m |= fx_mag(y[decltype(rc)::value]); });
        atomicOr(mag, m);
      }
    }
    __syncthreads();
    if (!act) return;
    if constexpr (INT) {
      fx_for<0, N>([&](auto rc) { R[t + A * decltype(rc)::value] = y[decltype(rc)::value]; });
    } else {
      const FxOut o = fx_out(*sc);
      double2 *D = reinterpret_cast<double2 *>(R);
      fx_for<0, N>([&](auto rc) {
        constexpr int r = decltype(rc)::value;
        D[t + A * r] = make_double2(fx_to_double(y[r].x, o), fx_to_double(y[r].y, o));
      });
    }
  });
}

// Forward pass 2: spectrum slot t + B r, integers, from the transposes at R
// into the line at out (the middle third is not read).  IN_PLACE: out is R,
// all threads call it (act: the thread has a transform); else no barrier.
template <int CLS, bool IN_PLACE = false>
__device__ __forceinline__ void fx_x_pass2_fwd(const FxPlan p, bool act, int t, const fxc *R, fxc *out) {
  const int B = p.B;
  if (!IN_PLACE && !act) return;
  fx_radix<CLS>(p.A, [&](auto n) {
    constexpr int N = decltype(n)::value, RS = fx_row(N);
    fxc y[N];
    if constexpr (IN_PLACE) fx_for<0, N>([&](auto rc) { y[decltype(rc)::value] = fxc{0, 0}; });
    if (act) {
      fx_for<0, N>([&](auto rc) { y[decltype(rc)::value] = R[t * RS + decltype(rc)::value]; });
      fx_dft<N, false>(y);
    }
    if constexpr (IN_PLACE) __syncthreads();
    if (!act) return;
    fx_for<0, N>([&](auto rc) {
      constexpr int r = decltype(rc)::value;
      if constexpr (N % 3 != 0 || r < N / 3 || r >= 2 * N / 3) out[t + B * r] = y[r];
    });
  });
}

template <int CLS>
__device__ __forceinline__ void xlamb_fx_group(const XformArgs &a, const unsigned pair0, fxc *R, const FxTw *tw,
                                               FxBound *bd, FxScale *sc, unsigned *mag) {
  constexpr int P = FxCfg<CLS>::P, H = P / 2, NF = 3 * H;
  const XformDims d = a.d;
  const FxPlan p = a.fpx;
  const int A = p.A, B = p.B, LS = fx_xline(A, B);
  const int q = threadIdx.x / p.T, t = threadIdx.x - q * p.T;
  const size_t fstride = (size_t)d.NY * d.NZ2 * d.NXH;
  // 1. backward pass 1: packed line q = H f + h holds pair h of field f
  if (t == 0) mag[q] = 0u;
  {
    const int f = q / H;
    const FxPair pr = fx_pair(d, pair0 + (q - f * H));
    const double2 *Af = reinterpret_cast<const double2 *>(a.zbuf) + (size_t)f * fstride + pr.line * d.NXH;
    fx_x_pass1<CLS, true>(
        p, t < B, q, t,
        [&](auto upper, int s) {
          return fx_bits(fx_hermitian<decltype(upper)::value>(Af, pr.have, pr.have_b, s, d.NXH, d.NX2));
        },
        R + q * LS, tw, bd, sc);
  }
  __syncthreads();
  // 2. backward pass 2
  fx_x_pass2_back<CLS, true>(p, t < A, t, R + q * LS, sc + q, mag + q);
  __syncthreads();
  // 3. lamb = u x omega in integers, component c of pair h into line H c + h,
  // in place: one thread owns point xx of every line
  int pk = 0;  // scale and finiteness of this thread's forward line
  bool ok = true;
#pragma unroll 1
  for (int h = 0; h < H; ++h) {
    int k[6];
    unsigned mg[6];
    bool fin = true;
#pragma unroll
    for (int f = 0; f < 6; ++f) {
      k[f] = fx_k(sc[f * H + h]);
      fin = fin && sc[f * H + h].finite;
      mg[f] = mag[f * H + h];
    }
    const FxProducts pr = fx_products(k, mg);
#pragma unroll
    for (int c = 0; c < 3; ++c)
      if (q == c * H + h) {
        pk = pr.k[c];
        ok = fin;
      }
    for (int xx = threadIdx.x; xx < A * B; xx += blockDim.x) {
      long long f0[6], f1[6], l0[3], l1[3];
#pragma unroll
      for (int f = 0; f < 6; ++f) {
        const fxc v = R[(f * H + h) * LS + xx];
        f0[f] = v.x;
        f1[f] = v.y;
      }
      fx_lamb(f0, pr, l0);
      fx_lamb(f1, pr, l1);
#pragma unroll
      for (int c = 0; c < 3; ++c) R[(c * H + h) * LS + xx] = fxc{l0[c], l1[c]};
    }
  }
  __syncthreads();
  // 4. forward pass 1 of the NF product lines, transposes into lines NF + q
  fx_x_pass1<CLS, false, true>(
      p, q < NF && t < A, q, t, [&](auto, int s) { return R[q * LS + s]; }, R + (NF + q) * LS,
      A == B ? tw : tw + A * B, bd, sc, pk, ok);
  __syncthreads();
  // 5. forward pass 2 into line q
  fx_x_pass2_fwd<CLS>(p, q < NF && t < B, t, R + (NF + q) * LS, R + q * LS);
  __syncthreads();
  // 6. unpack the real-pair spectra, keep kx < NXH, scale by 1/NX2:
  // Xa = (Z[m] + conj Z[-m]) / 2 ; Xb = (Z[m] - conj Z[-m]) / (2i)
  double2 *lb = reinterpret_cast<double2 *>(a.lbuf);
  const double half = 0.5 * a.inv_nx2;
  for (int idx = threadIdx.x; idx < H * d.NXH; idx += blockDim.x) {
    const int h = idx / d.NXH, km = idx - h * d.NXH;
    const FxPair pr = fx_pair(d, pair0 + h);
    if (!pr.have) continue;
    const int mc = (km == 0) ? 0 : d.NX2 - km;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double w = half * fx_factor(sc[c * H + h]);
      const fxc zm = R[(c * H + h) * LS + km], zc = R[(c * H + h) * LS + mc];
      double2 *o = lb + (size_t)c * fstride + pr.line * d.NXH + km;
      o[0] = make_double2(__dmul_rn(__ll2double_rn(zm.x + zc.x), w), __dmul_rn(__ll2double_rn(zm.y - zc.y), w));
      if (pr.have_b)
        o[d.NXH] = make_double2(__dmul_rn(__ll2double_rn(zm.y + zc.y), w), __dmul_rn(__ll2double_rn(zc.x - zm.x), w));
    }
  }
}

// Fetch the input lines of the pairs pair0 .. pair0 + PAIRS - 1 of the six
// fields into L2 (consecutive in memory: a plane's last line is followed by the
// next plane's first).
template <int PAIRS>
__device__ __forceinline__ void fx_prefetch_lines(const XformArgs &a, unsigned pair0) {
  const size_t fstride = (size_t)a.d.NY * a.d.NZ2 * a.d.NXH;
  const FxPair first = fx_pair(a.d, pair0);
  FxPair last = fx_pair(a.d, pair0 + PAIRS - 1);
  if (!last.have) last = first;
  const int nl = first.have ? (int)(last.line - first.line) + (last.have_b ? 2 : 1) : 0;
  const int per = (nl * a.d.NXH + 7) / 8;  // 128-byte lines per field
  for (int idx = threadIdx.x; idx < 6 * per; idx += blockDim.x) {
    const int f = idx / per, o = idx - f * per;
    const double2 *src =
        reinterpret_cast<const double2 *>(a.zbuf) + (size_t)f * fstride + first.line * a.d.NXH + 8 * o;
    asm volatile("prefetch.global.L2 [%0];" ::"l"(src));
  }
}

// The groups g0, g0 + step, ... < ngroups; args(g, pair0) gives the arguments
// and first pair of group g (several channels, all of one plan, in the batch).
template <int CLS, class Args>
__device__ __forceinline__ void xlamb_fx_run(int g0, int step, int ngroups, Args args) {
  constexpr int P = FxCfg<CLS>::P;
  extern __shared__ __align__(16) unsigned char smraw[];
  unsigned pair0;
  const XformArgs &a0 = args(g0 < ngroups ? g0 : 0, pair0);
  const int A = a0.fpx.A, B = a0.fpx.B;
  fxc *R = reinterpret_cast<fxc *>(smraw);
  FxTw *tw = reinterpret_cast<FxTw *>(R + 3 * P * fx_xline(A, B));
  const int ntw = fx_xtables(A, B);
  FxBound *bd = reinterpret_cast<FxBound *>(tw + ntw);
  FxScale *sc = reinterpret_cast<FxScale *>(bd + 3 * P * FxCfg<CLS>::T);
  unsigned *mag = reinterpret_cast<unsigned *>(sc + 3 * P);
  for (int k = threadIdx.x; k < ntw; k += blockDim.x) tw[k] = a0.fxx[k];
  for (int g = g0; g < ngroups; g += step) {
    __syncthreads();  // the last group's spectra are read (the first: the table is written)
    const XformArgs &ag = args(g, pair0);
    if (g + step < ngroups) {
      unsigned npair0;
      const XformArgs &an = args(g + step, npair0);
      fx_prefetch_lines<P / 2>(an, npair0);
    }
    xlamb_fx_group<CLS>(ag, pair0, R, tw, bd, sc, mag);
  }
}

template <int CLS>
__global__ void __launch_bounds__(FxCfg<CLS>::TX *FxCfg<CLS>::T, FxCfg<CLS>::ZB)
    k_zback_fx(const __grid_constant__ XformArgs a) {
  zback_fx_body<CLS>(a, blockIdx.x, blockIdx.y, blockIdx.z);
}
template <int CLS>
__global__ void __launch_bounds__(FxCfg<CLS>::TX *FxCfg<CLS>::T, FxCfg<CLS>::ZB)
    k_zfwd_fx(const __grid_constant__ XformArgs a) {
  zfwd_fx_body<CLS>(a, blockIdx.x, blockIdx.y, blockIdx.z);
}
template <int CLS>
__global__ void __launch_bounds__(3 * FxCfg<CLS>::P *FxCfg<CLS>::T, FxCfg<CLS>::XB)
    k_xlamb_fx(const __grid_constant__ XformArgs a) {
  constexpr int P = FxCfg<CLS>::P;
  const XformArgs *pa = &a;
  xlamb_fx_run<CLS>(blockIdx.x, gridDim.x, fx_groups(a.d, P), [pa](int g, unsigned &pair0) -> const XformArgs & {
    pair0 = (unsigned)g * (P / 2);
    return *pa;
  });
}

// Batched: as the kernels of transforms.cu, blocks numbered channel by channel.
template <int CLS>
__global__ void __launch_bounds__(FxCfg<CLS>::TX *FxCfg<CLS>::T, FxCfg<CLS>::ZB)
    k_zback_fx_batch(const __grid_constant__ BatchTable<XformArgs> t) {
  const int c = batch_channel(t.start, t.n, blockIdx.x);
  const XformArgs &a = t.a[c];
  const int gx = (a.d.NXH + FxCfg<CLS>::TX - 1) / FxCfg<CLS>::TX, lb = blockIdx.x - t.start[c], r = lb / gx;
  zback_fx_body<CLS>(a, lb - r * gx, r % a.d.NY, r / a.d.NY);
}
template <int CLS>
__global__ void __launch_bounds__(FxCfg<CLS>::TX *FxCfg<CLS>::T, FxCfg<CLS>::ZB)
    k_zfwd_fx_batch(const __grid_constant__ BatchTable<XformArgs> t) {
  const int c = batch_channel(t.start, t.n, blockIdx.x);
  const XformArgs &a = t.a[c];
  const int gx = (a.d.NXH + FxCfg<CLS>::TX - 1) / FxCfg<CLS>::TX, lb = blockIdx.x - t.start[c], r = lb / gx;
  zfwd_fx_body<CLS>(a, lb - r * gx, r % a.d.NY, r / a.d.NY);
}
template <int CLS>
__global__ void __launch_bounds__(3 * FxCfg<CLS>::P *FxCfg<CLS>::T, FxCfg<CLS>::XB)
    k_xlamb_fx_batch(const __grid_constant__ BatchTable<XformArgs> t) {
  xlamb_fx_run<CLS>(blockIdx.x, gridDim.x, t.start[t.n], [&](int g, unsigned &pair0) -> const XformArgs & {
    const int c = batch_channel(t.start, t.n, g);
    pair0 = (unsigned)(g - t.start[c]) * (FxCfg<CLS>::P / 2);
    return t.a[c];
  });
}

// The kernels of a class for z lines of NZ2 and x lines of NX2 points (each
// used where the line's plan is of this class).
template <int CLS>
FxXformKernels fx_kernels_of_class(int L) {
  const FxPlan p = fx_plan(L);
  FxXformKernels k;
  if (p.cls != CLS) return k;
  k.ok = true;
  k.zback = k_zback_fx<CLS>;
  k.zfwd = k_zfwd_fx<CLS>;
  k.xlamb = k_xlamb_fx<CLS>;
  k.zback_b = k_zback_fx_batch<CLS>;
  k.zfwd_b = k_zfwd_fx_batch<CLS>;
  k.xlamb_b = k_xlamb_fx_batch<CLS>;
  k.tx = FxCfg<CLS>::TX;
  k.zthreads = FxCfg<CLS>::TX * p.T;
  k.zsmem = fx_zsmem<CLS>(L);
  k.xlines = FxCfg<CLS>::P;
  k.xthreads = 3 * FxCfg<CLS>::P * p.T;
  k.xsmem = fx_xsmem<CLS>(p.A, p.B);
  return k;
}

}  // namespace owt
