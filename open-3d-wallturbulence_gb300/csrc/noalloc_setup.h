// The DY1 operator of owt_dy1_noalloc, built by each block of its kernel in
// shared memory: grid metric c11, the B1 rows and the A1 band, then the band
// LU.  Written as host/device functions so that a host program can build the
// same tables and compare them with setup_host.cpp's make_grid and
// make_stencils (the handle's DY1), which restate src/compdiff.hpp:11-69 and
// src/solver.cpp:77,94.
#pragma once
#include <math.h>
#include <stdint.h>

#ifndef __CUDACC__
#ifndef __host__
#define __host__
#define __device__
#endif
#endif

namespace owt {

// Largest NY the tables are laid out for (the entry point's OWT_NOALLOC_MAX_NY).
constexpr int kNoallocMaxNY = 1025;
constexpr int kNoallocKL = 2, kNoallocKU = 2, kNoallocKV = kNoallocKL + kNoallocKU;
constexpr int kNoallocBandRows = 2 * kNoallocKL + kNoallocKU + 1;

struct NoallocSetup {
  double *ab;    // kNoallocBandRows x NY band, LAPACK factorization layout (row KV = diagonal)
  double *c11;   // NY
  double *bval;  // NY x 5: B1 row entries, zero-padded
  int *bcol;     // NY x 5: their columns
  uint8_t *piv;  // NY: row interchange offset of each column
};

// The tables for up to nmax rows at base (8-byte aligned).
__host__ __device__ inline NoallocSetup noalloc_layout(unsigned char *base, int nmax = kNoallocMaxNY) {
  NoallocSetup s;
  s.ab = reinterpret_cast<double *>(base);
  s.c11 = s.ab + kNoallocBandRows * nmax;
  s.bval = s.c11 + nmax;
  s.bcol = reinterpret_cast<int *>(s.bval + 5 * nmax);
  s.piv = reinterpret_cast<uint8_t *>(s.bcol + 5 * nmax);
  return s;
}
// Bytes the layout spans.
__host__ __device__ constexpr size_t noalloc_setup_bytes(int nmax = kNoallocMaxNY) {
  return (size_t)nmax * (kNoallocBandRows + 1 + 5) * sizeof(double) + (size_t)nmax * 5 * sizeof(int) + (size_t)nmax;
}

// A1 entry (i, j): eighth-order interior, fourth-order rows 1 and NY-2,
// third-order closures at the walls.
__host__ __device__ inline double noalloc_a1(int i, int j, int NY) {
  const int d = i < j ? j - i : i - j;
  if (i < 0 || i >= NY || d > 2) return 0.0;
  if (i == 0 || i == NY - 1) return d == 0 ? 1.0 : d == 1 ? 3.0 : 0.0;
  if (i == 1 || i == NY - 2) return d == 0 ? 1.0 : d == 1 ? 0.25 : 0.0;
  return d == 0 ? 1.0 : d == 1 ? 4.0 / 9.0 : 1.0 / 36.0;
}

// c11 = 1/(dy/ds) on y = tanh(alpha s)/tanh(alpha), the B1 rows and the
// unfactored A1 band.  Everything the derivative kernel reads is written, fill
// rows cleared, so nothing depends on an earlier call.  Thread t of nt takes
// every nt-th row and column.
__host__ __device__ inline void noalloc_assemble(NoallocSetup s, int NY, double alpha, int t = 0, int nt = 1) {
  const double h = 2.0 / (NY - 1.0);
  const double coth_ap = 1.0 / tanh(alpha);
  const double a = 40.0 / 27.0, b = 25.0 / 54.0;
  const double a0 = -17.0 / 6.0, b0 = 1.5, c0 = 1.5, d0 = -1.0 / 6.0;
  for (int i = t; i < NY; i += nt) {
    const double si = 2 * i / (NY - 1.0) - 1.0;
    const double sech = 1.0 / cosh(alpha * si);
    s.c11[i] = 1.0 / (alpha * coth_ap * sech * sech);
    // entries of row i in increasing column order (the handle's B1 row order)
    auto put = [&](int k, int col, double v) {
      s.bcol[i * 5 + k] = col;
      s.bval[i * 5 + k] = v;
    };
    for (int k = 0; k < 5; ++k) put(k, 0, 0.0);
    if (i == 0) {
      put(0, 0, a0 / h);
      put(1, 1, b0 / h);
      put(2, 2, c0 / h);
      put(3, 3, d0 / h);
    } else if (i == NY - 1) {
      put(0, NY - 4, -d0 / h);
      put(1, NY - 3, -c0 / h);
      put(2, NY - 2, -b0 / h);
      put(3, NY - 1, -a0 / h);
    } else if (i == 1 || i == NY - 2) {
      put(0, i - 1, -1.5 / (2 * h));
      put(1, i + 1, 1.5 / (2 * h));
    } else {
      put(0, i - 2, -b / (4 * h));
      put(1, i - 1, -a / (2 * h));
      put(2, i + 1, a / (2 * h));
      put(3, i + 2, b / (4 * h));
    }
    // band column j = i: entry (q, j) at row KV + q - j
    for (int r = 0; r < kNoallocBandRows; ++r) s.ab[r * NY + i] = noalloc_a1(i + r - kNoallocKV, i, NY);
  }
}

// One column of the band LU with partial pivoting in place, the algorithm of
// LAPACK dgbtf2 (the handle's factorization order); ju: the last column
// touched so far.
__host__ __device__ inline void noalloc_factor_column(NoallocSetup s, int NY, int j, int &ju) {
  constexpr int KL = kNoallocKL, KU = kNoallocKU, KV = kNoallocKV;
  auto AB = [&](int r, int c) -> double & { return s.ab[r * NY + c]; };
  const int km = KL < NY - 1 - j ? KL : NY - 1 - j;
  int jp = 0;
  double best = fabs(AB(KV, j));
  for (int i = 1; i <= km; ++i) {
    const double v = fabs(AB(KV + i, j));
    if (v > best) {
      best = v;
      jp = i;
    }
  }
  s.piv[j] = (uint8_t)jp;
  const int reach = j + KU + jp < NY - 1 ? j + KU + jp : NY - 1;
  ju = ju > reach ? ju : reach;
  if (jp != 0)
    for (int c = j; c <= ju; ++c) {
      const double t = AB(KV + jp - (c - j), c);
      AB(KV + jp - (c - j), c) = AB(KV - (c - j), c);
      AB(KV - (c - j), c) = t;
    }
  const double rp = 1.0 / AB(KV, j);
  for (int i = 1; i <= km; ++i) AB(KV + i, j) *= rp;
  for (int c = j + 1; c <= ju; ++c) {
    const double t = AB(KV - (c - j), c);
    if (t != 0.0)
      for (int i = 1; i <= km; ++i) AB(KV + i - (c - j), c) -= AB(KV + i, j) * t;
  }
}

// The whole factorization; the diagonal row then holds 1/U_jj.
__host__ __device__ inline void noalloc_factor(NoallocSetup s, int NY) {
  int ju = 0;
  for (int j = 0; j < NY; ++j) noalloc_factor_column(s, NY, j, ju);
  for (int j = 0; j < NY; ++j) s.ab[kNoallocKV * NY + j] = 1.0 / s.ab[kNoallocKV * NY + j];
}

// The same factors by nt threads of a block; sync() is their barrier, state
// two ints they share.  The interior rows of A1 are all alike, so the
// elimination converges: once two successive columns, without interchange,
// leave the same 2 x 2 window behind (bit for bit), every further column whose
// rows are interior repeats them.  Thread 0 eliminates up to there (column 29
// or so), all threads write the repeated columns, thread 0 the last ones.
template <class Sync>
__host__ __device__ inline void noalloc_factor_block(NoallocSetup s, int NY, int t, int nt, int *state, Sync sync) {
  constexpr int KV = kNoallocKV;
  auto AB = [&](int r, int c) -> double & { return s.ab[r * NY + c]; };
  const int last = NY - 5;  // the last column that touches interior rows only
  if (t == 0) {
    int ju = 0, j = 0;
    double p = 0.0, q = 0.0, r = 0.0, w = 0.0;
    for (; j < NY; ++j) {
      noalloc_factor_column(s, NY, j, ju);
      if (j >= last) continue;
      const double p1 = AB(KV, j + 1), q1 = AB(KV - 1, j + 2), r1 = AB(KV + 1, j + 1), w1 = AB(KV, j + 2);
      if (j > 8 && s.piv[j] == 0 && s.piv[j - 1] == 0 && s.piv[j - 2] == 0 && ju == j + 2 && p1 == p && q1 == q &&
          r1 == r && w1 == w)
        break;
      p = p1; q = q1; r = r1; w = w1;
    }
    state[0] = j;  // NY: everything is done
    state[1] = ju;
  }
  sync();
  const int j0 = state[0];
  if (j0 < NY) {
    // columns j0 + 1 .. last repeat column j0; the window goes along
    const double w = AB(KV, j0 + 2), q = AB(KV - 1, j0 + 2), u = AB(KV, j0), u1 = AB(KV - 1, j0 + 1), u2 = AB(KV - 2, j0),
                 l1 = AB(KV + 1, j0), l2 = AB(KV + 2, j0), p = AB(KV, j0 + 1), r = AB(KV + 1, j0 + 1);
    sync();
    for (int c = j0 + 1 + t; c <= last; c += nt) {
      AB(0, c) = 0.0;
      AB(1, c) = 0.0;
      AB(KV - 2, c) = u2;
      AB(KV - 1, c) = u1;
      AB(KV, c) = u;
      AB(KV + 1, c) = l1;
      AB(KV + 2, c) = l2;
      s.piv[c] = 0;
    }
    sync();
    if (t == 0) {
      AB(KV - 1, last + 1) = u1;
      AB(KV, last + 1) = p;
      AB(KV + 1, last + 1) = r;
      AB(KV - 1, last + 2) = q;
      AB(KV, last + 2) = w;
      int ju = last + 2;
      for (int j = last + 1; j < NY; ++j) noalloc_factor_column(s, NY, j, ju);
    }
    sync();
  }
  for (int j = t; j < NY; j += nt) AB(KV, j) = 1.0 / AB(KV, j);
  sync();
}

}  // namespace owt
