// The mode kernel on packed factor streams: an omega_y warp and a v warp per
// 16 unique modes and sign of kz.  The omega_y warp forms source_g and solves
// for g and DY1 g, the v warp forms source_v and runs the v-system's forward
// sweep beside it; a named barrier of the two warps orders the omega_y results
// before the backward sweep that reads them.
//
// One warp issues an FP64 instruction every 64 clocks at best, so what a
// column costs beside its FP64 instructions decides the speed: the mappings
// that read the band storage spend 16 instructions for each FP64 one (address
// arithmetic, edge tests, unrolled ring phases that miss the instruction
// cache).  Here
//  - the factors of 16 unique modes are packed into one contiguous stream per
//    sweep, in the order the sweep reads them and without the entries outside
//    the interior masks; a warp copies it into a three-slot ring in shared
//    memory with 16-byte cp.async, two units ahead (unit: four interior
//    columns, or one column near a wall), and reads it at constant offsets;
//  - the window of the solve is a shift register (moves, not ring phases), so
//    each sweep is two short loops;
//  - right-hand sides and forward-swept values live in scratch of the warp's
//    own, one row of 32 lanes per unknown, read four rows ahead.
// Every value comes from the operations of mode_body in the same order, so
// results are bitwise those of the other mappings.
//
// Measured, best other mapping -> this one: 384x257x384 13.85 -> 11.6 ms (bound
// by the FP64 pipe, 84% busy in a capture of 384x33x384), 320x160x320 7.5 -> 5.6,
// 128x129x128 1.81 -> 1.0, 64x97x48 1.38 -> 0.73, 32x65x32 0.62 -> 0.49 (a warp's
// own FP64 instructions 0.53 of the 128x129x128 time; the fullest SMs have four of
// the 520 blocks there, the average 3.4), the 64-channel ensemble 4.79 -> 3.76.  A
// cp.async ring over the band storage without packing gave 1.50 at
// 128x129x128: 16 instructions for each FP64 one, against 9.8 here.
//
// Lanes 2q, 2q + 1 are Re, Im of unique mode 16 g + q (group g = warp / 2) with
// the sign of kz of the warp (warp & 1: -kz); kz = 0 and the Nyquist row have
// no negative partner, those lanes idle.
#pragma once
#include "modes_kernel.cuh"

namespace owt {

__device__ __forceinline__ void named_bar_sync(int id, int nthreads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}
__device__ __forceinline__ void named_bar_arrive(int id, int nthreads) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}

constexpr int kStrModes = 16;  // unique modes of a group
constexpr int kStrSlots = 3;   // units in the shared-memory ring

__host__ __device__ constexpr int bits_in(unsigned long long m) {
  int c = 0;
  for (; m; m &= m - 1) ++c;
  return c;
}
// set bits of m below bit t
__host__ __device__ constexpr int bits_below(unsigned long long m, int t) { return bits_in(m & ((1ull << t) - 1ull)); }

// One of the two systems: band widths, unknowns per node, masks, and the
// windows of its interior loops (rows in flight while four columns are done).
template <class VM>
struct StrV : VM {
  static constexpr int KL = kVKL, KU = kVKU, KV = KL + KU, NT = 4, OFF = 2, WF = 16, WI = 24;
};
struct StrG : GMasks {
  static constexpr int KL = 6, KU = 6, KV = 12, NT = 2, OFF = 0, WF = 8, WI = 8;
};

// Layout of the streams (in doubles, per group): the forward stream holds for
// each unit 16 words of pivot offsets (one byte per column), then the entries
// [column][entry][mode]; the backward stream the entries, diagonal first.
template <class S>
struct StrLayout {
  __host__ __device__ static constexpr int type_f(int s) { return (s + S::OFF) % S::NT; }               // column lo + 4 q + s
  __host__ __device__ static constexpr int type_b(int s) { return (S::OFF - 1 - s + 4 * S::NT) % S::NT; }  // column n - 1 - hi - 4 q - s
  __host__ __device__ static constexpr unsigned long long mask_f(int s) { return S::l(type_f(s)); }
  __host__ __device__ static constexpr unsigned long long mask_b(int s) { return S::u(type_b(s)) | 1ull; }
  __host__ __device__ static constexpr int before_f(int s) { return s == 0 ? 0 : before_f(s - 1) + bits_in(mask_f(s - 1)); }
  __host__ __device__ static constexpr int before_b(int s) { return s == 0 ? 0 : before_b(s - 1) + bits_in(mask_b(s - 1)); }
  static constexpr int EF = 16 + S::KL * 16, EB = (S::KV + 1) * 16;              // an edge column
  static constexpr int IF = 16 + before_f(4) * 16, IB = before_b(4) * 16;        // four interior columns
  static constexpr int slot = IB > EB ? (IB > IF ? IB : IF) : (EB > IF ? EB : IF);
  // columns up to lo and from n - hi are edge columns (all of a short system;
  // two more than the masks ask for where n is not a multiple of 4)
  __host__ __device__ static int quads(int n) { return n >= S::lo + S::hi ? (n - S::lo - S::hi) / 4 : 0; }
  __host__ __device__ static int lo(int n) { return quads(n) ? n - S::hi - 4 * quads(n) : n; }
  __host__ __device__ static int hi(int n) { return quads(n) ? S::hi : 0; }
  __host__ __device__ static size_t fwd_size(int n) { return (size_t)(lo(n) + hi(n)) * EF + (size_t)quads(n) * IF; }
  __host__ __device__ static size_t bwd_size(int n) { return (size_t)(lo(n) + hi(n)) * EB + (size_t)quads(n) * IB; }
  static_assert(S::lo % S::NT == 0 && S::hi % S::NT == 0 && 4 % S::NT == 0, "types in whole quads");
};

// Pack the factors of every group: grid (groups, blocks of columns), 16 threads
// (modes) per column.
template <class S>
__global__ void k_str_pack(const double *__restrict__ ab, const uint8_t *__restrict__ piv, int n, int U,
                           double *__restrict__ fwd, double *__restrict__ bwd) {
  using Y = StrLayout<S>;
  const int q = threadIdx.x, c = blockIdx.y * blockDim.y + threadIdx.y, g = blockIdx.x;
  if (c >= n) return;
  const int u = min(g * kStrModes + q, U - 1);  // the last group repeats the last mode
  const size_t sn = (size_t)n * U;
  const double *col = ab + (size_t)c * U + u;
  const int lo = Y::lo(n), hi = Y::hi(n), nq = Y::quads(n);
  const unsigned off = piv[(size_t)c * U + u];
  double *f = fwd + (size_t)g * Y::fwd_size(n), *b = bwd + (size_t)g * Y::bwd_size(n);
  const bool interior = nq > 0 && c >= lo && c < n - hi;
  if (!interior) {
    f += c < lo ? (size_t)c * Y::EF : (size_t)lo * Y::EF + (size_t)nq * Y::IF + (size_t)(c - (n - hi)) * Y::EF;
    reinterpret_cast<unsigned *>(f)[q] = off;
    for (int t = 1; t <= S::KL; ++t) f[16 + (t - 1) * 16 + q] = col[(size_t)(S::KV + t) * sn];
    const int k = n - 1 - c;
    b += k < hi ? (size_t)k * Y::EB
                : nq > 0 ? (size_t)hi * Y::EB + (size_t)nq * Y::IB + (size_t)(k - hi - 4 * nq) * Y::EB : (size_t)k * Y::EB;
    for (int t = 0; t <= S::KV; ++t) b[t * 16 + q] = col[(size_t)(S::KV - t) * sn];
    return;
  }
  {
    const int x = c - lo, s = x & 3, ty = (s + S::OFF) % S::NT;
    f += (size_t)lo * Y::EF + (size_t)(x >> 2) * Y::IF;
    reinterpret_cast<unsigned char *>(reinterpret_cast<unsigned *>(f) + q)[s] = (unsigned char)off;
    int before = 0;
    for (int r = 0; r < s; ++r) before += bits_in(S::l((r + S::OFF) % S::NT));
    const unsigned long long m = S::l(ty);
    for (int t = 1, e = before; t <= S::KL; ++t)
      if ((m >> t) & 1ull) f[16 + 16 * (e++) + q] = col[(size_t)(S::KV + t) * sn];
  }
  {
    const int x = n - 1 - c - hi, s = x & 3, ty = (S::OFF - 1 - s + 4 * S::NT) % S::NT;
    b += (size_t)hi * Y::EB + (size_t)(x >> 2) * Y::IB;
    int before = 0;
    for (int r = 0; r < s; ++r) before += 1 + bits_in(S::u((S::OFF - 1 - r + 4 * S::NT) % S::NT));
    const unsigned long long m = S::u(ty) | 1ull;
    for (int t = 0, e = before; t <= S::KV; ++t)
      if ((m >> t) & 1ull) b[16 * (e++) + q] = col[(size_t)(S::KV - t) * sn];
  }
}

__device__ __forceinline__ void str_copy16(void *smem, const void *g) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(g));
}
__device__ __forceinline__ void str_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void str_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// The compiler cannot tell scratch pointers from shared memory by itself, and
// would not read a column's entries ahead of an earlier store.
template <class T>
__device__ __forceinline__ T *str_global(T *p) {
  __builtin_assume(__isGlobal(p));
  return p;
}

// The stream of one sweep: units in turn through the ring.  All lanes of the
// warp call it together.
template <int SLOT>
struct StrFeed {
  const double *next;  // the next unit to fetch
  double *ring;
  int lane, put, get;
  __device__ __forceinline__ StrFeed(const double *stream, double *r, int ln) : next(stream), ring(r), lane(ln), put(0), get(0) {}
  // fetch a unit of SIZE doubles (SIZE = 0: none left) and close its group
  template <int SIZE>
  __device__ __forceinline__ void fetch() {
    constexpr int chunks = SIZE / 2;  // of 16 bytes
    double *dst = ring + put * SLOT + 2 * lane;
    const double *src = next + 2 * lane;
#pragma unroll
    for (int i = 0; i < (chunks + 31) / 32; ++i)
      if (32 * (i + 1) <= chunks || lane + 32 * i < chunks) str_copy16(dst + 64 * i, src + 64 * i);
    str_commit();
    next += SIZE;
    put = put == kStrSlots - 1 ? 0 : put + 1;
  }
  // wait for the current unit (two fetches follow it); its address
  __device__ __forceinline__ const double *ready() {
    str_wait<1>();
    __syncwarp();
    const double *p = ring + get * SLOT;
    get = get == kStrSlots - 1 ? 0 : get + 1;
    return p;
  }
};

// The same for the transposed solves, which read a sweep's stream from its end:
// units in descending order.
template <int SLOT>
struct StrFeedBack : StrFeed<SLOT> {
  using Base = StrFeed<SLOT>;
  __device__ __forceinline__ StrFeedBack(const double *end, double *r, int ln) : Base(end, r, ln) {}
  template <int SIZE>
  __device__ __forceinline__ void fetch() {
    this->next -= SIZE;
    Base::template fetch<SIZE>();
    this->next -= SIZE;
  }
};

// Forward sweep.  rows: the warp's scratch plus the lane, row p at rows[32 p],
// right-hand sides on entry, forward-swept values on return.
template <class S>
__device__ __forceinline__ void str_forward(const double *stream, int n, double *ring, int lane, double *rows) {
  using Y = StrLayout<S>;
  constexpr int KL = S::KL, W = S::WF;
  const int lo = Y::lo(n), nq = Y::quads(n), q = lane >> 1;
  StrFeed<Y::slot> feed(stream, ring, lane);
  // unit i: edge for i < lo and i >= lo + nq
  const int units = lo + Y::hi(n) + nq;
  auto fetch = [&](int i) {
    if (i >= lo && i < lo + nq) feed.template fetch<Y::IF>();
    else if (i < units) feed.template fetch<Y::EF>();
    else feed.template fetch<0>();
  };
  fetch(0);
  fetch(1);
  double w[W];
  auto row = [&](int p) { return p < n ? rows[32 * p] : 0.0; };
#pragma unroll
  for (int t = 0; t < W; ++t) w[t] = row(t);
  double nx = row(W);  // the row that enters next
  int j = 0, unit = 0;
  auto edge = [&](int count) {
#pragma unroll 1
    for (int e = 0; e < count; ++e, ++j, ++unit) {
      const double *c = feed.ready();
      fetch(unit + 2);
      const int off = (int)reinterpret_cast<const unsigned *>(c)[q];
      const double *l = c + 16 + q;
      if (off) {
#pragma unroll
        for (int t = 1; t <= KL; ++t)
          if (off == t) {
            const double tmp = w[0];
            w[0] = w[t];
            w[t] = tmp;
          }
      }
      const double y = w[0];
      rows[32 * j] = y;
#pragma unroll
      for (int t = 1; t <= KL; ++t) fms(w[t], l[(t - 1) * 16], y);
#pragma unroll
      for (int t = 0; t < W - 1; ++t) w[t] = w[t + 1];
      w[W - 1] = nx;
      nx = row(j + W + 1);
    }
  };
  edge(lo);
  if (nq > 0) {
    // rows j + W .. j + W + 3 enter after the next four columns
    double in[4] = {nx, row(j + W + 1), row(j + W + 2), row(j + W + 3)};
#pragma unroll 1
    for (int e = 0; e < nq; ++e, j += 4, ++unit) {
      const double *c = feed.ready();
      fetch(unit + 2);
      const unsigned off = reinterpret_cast<const unsigned *>(c)[q];
      const double *l = c + 16 + q;
      double *o = rows + 32 * j;
      fx_for<0, 4>([&](auto sc) {
        constexpr int s = decltype(sc)::value;
        constexpr unsigned long long ml = Y::mask_f(s), mp = S::p(Y::type_f(s));
        static_assert((ml >> (W - s)) == 0, "window too short for the masks");
        if constexpr (mp != 0) {
          const int of = (off >> (8 * s)) & 0xff;
          fx_for<1, KL + 1>([&](auto tc) {
            constexpr int t = decltype(tc)::value;
            if constexpr ((mp >> t) & 1ull)
              if (of == t) {
                const double tmp = w[s];
                w[s] = w[s + t];
                w[s + t] = tmp;
              }
          });
        }
        const double y = w[s];
        o[32 * s] = y;
        fx_for<1, KL + 1>([&](auto tc) {
          constexpr int t = decltype(tc)::value;
          if constexpr ((ml >> t) & 1ull) fms(w[s + t], l[(Y::before_f(s) + bits_below(ml, t)) * 16], y);
        });
      });
#pragma unroll
      for (int t = 0; t < W - 4; ++t) w[t] = w[t + 4];
#pragma unroll
      for (int t = 0; t < 4; ++t) w[W - 4 + t] = in[t];
#pragma unroll
      for (int t = 0; t < 4; ++t) in[t] = row(j + 4 + W + t);
    }
    nx = in[0];
    edge(Y::hi(n));
  }
  str_wait<0>();
  __syncwarp();
}

// Backward sweep; out(type, c, x) for c = n - 1 .. 0, `type` the interior
// column's step s in its quad, or 4 for an edge column.
template <class S, class Out>
__device__ __forceinline__ void str_backward(const double *stream, int n, double *ring, int lane, double *rows, Out out) {
  using Y = StrLayout<S>;
  constexpr int KV = S::KV, W = (KV + 1 + 3) / 4 * 4, WI = S::WI;
  static_assert(WI < W, "interior window");
  const int hi = Y::hi(n) + (Y::quads(n) ? 0 : Y::lo(n)), nq = Y::quads(n), q = lane >> 1;
  StrFeed<Y::slot> feed(stream, ring, lane);
  const int units = Y::lo(n) + Y::hi(n) + nq;
  auto fetch = [&](int i) {
    if (i >= hi && i < hi + nq) feed.template fetch<Y::IB>();
    else if (i < units) feed.template fetch<Y::EB>();
    else feed.template fetch<0>();
  };
  fetch(0);
  fetch(1);
  auto row = [&](int p) { return p >= 0 ? rows[32 * p] : 0.0; };
  double w[W];
#pragma unroll
  for (int t = 0; t < W; ++t) w[t] = row(n - 1 - t);
  double nx = row(n - 1 - W);
  int j = n - 1, unit = 0;
  auto edge = [&](int count) {
#pragma unroll 1
    for (int e = 0; e < count; ++e, --j, ++unit) {
      const double *c = feed.ready();
      fetch(unit + 2);
      c += q;
      const double x = w[0] * c[0];
      out(std::integral_constant<int, 4>{}, j, x);
#pragma unroll
      for (int t = 1; t <= KV; ++t) fms(w[t], c[t * 16], x);
#pragma unroll
      for (int t = 0; t < W - 1; ++t) w[t] = w[t + 1];
      w[W - 1] = nx;
      nx = row(j - W - 1);
    }
  };
  edge(hi);
  if (nq > 0) {
    // rows beyond the interior window go back with their pending updates
#pragma unroll
    for (int t = WI; t < W; ++t) rows[32 * (j - t)] = w[t];
    double in[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) in[t] = row(j - WI - t);
#pragma unroll 1
    for (int e = 0; e < nq; ++e, j -= 4, ++unit) {
      const double *c = feed.ready();
      fetch(unit + 2);
      c += q;
      fx_for<0, 4>([&](auto sc) {
        constexpr int s = decltype(sc)::value;
        constexpr unsigned long long m = Y::mask_b(s);
        static_assert((m >> (WI - s)) == 0, "window too short for the masks");
        const double x = w[s] * c[Y::before_b(s) * 16];
        out(sc, j - s, x);
        fx_for<1, KV + 1>([&](auto tc) {
          constexpr int t = decltype(tc)::value;
          if constexpr ((m >> t) & 1ull) fms(w[s + t], c[(Y::before_b(s) + bits_below(m, t)) * 16], x);
        });
      });
#pragma unroll
      for (int t = 0; t < WI - 4; ++t) w[t] = w[t + 4];
#pragma unroll
      for (int t = 0; t < 4; ++t) w[WI - 4 + t] = in[t];
#pragma unroll
      for (int t = 0; t < 4; ++t) in[t] = row(j - 4 - WI - t);
    }
#pragma unroll
    for (int t = WI; t < W; ++t) w[t] = row(j - t);
    nx = row(j - W);
    edge(Y::lo(n));
  }
  str_wait<0>();
  __syncwarp();
}

// This lane's mode.
struct StrLane {
  int m, comp, u, lane;
  bool active;
};
template <class Args>
__device__ __forceinline__ StrLane str_lane(const Args &a, int warp, int lane) {
  StrLane l;
  l.lane = lane;
  l.comp = lane & 1;
  const int uq = (warp >> 1) * kStrModes + (lane >> 1);
  l.active = uq >= a.u0 && uq < a.u1;
  l.u = min(uq, a.U - 1);
  const int kabs = l.u / a.NXH, i = l.u - kabs * a.NXH;
  int k = kabs;
  if (warp & 1) {
    if (kabs == 0 || kabs == a.NZH) l.active = false;  // no -kz partner
    else k = a.NZ - kabs;
  }
  l.m = k * a.NXH + i;
  return l;
}

// The omega_y warp: steps 1 and 2 of mode_body.  sg, dg: rows j of the warp's
// scratch (source_g; DY1 g, read by the v warp); yg: rows p.
__device__ __forceinline__ void str_g(const ModeArgs &a, const StrLane &L, int warp, double *ring) {
  const int M = a.M, NY = a.NY, n = a.n_g;
  const int h = ring_head(*a.step);
  const size_t fs2 = 2 * (size_t)NY * M;
  const size_t e0 = 2 * (size_t)L.m + L.comp, row = 2 * (size_t)M;
  auto lvl = [&](const double2 *r, int l) { return reinterpret_cast<const double *>(r) + (size_t)((h + l) % 3) * fs2 + e0; };
  const double *in[6] = {lvl(a.g_ring, 0), lvl(a.g_ring, 1), lvl(a.g_ring, 2),
                         lvl(a.hg_ring, 0), lvl(a.hg_ring, 1), lvl(a.hg_ring, 2)};
  double *sg = str_global(reinterpret_cast<double *>(a.sg) + (size_t)warp * NY * 32 + L.lane);
  double *dg = str_global(reinterpret_cast<double *>(a.dg) + (size_t)warp * NY * 32 + L.lane);
  double *yg = str_global(reinterpret_cast<double *>(a.yg) + (size_t)warp * n * 32 + L.lane);
  const double idt = a.inv_dt, ag0 = 3.0 * idt, ag1 = -1.5 * idt, ag2 = (1.0 / 3.0) * idt, be0 = 3.0;
  {
    // source_g row by row, and the right-hand sides whose last node it is:
    // weights on the last five nodes (r[4] the newest)
    double r[5] = {0.0, 0.0, 0.0, 0.0, 0.0}, x[2][6];
    const double *rsp = a.grs + L.u;  // row scales in the order of the rows, read four ahead
    const int last = a.gptr[NY] - 1;
    double rs[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) rs[i] = rsp[(size_t)min(i, last) * a.U];
    int e = 0;
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      x[0][i] = in[i][0];
      x[1][i] = in[i][row];
    }
#pragma unroll 2
    for (int j = 0; j < NY; ++j) {
      double v[6];
      const size_t at = (size_t)(j + 2 < NY ? j + 2 : NY - 1) * row;
#pragma unroll
      for (int i = 0; i < 6; ++i) {
        v[i] = x[0][i];
        x[0][i] = x[1][i];
        x[1][i] = in[i][at];
      }
      double s = 0.0;
      if (j != 0 && j != NY - 1) s = fma(v[2], ag2, fma(v[1], ag1, fma(v[0], ag0, fma(v[3] - v[4], be0, v[5]))));
      sg[32 * j] = s;
#pragma unroll
      for (int i = 0; i < 4; ++i) r[i] = r[i + 1];
      r[4] = s;
      for (const int end = a.gptr[j + 1]; e < end; ++e) {
        const StrRow &w = a.grows[e];
        const double sc = rs[0];
#pragma unroll
        for (int i = 0; i < 3; ++i) rs[i] = rs[i + 1];
        rs[3] = rsp[(size_t)min(e + 4, last) * a.U];
        double acc = 0.0;
#pragma unroll
        for (int i = 0; i < 5; ++i)
          if (i != 2 || nonzero(w.w[2])) acc = fma(w.w[i], r[i], acc);  // no centre tap in the first derivative's rows
        yg[32 * w.p] = __dmul_rn(acc, sc);
      }
    }
  }
  const size_t g = warp >> 1;
  str_forward<StrG>(a.gf + g * StrLayout<StrG>::fwd_size(n), n, ring, L.lane, yg);
  const double icg = a.inv_cg[L.u];
  double *gn = str_global(const_cast<double *>(lvl(a.g_ring, 2)));
  double d2 = 0.0, s = sg[32 * (NY - 1)], c1 = a.nc21h[NY - 1], c2 = a.nc22h[NY - 1], c11 = a.c11h[NY - 1];
  auto out = [&](auto, int c, double x) {
    const int jn = c >> 1;
    if (c & 1) {
      d2 = x;
      return;
    }
    double v = 0.0;
    if (jn != 0 && jn != NY - 1) v = fma(c2, d2, fma(c1, x, s)) * icg;
    if (L.active) gn[(size_t)jn * row] = v;
    dg[32 * jn] = c11 * x;
    const int jp = jn > 0 ? jn - 1 : 0;  // the next node's values
    s = sg[32 * jp];
    c1 = a.nc21h[jp];
    c2 = a.nc22h[jp];
    c11 = a.c11h[jp];
  };
  str_backward<StrG>(a.gb + g * StrLayout<StrG>::bwd_size(n), n, ring, L.lane, yg, out);
}

// The v warp: steps 1, 3-5 of mode_body; `bar` orders the omega_y warp's
// results before the backward sweep that reads them.
template <class VM>
__device__ __forceinline__ void str_v(const ModeArgs &a, const StrLane &L, int warp, double *ring, int bar) {
  using S = StrV<VM>;
  const int M = a.M, NY = a.NY, n = a.n_v;
  const int h = ring_head(*a.step);
  const size_t fs2 = 2 * (size_t)NY * M;
  const size_t e0 = 2 * (size_t)L.m + L.comp, row = 2 * (size_t)M;
  auto lvl = [&](const double2 *r, int l) { return reinterpret_cast<const double *>(r) + (size_t)((h + l) % 3) * fs2 + e0; };
  const int kk = L.m / a.NXH;
  const double kx = a.kx[L.m - kk * a.NXH], kz = a.kz[kk], k2 = fma(kx, kx, kz * kz);
  double *yv = str_global(reinterpret_cast<double *>(a.yv) + (size_t)warp * n * 32 + L.lane);
  {
    const double *in[9] = {lvl(a.v_ring, 0),  lvl(a.v_ring, 1),  lvl(a.v_ring, 2),  lvl(a.hv_ring, 0), lvl(a.hv_ring, 1),
                           lvl(a.hv_ring, 2), lvl(a.q_ring, 0),  lvl(a.q_ring, 1),  lvl(a.q_ring, 2)};
    const double idt = a.inv_dt, k2dt = k2 * idt;
    const double ag0 = 3.0 * idt, ag1 = -1.5 * idt, ag2 = (1.0 / 3.0) * idt, be0 = 3.0;
    const double av0 = -k2dt * 3.0, av1 = -k2dt * -1.5, av2 = -k2dt * (1.0 / 3.0);
    // rows without interior equations: zero, or v = v_w on the walls (solver.cpp:593-596)
    for (int p = 0; p < n; ++p) {
      const int tag = a.rhs_node_v[p];
      if (tag == kRhsTable) continue;
      double r = 0.0;
      if (tag != kRhsNone && a.vw) {
        const double *vw = reinterpret_cast<const double *>(a.vw) + (tag == kRhsWallBottom ? 0 : 2 * (size_t)M);
        r = __dmul_rn(vw[e0], a.rs_v[(size_t)p * a.U + L.u]);
      }
      yv[32 * p] = r;
    }
    double r[3] = {0.0, 0.0, 0.0}, x[9];
    const double *rsp = a.vrs + L.u;  // row scales in the order of the rows, read two ahead
    const int last = a.vptr[NY] - 1;
    double rs[2] = {rsp[0], rsp[(size_t)min(1, last) * a.U]};
    int e = 0;
#pragma unroll
    for (int i = 0; i < 9; ++i) x[i] = in[i][0];
#pragma unroll 2
    for (int j = 0; j < NY; ++j) {
      double v[9];
      const size_t at = (size_t)(j + 1 < NY ? j + 1 : NY - 1) * row;
#pragma unroll
      for (int i = 0; i < 9; ++i) {
        v[i] = x[i];
        x[i] = in[i][at];
      }
      double rv = 0.0;
      if (j >= 2 && j <= NY - 3) {
        rv = fma(v[3] - v[4], be0, v[5]);
        rv = fma(v[0], av0, rv);
        rv = fma(v[1], av1, rv);
        rv = fma(v[2], av2, rv);
        rv = fma(v[6], ag0, rv);
        rv = fma(v[7], ag1, rv);
        rv = fma(v[8], ag2, rv);
      }
      r[0] = r[1];
      r[1] = r[2];
      r[2] = rv;
      for (const int end = a.vptr[j + 1]; e < end; ++e) {
        const StrRow &w = a.vrows[e];
        const double sc = rs[0];
        rs[0] = rs[1];
        rs[1] = rsp[(size_t)min(e + 2, last) * a.U];
        double acc = 0.0;
#pragma unroll
        for (int i = 0; i < 3; ++i) acc = fma(w.w[2 + i], r[i], acc);
        yv[32 * w.p] = __dmul_rn(acc, sc);
      }
    }
  }
  const size_t g = warp >> 1;
  str_forward<S>(a.vf + g * StrLayout<S>::fwd_size(n), n, ring, L.lane, yv);
  named_bar_sync(bar, 64);
  const bool horiz = L.active && !(k2 < 1.e-8);
  const double ik2 = horiz ? 1.0 / k2 : 0.0;
  const double sgn = L.comp ? 1.0 : -1.0;
  const double sax = sgn * kx * ik2, saz = sgn * kz * ik2, skx = sgn * kx, skz = sgn * kz;
  double *vn = str_global(const_cast<double *>(lvl(a.v_ring, 2)));
  double *qn = str_global(const_cast<double *>(lvl(a.q_ring, 2)));
  double *uo = str_global(reinterpret_cast<double *>(a.u_out) + e0), *wo = str_global(reinterpret_cast<double *>(a.w_out) + e0);
  double *oxo = str_global(reinterpret_cast<double *>(a.ox_out) + e0);
  double *ozo = str_global(reinterpret_cast<double *>(a.oz_out) + e0);
  // the omega_y values of the partner lane's component
  const double *go_ = lvl(a.g_ring, 2) + 1 - 2 * L.comp;
  const double *dg = reinterpret_cast<const double *>(a.dg) + (size_t)warp * NY * 32 + (L.lane ^ 1);
  double xv = 0.0, d1 = 0.0;
  double go = go_[(size_t)(NY - 1) * row], dgo = dg[32 * (NY - 1)];
  double c11 = a.c11h[NY - 1], c21 = a.c21h[NY - 1], c22 = a.c22h[NY - 1];
  auto finish = [&](int jn, double x, double d1, double d2) {
    const size_t e = (size_t)jn * row;
    const double q = fma(c22, d2, c21 * d1);
    const double dv = c11 * d1;
    const double xo = __shfl_xor_sync(0xffffffffu, x, 1), dvo = __shfl_xor_sync(0xffffffffu, dv, 1),
                 qo = __shfl_xor_sync(0xffffffffu, q, 1);
    if (L.active) {
      vn[e] = x;
      qn[e] = q;
    }
    if (horiz) {
      uo[e] = fma(sax, dvo, -(saz * go));
      wo[e] = fma(saz, dvo, sax * go);
      oxo[e] = fma(-skz, xo, fma(saz, qo, sax * dgo));
      ozo[e] = fma(skx, xo, fma(-sax, qo, saz * dgo));
    }
    const int jp = jn > 0 ? jn - 1 : 0;  // the next node's values
    go = go_[(size_t)jp * row];
    dgo = dg[32 * jp];
    c11 = a.c11h[jp];
    c21 = a.c21h[jp];
    c22 = a.c22h[jp];
  };
  double d2e = 0.0;
  auto out = [&](auto sc, int c, double x) {
    constexpr int s = decltype(sc)::value;
    if constexpr (s == 0) {  // column 4a + 3: d2 of node a, finished
      finish(c >> 2, xv, d1, x);
    } else if constexpr (s == 2) {  // v of the node below
      xv = x;
    } else if constexpr (s == 3) {
      d1 = x;
    } else if constexpr (s == 4) {
      int t, jn;
      vcol_split(c, NY, t, jn);
      const bool wall = jn < 2 || jn >= NY - 2;
      if (t == 0) {
        xv = x;
        if (wall) finish(jn, xv, d1, d2e);
      } else if (t == 1) {
        d1 = x;
      } else if (t == 2) {
        d2e = x;
        if (!wall) finish(jn, xv, d1, x);
      }
    }
  };
  str_backward<S>(a.vb + g * StrLayout<S>::bwd_size(n), n, ring, L.lane, yv, out);
}

constexpr int kStrRingV = kStrSlots * (StrLayout<StrV<VMasks>>::slot > StrLayout<StrV<VMasks6>>::slot
                                           ? StrLayout<StrV<VMasks>>::slot
                                           : StrLayout<StrV<VMasks6>>::slot);
constexpr int kStrRingG = kStrSlots * StrLayout<StrG>::slot;

// The 64 threads of one omega_y warp and one v warp; `warp` counts groups and
// signs.
template <class VM>
__device__ __forceinline__ void stream_body(const ModeArgs &a, int warp, double *ring) {
  const int lane = threadIdx.x & 31;
  const StrLane L = str_lane(a, warp, lane);
  if (!__any_sync(0xffffffffu, L.active)) return;  // both warps alike
  if (threadIdx.x < 32) {
    str_g(a, L, warp, ring + kStrRingV);
    __threadfence_block();  // g, DY1 g before the v warp's backward sweep reads them
    named_bar_arrive(1, 64);
  } else {
    str_v<VM>(a, L, warp, ring, 1);
  }
}

template <int MINB, class VM>
__global__ void __launch_bounds__(64, MINB) k_modes_stream(const __grid_constant__ ModeArgs a) {
  __shared__ __align__(16) double ring[kStrRingV + kStrRingG];
  stream_body<VM>(a, 2 * (a.u0 / kStrModes) + blockIdx.x, ring);
}

// Every channel of a batch, persistent as k_modes_batch: work items are the
// channels' groups and signs.
template <int MINB>
__global__ void __launch_bounds__(64, MINB)
    k_modes_stream_batch(const __grid_constant__ BatchTable<ModeArgs> t, int *work) {
  __shared__ __align__(16) double ring[kStrRingV + kStrRingG];
  __shared__ int item;
  const int total = t.start[t.n];
  for (;;) {
    if (threadIdx.x == 0) item = atomicAdd(work, 1);
    __syncthreads();  // also: both warps are done with the last item's ring and scratch
    const int it = item;
    __syncthreads();
    if (it >= total) break;
    const int c = batch_channel(t.start, t.n, it);
    stream_body<VMasks>(t.a[c], it - t.start[c], ring);
  }
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(work + 1, 1) == (int)gridDim.x - 1) {
      work[0] = 0;
      work[1] = 0;
    }
  }
}

}  // namespace owt
