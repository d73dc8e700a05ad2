// swm_strip.cuh -- the Jacobi solver's sweeps (jacobi_iteration.f90:25-87): a pass of up
// to kPassT sweeps over a piece of a system whose rows are held in registers.
//
// Two forms of the pass, with the same arithmetic:
//  strips  a warp owns 64 columns (a pair of adjacent cells per lane, kPassT of them halo
//          on each side) and walks down the rows of its chunk: when row s arrives, sweep t
//          computes row s - t from the rows of x^{t-1} that the previous step and the
//          previous sweep left in registers.  Rows come through a ring in shared memory
//          that only their own lane reads, so there is no barrier in the walk;
//  tiles   (passes of up to 4 or 8 sweeps) a block holds a 64-column tile, a few rows per
//          warp; the warps exchange their edge rows through shared memory after every
//          sweep.
// In both, west and east neighbours come from the next lanes, and each row of the system
// is read once per pass (tiles: once per solve when every block has one tile).
//
// Why: the pass these replace staged a haloed tile in shared memory and re-read it in
// every sweep: 11 loads per 2 cells and sweep, bound by shared-memory bandwidth (1.2 us
// per sweep of a 64 x 16 tile), after a load phase with no sweeps in flight.  A strip
// moves only what it must and suits grids that fill the GPU many times; a tile has a
// short serial path (all its loads in flight at once, then kPassT sweeps) and suits the
// others.
#pragma once
#include <cstdint>

#include "swm_solve.cuh"

namespace swm {

constexpr int kStripWarps = kJacobiBatchWarps;   // warps of a CTA (independent of each other)
constexpr int kStripNT = 32 * kStripWarps;
constexpr int kStripSlots = 4;                   // ring rows: three copies ahead of the sweeps
constexpr int kStripCols = 64;                   // columns a warp loads
static_assert(kPassT % 2 == 0, "pairs keep their alignment");

template <int FORM>
struct Strip {
  static constexpr int T = kPassT;
  static constexpr int H = T;                            // halo columns on each side
  static constexpr int U = kStripCols - 2 * H;           // columns a strip delivers
  static constexpr int XPL = FORM == kSysRecip ? 5 : (FORM == kSysDiv ? 6 : 7);  // the iterate
  static constexpr int PL = XPL + 1;                     // 16-byte words per lane and row
  static constexpr size_t warp_bytes = (size_t)kStripSlots * PL * 32 * 16;
  static constexpr size_t bytes = warp_bytes * kStripWarps;
};

// One row of a lane's pair of cells in registers.
template <int FORM>
struct StripRow {
  double2 S, W, E, N, D;
  double2 B, R;  // DIV, CSR: b and RN(1/D)
};

template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}

// A lane's view of a strip: where its two columns lie and which of them it delivers.
struct StripLane {
  int c0, c1;       // columns (wrapped)
  bool own0, own1;  // delivered, and counted in the residual
  bool wide;        // the pair is one 16-byte word of every array
};

// H halo columns on each side, U = kStripCols - 2 H delivered.
template <int H>
__device__ __forceinline__ StripLane strip_lane(int nx, int pitch, int strip, bool aligned) {
  constexpr int U = kStripCols - 2 * H;
  const int lane = threadIdx.x & 31, i0 = strip * U;
  StripLane L;
  const int q = 2 * lane - H;  // first column of the pair relative to the strip's own
  L.c0 = wrap(i0 + q, nx);
  L.c1 = L.c0 + 1 == nx ? 0 : L.c0 + 1;
  L.own0 = q >= 0 && q < U && i0 + q < nx;
  L.own1 = q >= 0 && q < U && i0 + q + 1 < nx;
  L.wide = aligned && (pitch & 1) == 0 && (L.c0 & 1) == 0 && L.c0 + 1 < nx;
  return L;
}

// (checked build) the pair's columns and row lie in the grid
__device__ __forceinline__ bool pair_in_grid([[maybe_unused]] const StripLane& L,
                                             [[maybe_unused]] int gj, [[maybe_unused]] int nx,
                                             [[maybe_unused]] int ny, [[maybe_unused]] int site) {
  return SWM_IN_RANGE(L.c0, nx, site) && SWM_IN_RANGE(L.c1, nx, site) && SWM_IN_RANGE(gj, ny, site);
}

__device__ __forceinline__ double2 ldcg2(const double* p) {
  return __ldcg(reinterpret_cast<const double2*>(p));
}
// A lane's pair of one row (iterates are written by other blocks: L2 loads).
__device__ __forceinline__ double2 pair_load(const double* row, const StripLane& L) {
  if (L.wide) return ldcg2(row + L.c0);
  return make_double2(__ldcg(row + L.c0), __ldcg(row + L.c1));
}
__device__ __forceinline__ void pair_store(double* row, const StripLane& L, double2 v) {
  if (L.wide && L.own0) {  // wide: c1 = c0 + 1 < nx, so both are delivered
    *reinterpret_cast<double2*>(row + L.c0) = v;
  } else {
    if (L.own0) row[L.c0] = v.x;
    if (L.own1) row[L.c1] = v.y;
  }
}

// Copy of row gj of the system and of the iterate into ring words dst[0 .. PL) (stride 32
// words: one per lane).
template <int FORM, typename Sys>
__device__ __forceinline__ void strip_copy(const Sys& y, const double* xin, int nx, int ny,
                                           int pitch, int gj, const StripLane& L, double2* dst) {
  using G = Strip<FORM>;
  const size_t row = (size_t)gj * pitch;
  const size_t k0 = row + L.c0, k1 = row + L.c1;
  if (!pair_in_grid(L, gj, nx, ny, kChkJacStrip)) return;
  auto plane = [&](int w, const double* p) {
    if (L.wide) {
      cp_async16(dst + 32 * w, p + k0);
    } else {
      cp_async8(dst + 32 * w, p + k0);
      cp_async8(reinterpret_cast<double*>(dst + 32 * w) + 1, p + k1);
    }
  };
  if constexpr (FORM == kSysCsr) {
    // the pair's two CSR rows, 10 values: words 0..4 hold them back to back
    if (L.wide) {
#pragma unroll
      for (int w = 0; w < 5; ++w) cp_async16(dst + 32 * w, y.mass + 5 * k0 + 2 * w);
    } else {
#pragma unroll
      for (int w = 0; w < 10; ++w)
        cp_async8(reinterpret_cast<double*>(dst + 32 * (w / 2)) + (w & 1),
                  y.mass + (w < 5 ? 5 * k0 + w : 5 * k1 + w - 5));
    }
    plane(5, y.diag);
    plane(6, y.b);
  } else {
    plane(0, y.cS);
    plane(1, y.cW);
    plane(2, y.cE);
    plane(3, y.cN);
    plane(4, y.cD);
    if constexpr (FORM == kSysDiv) plane(5, y.b);
  }
  plane(G::XPL, xin);
}

// div_rn's fast path needs |x| in [2^-400, 2^400) (mk_range): the biased exponent field
// of the high word, one subtraction and one unsigned compare.  A zero numerator +0 is
// right too: div_mk gives the correctly signed zero.
__device__ __forceinline__ bool strip_range(double x) {
  return ((unsigned)__double2hiint(x) & 0x7fffffffu) - (623u << 20) < (800u << 20);
}
__device__ __forceinline__ bool strip_num(double x) {
  return strip_range(x) || (__double2hiint(x) | __double2loint(x)) == 0;
}
// RN(1/D) of a row: strips form one per step, without a branch; tiles once per load, by
// __drcp_rn, whose branches keep the registers of a thread's rows from all being live.
// (SAFE passes divide by D.)
template <int FORM, bool TILE, bool SAFE>
__device__ __forceinline__ void strip_rcp(StripRow<FORM>& r, bool& bad) {
  if constexpr (FORM != kSysRecip && !SAFE) {
    bad |= !strip_range(r.D.x) || !strip_range(r.D.y);
    if constexpr (TILE) {
      r.R = make_double2(__drcp_rn(r.D.x), __drcp_rn(r.D.y));
    } else {
      r.R = make_double2(rcp_mk(r.D.x), rcp_mk(r.D.y));
      bad |= !mk_plain(r.D.x) || !mk_plain(r.D.y);
    }
  }
}

// The pair's cells: x = (b - (((S x_S + W x_W) + E x_E) + N x_N)) / D, every product and
// sum rounded, in the reference's CSR order (the zero centre slot adds an exact zero);
// RECIP: b/D - sum of the divided row.  part: the S, W and E products; full: the rest.
// The quotient is formed by div_mk from RN(1/D), the correctly rounded one for operands
// in strip_range; SAFE: by the IEEE division, for any operands.
template <int FORM>
__device__ __forceinline__ double2 pair_part(const StripRow<FORM>& c, double2 south, double2 mid,
                                             double west, double east) {
  double2 p;
  p.x = __dadd_rn(__dmul_rn(c.S.x, south.x), __dmul_rn(c.W.x, west));
  p.y = __dadd_rn(__dmul_rn(c.S.y, south.y), __dmul_rn(c.W.y, mid.x));
  p.x = __dadd_rn(p.x, __dmul_rn(c.E.x, mid.y));
  p.y = __dadd_rn(p.y, __dmul_rn(c.E.y, east));
  return p;
}
template <int FORM, bool SAFE>
__device__ __forceinline__ double2 pair_full(const StripRow<FORM>& c, double2 part, double2 north,
                                             bool& bad) {
  const double px = __dadd_rn(part.x, __dmul_rn(c.N.x, north.x));
  const double py = __dadd_rn(part.y, __dmul_rn(c.N.y, north.y));
  if constexpr (FORM == kSysRecip) {
    return make_double2(__dsub_rn(c.D.x, px), __dsub_rn(c.D.y, py));
  } else {
    const double ax = __dsub_rn(c.B.x, px), ay = __dsub_rn(c.B.y, py);
    if constexpr (SAFE) return make_double2(__ddiv_rn(ax, c.D.x), __ddiv_rn(ay, c.D.y));
    bad |= !strip_num(ax) || !strip_num(ay);
    return make_double2(div_mk(ax, c.D.x, c.R.x), div_mk(ay, c.D.y, c.R.y));
  }
}

// A chunk or tile with an operand outside those ranges adds this to its first residual
// sum: the pass is redone, and the solve goes on, with SAFE passes.  So does one with a
// non-zero CSR centre slot, whose product all passes leave out as the exact zero it is in a
// Patankar system; a SAFE pass that reports it leaves the solve to solve_exact.
constexpr double kBadSum = 0x1p1000;

// bad: an operand the pass does not take.
template <int FORM, bool SAFE>
__device__ __forceinline__ StripRow<FORM> strip_row(const double2* w, bool& bad) {
  StripRow<FORM> r;
  if constexpr (FORM == kSysCsr) {
    const double2 a = w[0], b = w[32], c = w[64], d = w[96], e = w[128];
    r.S = make_double2(a.x, c.y);
    r.W = make_double2(a.y, d.x);
    bad |= b.x != 0. || d.y != 0.;
    r.E = make_double2(b.y, e.x);
    r.N = make_double2(c.x, e.y);
    r.D = w[160];
    r.B = w[192];
  } else {
    r.S = w[0];
    r.W = w[32];
    r.E = w[64];
    r.N = w[96];
    r.D = w[128];
    if constexpr (FORM == kSysDiv) r.B = w[160];
  }
  strip_rcp<FORM, false, SAFE>(r, bad);
  return r;
}

// Up to NL sweeps (Tp of them delivered) of the system over one chunk: rows
// [j0, j0 + rows) of a strip, from xin into xout.  sum[t] += the lane's |x^t - x^{t-1}|
// over the cells it delivers (t >= 1), sum[0] += |b| (first pass only: the initial
// residual, jacobi_iteration.f90:69).
//
// Of a step only the N product depends on the sweep before, so the other products of all
// NL sweeps are formed first: few dependent operations per sweep are left in series.
// Steps before a sweep's first row compute on the zeros and unit rows set below and
// deliver nothing.
template <int FORM, int NL, bool SAFE, typename Sys>
__device__ __forceinline__ void strip_chunk(const Sys& y, const double* xin, double* xout,
                                            int nx, int ny, int pitch, int opitch, int Tp,
                                            bool first, int strip, int j0, int rows, bool aligned,
                                            double2* ring, double (&sum)[kPassT + 1]) {
  using G = Strip<FORM>;
  constexpr int NS = kStripSlots;
  static_assert(NL % 2 == 0 && NL <= G::T, "row parities are static");
  const StripLane L = strip_lane<G::H>(nx, pitch, strip, aligned);
  double2* mine = ring + (threadIdx.x & 31);
  constexpr int SLOT = G::PL * 32;
  const int total = rows + 2 * Tp;  // input rows j0 - Tp .. j0 + rows - 1 + Tp
  int gj = wrap(j0 - Tp, ny);       // row of the next copy
#pragma unroll
  for (int q = 0; q < NS - 1; ++q) {
    if (q < total) strip_copy<FORM>(y, xin, nx, ny, pitch, gj, L, mine + q * SLOT);
    cp_async_commit();
    gj = gj + 1 == ny ? 0 : gj + 1;
  }
  // a row of the identity in the last slot, which step 0 reads as row -1
#pragma unroll
  for (int w = 0; w < G::PL; ++w)
    mine[(NS - 1) * SLOT + 32 * w] = w >= (FORM == kSysCsr ? 5 : 4) ? make_double2(1., 1.)
                                                                   : make_double2(0., 0.);
  StripRow<FORM> cf[NL];  // row s - t of the system at index (s - t) mod NL
  double2 x[NL][2];       // x^{t}: its last two rows, by row parity
#pragma unroll
  for (int t = 0; t < NL; ++t) {
    x[t][0] = x[t][1] = make_double2(0., 0.);
    cf[t].S = cf[t].W = cf[t].E = cf[t].N = make_double2(0., 0.);
    cf[t].D = cf[t].B = cf[t].R = make_double2(1., 1.);
  }
  bool bad = false;
  int gs = wrap(j0 - 2 * Tp, ny);  // row of x^{Tp} a step delivers
  for (int s0 = 0; s0 < total; s0 += NL) {
#pragma unroll
    for (int u = 0; u < NL; ++u) {
      const int s = s0 + u;
      if (s >= total) break;
      cp_async_wait<NS - 2>();  // row s has arrived
      double2 n = mine[(s & (NS - 1)) * SLOT + 32 * G::XPL];
      double2* prev = mine + ((s - 1) & (NS - 1)) * SLOT;
      cf[(u + NL - 1) % NL] = strip_row<FORM, SAFE>(prev, bad);  // row s - 1 of the system
      // the slot of row s - 1 is free: copy row s + NS - 1 into it
      if (s + NS - 1 < total) strip_copy<FORM>(y, xin, nx, ny, pitch, gj, L, prev);
      cp_async_commit();
      gj = gj + 1 == ny ? 0 : gj + 1;
      if (first && (unsigned)(s - Tp) < (unsigned)rows) {  // x^0 = b
        if (L.own0) sum[0] = __dadd_rn(sum[0], fabs(n.x));
        if (L.own1) sum[0] = __dadd_rn(sum[0], fabs(n.y));
      }
      double2 part[NL];
#pragma unroll
      for (int t = 1; t <= NL; ++t) {
        const double2 o = x[t - 1][(u + 2 * NL - t - 1) & 1];  // row s - t - 1 of x^{t-1}
        const double2 m = x[t - 1][(u + 2 * NL - t) & 1];      // row s - t
        part[t - 1] = pair_part<FORM>(cf[(u + NL - t) % NL], o, m,
                                      __shfl_up_sync(0xffffffffu, m.y, 1),
                                      __shfl_down_sync(0xffffffffu, m.x, 1));
      }
      double2 res = n;
#pragma unroll
      for (int t = 1; t <= NL; ++t) {
        const double2 m = x[t - 1][(u + 2 * NL - t) & 1];
        const double2 v = pair_full<FORM, SAFE>(cf[(u + NL - t) % NL], part[t - 1], n, bad);
        const bool in = (unsigned)(s - t - Tp) < (unsigned)rows;
        if (in && L.own0) sum[t] = __dadd_rn(sum[t], fabs(__dsub_rn(v.x, m.x)));
        if (in && L.own1) sum[t] = __dadd_rn(sum[t], fabs(__dsub_rn(v.y, m.y)));
        x[t - 1][(u + 2 * NL - t - 1) & 1] = n;  // row s - t + 1
        n = v;
        if (t == Tp) res = v;
      }
      if ((unsigned)(s - 2 * Tp) < (unsigned)rows &&  // row s - Tp of x^{Tp}
          pair_in_grid(L, gs, nx, ny, kChkJacStrip))
        pair_store(xout + (size_t)gs * opitch, L, res);
      gs = gs + 1 == ny ? 0 : gs + 1;
    }
  }
  cp_async_wait<0>();
  if (FORM != kSysRecip && bad) sum[1] = kBadSum;
}

// Tp sweeps over one chunk by the code of the next even number of sweeps, the lane's
// sums in sum.
template <int FORM, bool SAFE, typename Sys>
__device__ __forceinline__ void strip_pass(const Sys& y, const double* xin, double* xout,
                                           int nx, int ny, int pitch, int opitch, int Tp,
                                           bool first, int strip, int j0, int rows, bool aligned,
                                           double2* ring, double (&sum)[kPassT + 1]) {
  static_assert(kPassT == 4, "the pass lengths below");
#pragma unroll
  for (int t = 0; t <= kPassT; ++t) sum[t] = 0.;
  if (Tp <= 2 && !SAFE)
    strip_chunk<FORM, 2, SAFE>(y, xin, xout, nx, ny, pitch, opitch, Tp, first, strip, j0, rows,
                               aligned, ring, sum);
  else
    strip_chunk<FORM, 4, SAFE>(y, xin, xout, nx, ny, pitch, opitch, Tp, first, strip, j0, rows,
                               aligned, ring, sum);
}
// SAFE out of line, for a loop that also holds the other: its registers must not come out
// of that one's.
template <int FORM, typename Sys>
__device__ __noinline__ void strip_pass_safe(const Sys& y, const double* xin, double* xout,
                                             int nx, int ny, int pitch, int opitch, int Tp,
                                             bool first, int strip, int j0, int rows, bool aligned,
                                             double2* ring, double (&sum)[kPassT + 1]) {
  strip_pass<FORM, true>(y, xin, xout, nx, ny, pitch, opitch, Tp, first, strip, j0, rows, aligned,
                         ring, sum);
}

// ---------------------------------------------------------------------------
// Tiles: kTileWarps warps of RW rows each, T of the tile's rows and columns halo on each
// side for passes of at most T sweeps.  RW is what a thread's registers hold at one block
// of kTileNT threads per SM.
// ---------------------------------------------------------------------------
constexpr int kTileWarps = 12, kTileNT = 32 * kTileWarps;

template <int FORM, int T>
struct Tile {
  static constexpr int RW = FORM == kSysRecip ? 5 : 4;
  static constexpr int ROWS = kTileWarps * RW;
  static constexpr int UX = kStripCols - 2 * T, UY = ROWS - 2 * T;  // delivered
  // edge rows of x, by sweep parity: [2][warp][top, bottom][lane]
  static constexpr size_t bytes = sizeof(double2) * 2 * kTileWarps * 2 * 32;
};

// The rows of the system a thread holds (pair of columns L.c0, L.c1; rows gj, gj + 1, ..).
template <int FORM, bool SAFE, int RW>
__device__ __forceinline__ void tile_rows(const JacobiSys& y, int nx, int ny, int pitch, int gj,
                                          const StripLane& L, StripRow<FORM> (&cf)[RW], bool& bad) {
#pragma unroll
  for (int r = 0; r < RW; ++r) {
    const size_t row = (size_t)gj * pitch;
    const bool in = pair_in_grid(L, gj, nx, ny, kChkJacTile);
    gj = gj + 1 == ny ? 0 : gj + 1;
    if (!in) {
      cf[r] = StripRow<FORM>{};
      continue;
    }
    if constexpr (FORM == kSysCsr) {
      const double *m0 = y.mass + 5 * (row + L.c0), *m1 = y.mass + 5 * (row + L.c1);
      if (L.wide) {
        const double2 a = ldcg2(m0), b = ldcg2(m0 + 2), c = ldcg2(m0 + 4), d = ldcg2(m0 + 6),
                      e = ldcg2(m0 + 8);
        cf[r].S = make_double2(a.x, c.y);
        cf[r].W = make_double2(a.y, d.x);
        bad |= b.x != 0. || d.y != 0.;
        cf[r].E = make_double2(b.y, e.x);
        cf[r].N = make_double2(c.x, e.y);
      } else {
        cf[r].S = make_double2(__ldcg(m0), __ldcg(m1));
        cf[r].W = make_double2(__ldcg(m0 + 1), __ldcg(m1 + 1));
        bad |= __ldcg(m0 + 2) != 0. || __ldcg(m1 + 2) != 0.;
        cf[r].E = make_double2(__ldcg(m0 + 3), __ldcg(m1 + 3));
        cf[r].N = make_double2(__ldcg(m0 + 4), __ldcg(m1 + 4));
      }
      cf[r].D = pair_load(y.diag + row, L);
    } else {
      cf[r].S = pair_load(y.cS + row, L);
      cf[r].W = pair_load(y.cW + row, L);
      cf[r].E = pair_load(y.cE + row, L);
      cf[r].N = pair_load(y.cN + row, L);
      cf[r].D = pair_load(y.cD + row, L);
    }
    if constexpr (FORM != kSysRecip) cf[r].B = pair_load(y.b + row, L);
  }
#pragma unroll
  for (int r = 0; r < RW; ++r) strip_rcp<FORM, true, SAFE>(cf[r], bad);
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Tp <= T sweeps over the tile at (i0, j0) whose rows of the system are in cf; the warp's
// residual sums are added to sum[0..T] (shared memory) as strip_chunk's.  Every thread of
// the block takes part.
template <int FORM, int T, bool SAFE>
__device__ __forceinline__ void tile_pass(const double* xin, double* xout, int nx, int ny,
                                          int pitch, int Tp, bool first, int j0,
                                          const StripLane& L,
                                          const StripRow<FORM> (&cf)[Tile<FORM, T>::RW], bool bad,
                                          double2* edge, double* sum) {
  constexpr int RW = Tile<FORM, T>::RW;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r0 = warp * RW - T;  // this warp's first row relative to the tile's own
  const int g0 = wrap(j0 + r0, ny);
  double2 x[RW];
  int gj = g0;
#pragma unroll
  for (int r = 0; r < RW; ++r) {
    x[r] = pair_in_grid(L, gj, nx, ny, kChkJacTile) ? pair_load(xin + (size_t)gj * pitch, L)
                                                    : make_double2(0., 0.);
    gj = gj + 1 == ny ? 0 : gj + 1;
  }
  // rows this tile delivers, and counts
  const unsigned rows = min(Tile<FORM, T>::UY, ny - j0);
  auto put = [&](int t, double s) {
    s = warp_sum(s);
    if (lane == 0) sum[t] += s;
  };
  if (first) {
    double s = 0.;
#pragma unroll
    for (int r = 0; r < RW; ++r) {
      const bool in = (unsigned)(r0 + r) < rows;
      if (in && L.own0) s = __dadd_rn(s, fabs(x[r].x));
      if (in && L.own1) s = __dadd_rn(s, fabs(x[r].y));
    }
    put(0, s);
  }
  for (int t = 1; t <= Tp; ++t) {
    double2* e = edge + (t & 1) * (kTileWarps * 64);
    e[warp * 64 + lane] = x[0];
    e[warp * 64 + 32 + lane] = x[RW - 1];
    __syncthreads();
    // the rows above and below (the tile's outermost rows have none; their results are
    // in the halo and not used)
    const double2 lo = e[(warp == 0 ? 0 : warp - 1) * 64 + 32 + lane];
    const double2 hi = e[(warp == kTileWarps - 1 ? warp : warp + 1) * 64 + lane];
    double2 south = lo;
    double s = 0.;
#pragma unroll
    for (int r = 0; r < RW; ++r) {
      const double2 m = x[r];
      const double2 part = pair_part<FORM>(cf[r], south, m, __shfl_up_sync(0xffffffffu, m.y, 1),
                                           __shfl_down_sync(0xffffffffu, m.x, 1));
      const double2 v = pair_full<FORM, SAFE>(cf[r], part, r + 1 < RW ? x[r + 1 < RW ? r + 1 : r] : hi, bad);
      const bool in = (unsigned)(r0 + r) < rows;
      if (in && L.own0) s = __dadd_rn(s, fabs(__dsub_rn(v.x, m.x)));
      if (in && L.own1) s = __dadd_rn(s, fabs(__dsub_rn(v.y, m.y)));
      south = m;
      x[r] = v;
    }
    put(t, s);
  }
  gj = g0;
#pragma unroll
  for (int r = 0; r < RW; ++r) {
    if ((unsigned)(r0 + r) < rows && pair_in_grid(L, gj, nx, ny, kChkJacTile))
      pair_store(xout + (size_t)gj * pitch, L, x[r]);
    gj = gj + 1 == ny ? 0 : gj + 1;
  }
  if constexpr (FORM != kSysRecip) {
    if (__any_sync(0xffffffffu, bad) && lane == 0) sum[1] = kBadSum;
  }
}

}  // namespace swm
