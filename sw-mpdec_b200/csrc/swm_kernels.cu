// swm_kernels.cu -- memory-bound kernels of the mPDeC5 step (sm_100a).
// Built with -fmad=false: every FP64 expression here rounds exactly as the
// reference's source order does (no contraction), which makes the Patankar
// matrix and the Jacobi iterates bit-identical to the CPU restatement given the
// same fluxes, and the CSR and matrix-free solvers bit-identical to each other.
#include <cooperative_groups.h>

#include <cstdio>
#include <cstring>

#include "../../include/swm.h"
#include "swm_kernels.cuh"
#include "swm_solve.cuh"
#include "swm_strip.cuh"

namespace swm {

SWM_CHECK_READER(check_record_kernels)

void residual_limbs_host(double v, unsigned long long out[3]) {
  unsigned long long a, b, c;
  residual_limbs(v, a, b, c);
  out[0] = a;
  out[1] = b;
  out[2] = c;
}

// ---------------------------------------------------------------------------
// TimeStep (equation.f90:791-837): LambdaMaxX/Y = max |u + sqrt(g h)|, |v + sqrt(g h)|
// ---------------------------------------------------------------------------
// Load latency bounds it: four cells' loads in flight per thread, and one pair of atomics
// per block (they all go to the same two words): 2048^2 42 -> 29 us, 512 x 256 8.5 -> 4.8 us.
constexpr int kDtNT = 256, kDtCells = 4;
__global__ void __launch_bounds__(kDtNT) dt_kernel(const DtArgs a) {
  const int n = a.nx * a.ny, stride = gridDim.x * kDtNT;
  double lx = 0.0, ly = 0.0;
  int bad = 0;
  for (int k0 = blockIdx.x * kDtNT + threadIdx.x; k0 < n; k0 += kDtCells * stride) {
    double h[kDtCells], hu[kDtCells], hv[kDtCells];
#pragma unroll
    for (int q = 0; q < kDtCells; ++q) {
      const int k = k0 + q * stride;  // n <= 2^28: no overflow
      const bool in = k < n;
      h[q] = in ? a.h[k] : 0.0;
      hu[q] = in ? a.hu[k] : 0.0;
      hv[q] = in ? a.hv[k] : 0.0;
    }
#pragma unroll
    for (int q = 0; q < kDtCells; ++q) {
      if (k0 + q * stride >= n) break;
      double u, v;
      if (!(h[q] >= 0.0) || !isfinite(h[q]) || !isfinite(hu[q]) || !isfinite(hv[q])) bad = 1;
      cons_to_prim<true>(h[q], hu[q], hv[q], u, v);
      const double c = sqrt(a.g * h[q]);
      lx = dmax(lx, fabs(u + c));
      ly = dmax(ly, fabs(v + c));
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lx = dmax(lx, __shfl_down_sync(0xffffffffu, lx, o));
    ly = dmax(ly, __shfl_down_sync(0xffffffffu, ly, o));
  }
  __shared__ double s_lx[kDtNT / 32], s_ly[kDtNT / 32];
  if ((threadIdx.x & 31) == 0) {
    s_lx[threadIdx.x >> 5] = lx;
    s_ly[threadIdx.x >> 5] = ly;
  }
  bad = __syncthreads_or(bad);
  if (threadIdx.x == 0) {
    for (int w = 1; w < kDtNT / 32; ++w) {
      lx = dmax(lx, s_lx[w]);
      ly = dmax(ly, s_ly[w]);
    }
    // non-negative doubles order like their bit patterns
    atomicMax(&a.lam[0], (unsigned long long)__double_as_longlong(lx));
    atomicMax(&a.lam[1], (unsigned long long)__double_as_longlong(ly));
    if (bad) atomicOr(a.bad, 1);
  }
}

cudaError_t launch_dt(const DtArgs& a, cudaStream_t s) {
  int n = a.nx * a.ny;
  int blocks = (n + kDtNT - 1) / kDtNT;
  if (blocks > 148 * 8) blocks = 148 * 8;
  dt_kernel<<<blocks, kDtNT, 0, s>>>(a);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Layout conversion between the reference's ghosted array U(1:3,-2:nx+3,-2:ny+3)
// and the device planes [ny][nx].
// ---------------------------------------------------------------------------
__global__ void ghosted_to_planes_kernel(const double* __restrict__ G, int nx, int ny, double* h,
                                         double* hu, double* hv) {
  int n = nx * ny;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    int i = k % nx, j = k / nx;
    size_t g = 3 * ((size_t)(i + 3) + (size_t)(nx + 6) * (j + 3));
    h[k] = G[g];
    hu[k] = G[g + 1];
    hv[k] = G[g + 2];
  }
}

// Ghost frame filled periodically (the values BoundaryConditions would write,
// equation.f90:556-776); Vg (nullable) = ConsToPrim on the whole array.
__global__ void planes_to_ghosted_kernel(const double* h, const double* hu, const double* hv,
                                         int nx, int ny, double* G, double* Vg) {
  int W = nx + 6, n = W * (ny + 6);
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    int gi = k % W - 3, gj = k / W - 3;
    int i = wrap(gi, nx), j = wrap(gj, ny);
    size_t s = (size_t)j * nx + i;
    double a = h[s], b = hu[s], c = hv[s];
    G[3 * (size_t)k] = a;
    G[3 * (size_t)k + 1] = b;
    G[3 * (size_t)k + 2] = c;
    if (Vg) {
      double u, v;
      cons_to_prim<true>(a, b, c, u, v);
      Vg[3 * (size_t)k] = a;
      Vg[3 * (size_t)k + 1] = u;
      Vg[3 * (size_t)k + 2] = v;
    }
  }
}

cudaError_t launch_ghosted_to_planes(const double* G, int nx, int ny, double* h, double* hu,
                                     double* hv, cudaStream_t s) {
  int n = nx * ny, blocks = (n + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  ghosted_to_planes_kernel<<<blocks, 256, 0, s>>>(G, nx, ny, h, hu, hv);
  return cudaGetLastError();
}

cudaError_t launch_planes_to_ghosted(const double* h, const double* hu, const double* hv, int nx,
                                     int ny, double* G, double* Vg, cudaStream_t s) {
  int n = (nx + 6) * (ny + 6), blocks = (n + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  planes_to_ghosted_kernel<<<blocks, 256, 0, s>>>(h, hu, hv, nx, ny, G, Vg);
  return cudaGetLastError();
}

// mass = sum h (per-block partials in fixed order, then one block), min h.
__global__ void summary_kernel(const double* h, int n, double* part_sum, double* part_min) {
  __shared__ double ss[256], sm[256];
  double s = 0.0, m = 1e300;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    s += h[k];
    m = dmin(m, h[k]);
  }
  ss[threadIdx.x] = s;
  sm[threadIdx.x] = m;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) {
      ss[threadIdx.x] += ss[threadIdx.x + o];
      sm[threadIdx.x] = dmin(sm[threadIdx.x], sm[threadIdx.x + o]);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    part_sum[blockIdx.x] = ss[0];
    part_min[blockIdx.x] = sm[0];
  }
}
__global__ void summary_final_kernel(const double* ps, const double* pm, int nb, double* out) {
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    double s = 0.0, m = 1e300;
    for (int b = 0; b < nb; ++b) {
      s += ps[b];
      m = dmin(m, pm[b]);
    }
    out[0] = s;
    out[1] = m;
  }
}
cudaError_t launch_summary(const double* h, int n, double* out, cudaStream_t s) {
  // out must have room for 2 + 2*256 doubles (partials after the result)
  const int nb = 256;
  summary_kernel<<<nb, 256, 0, s>>>(h, n, out + 2, out + 2 + nb);
  summary_final_kernel<<<1, 32, 0, s>>>(out + 2, out + 2 + nb, nb, out);
  return cudaGetLastError();
}

// The three substeps of one mPDeC5 correction iteration in one pass (split and FMA
// forms, stencil layout): the stage RHS planes, face fluxes and U^n momentum are
// read once for all of them; hp(m) and the outputs are per substep.  Every load is
// issued before the arithmetic.  Each substep's arithmetic is that of
// assemble_kernel<true, 4>, so the results are identical.
__global__ void __launch_bounds__(128, 4) assemble_multi_kernel(const AssembleMultiArgs a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y;
  if (i >= a.base.nx || j >= a.base.ny) return;
  assemble_multi_cell(a, i, j);
}

// The same for the exact forms (FP64; any form with the CSR solver).
__global__ void __launch_bounds__(128, 4)
    assemble_multi_exact_kernel(const __grid_constant__ AssembleMultiArgs a, bool csr) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y;
  if (i >= a.base.nx || j >= a.base.ny) return;
  assemble_multi_exact_cell(a, csr, i, j);
}

cudaError_t launch_assemble_multi(const AssembleMultiArgs& a, bool csr, cudaStream_t s) {
  if (a.nm != kMaxFusedStages || a.base.msteps != 4) return cudaErrorInvalidValue;
  dim3 blk(128), grd((a.base.nx + 127) / 128, a.base.ny);
  if (a.base.fast && !csr)
    assemble_multi_kernel<<<grd, blk, 0, s>>>(a);
  else
    assemble_multi_exact_kernel<<<grd, blk, 0, s>>>(a, csr);
  return cudaGetLastError();
}

template <bool FAST, int MS>
__global__ void __launch_bounds__(128) assemble_kernel(const __grid_constant__ AssembleArgs a,
                                                       bool csr) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y;
  if (i >= a.nx || j >= a.ny) return;
  assemble_cell<FAST, MS>(a, csr, i, j);
}

// Ensembles: block b covers cells [cell0, cell0+128) of problem blk[b].x, with
// cell0 = blk[b].y; descriptors staged in shared memory (stencil layout only).
template <bool FAST>
__global__ void __launch_bounds__(128)
    assemble_batch_kernel(const AssembleArgs* __restrict__ descs, const int2* __restrict__ blk) {
  static_assert(sizeof(AssembleArgs) % 8 == 0 && sizeof(AssembleArgs) / 8 <= 128, "copy");
  __shared__ __align__(16) AssembleArgs sa;
  const int2 w = blk[blockIdx.x];
  if (threadIdx.x < sizeof(AssembleArgs) / 8)
    reinterpret_cast<unsigned long long*>(&sa)[threadIdx.x] =
        reinterpret_cast<const unsigned long long*>(&descs[w.x])[threadIdx.x];
  __syncthreads();
  const int c = w.y + threadIdx.x;
  if (c >= sa.nx * sa.ny) return;
  if (sa.msteps == 4)
    assemble_cell<FAST, 4>(sa, false, c % sa.nx, c / sa.nx);
  else
    assemble_cell<FAST, 2>(sa, false, c % sa.nx, c / sa.nx);
}

// Ensembles, fast forms: the fused assembly of a correction's three substeps; block b
// covers 128 cells of problem blk[b].x from blk[b].y (descriptor staged in shared memory).
__global__ void __launch_bounds__(128, 4)
    assemble_multi_batch_kernel(const AssembleMultiArgs* __restrict__ descs,
                                const int2* __restrict__ blk) {
  static_assert(sizeof(AssembleMultiArgs) % 8 == 0, "copy");
  __shared__ __align__(16) AssembleMultiArgs sa;
  const int2 w = blk[blockIdx.x];
  for (int q = threadIdx.x; q < (int)(sizeof(AssembleMultiArgs) / 8); q += blockDim.x)
    reinterpret_cast<unsigned long long*>(&sa)[q] =
        reinterpret_cast<const unsigned long long*>(&descs[w.x])[q];
  __syncthreads();
  const int c = w.y + threadIdx.x;
  if (c < sa.base.nx * sa.base.ny) assemble_multi_cell(sa, c % sa.base.nx, c / sa.base.nx);
}

cudaError_t launch_assemble_multi_batch(const AssembleMultiArgs* descs, const int2* blk, int nblk,
                                        cudaStream_t s) {
  if (nblk < 1) return cudaSuccess;
  assemble_multi_batch_kernel<<<nblk, 128, 0, s>>>(descs, blk);
  return cudaGetLastError();
}

cudaError_t launch_assemble_batch(const AssembleArgs* descs, const int2* blk, int nblk, bool fast,
                                  cudaStream_t s) {
  if (nblk < 1) return cudaSuccess;
  if (fast)
    assemble_batch_kernel<true><<<nblk, 128, 0, s>>>(descs, blk);
  else
    assemble_batch_kernel<false><<<nblk, 128, 0, s>>>(descs, blk);
  return cudaGetLastError();
}

cudaError_t launch_assemble(const AssembleArgs& a, bool csr, cudaStream_t s) {
  dim3 blk(128), grd((a.nx + 127) / 128, a.ny);
  const bool fast = a.fast && !csr;
  if (a.msteps == 4) {
    if (fast)
      assemble_kernel<true, 4><<<grd, blk, 0, s>>>(a, csr);
    else
      assemble_kernel<false, 4><<<grd, blk, 0, s>>>(a, csr);
  } else {
    if (fast)
      assemble_kernel<true, 2><<<grd, blk, 0, s>>>(a, csr);
    else
      assemble_kernel<false, 2><<<grd, blk, 0, s>>>(a, csr);
  }
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Explicit schemes (timediscretization.f90:104-451): stage combinations.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) combo_kernel(const ComboArgs a) {
  const double dt = *a.dt;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < a.n; k += gridDim.x * blockDim.x) {
#pragma unroll
    for (int v = 0; v < 3; ++v) {
      double acc;
      if (a.form == kComboSsp) {
        acc = a.c[0] * a.X[0][v][k];
        for (int i = 1; i < a.nx; ++i) acc = acc + a.c[i] * a.X[i][v][k];
        for (int j = 0; j < a.ny; ++j) acc = acc + a.d[j] * a.Y[j][v][k] * dt;
      } else if (a.form == kComboRk) {
        double sum = a.d[0] * a.Y[0][v][k];
        for (int j = 1; j < a.ny; ++j) sum = sum + a.d[j] * a.Y[j][v][k];
        acc = a.X[0][v][k] + sum * dt;
      } else {
        acc = a.X[0][v][k];
        for (int j = 0; j < a.ny; ++j) acc = acc + dt * a.d[j] * a.Y[j][v][k];
      }
      a.out[v][k] = acc;
    }
  }
}

cudaError_t launch_combo(const ComboArgs& a, cudaStream_t s) {
  int blocks = (a.n + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  combo_kernel<<<blocks, 256, 0, s>>>(a);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Jacobi on the systems of one grid: one cooperative launch, passes of up to T sweeps
// (strip_chunk) separated by a bounded grid barrier; every CTA takes the same decisions
// from the same sums.
//
// Stop rule: mean|x^{k+1} - x^k| <= tol after every sweep (jacobi_iteration.f90:71-81)
// on the exact sum of |dx| rounded to multiples of 2^-100.  A pass sums |dx| in FP64, in
// any order: n terms, so within n 2^-53 < 2^-24 of the sum of the unrounded terms, and
// those are within n 2^-101 of the rounded ones.  Outside kBand of the threshold the
// order therefore cannot change the decision (stop_decision); a sum inside the band (about one solve in
// 10^5, or tol = 0) hands the system to solve_exact, which goes on from the pass's input
// one sweep at a time with exact integer sums.  The iterates and the stop index depend
// on neither tiling, launch shape nor atomic order.
// ---------------------------------------------------------------------------
// Grid barrier number `nth` (1, 2, ..) of a launch on its own arrival counter (zero when
// the launch starts), by one thread: everything its block wrote before a block barrier is
// visible to every block after it (the arrival releases, the poll acquires; both are
// ordered with the block's other threads by the block barriers around this).  The count
// only grows, modulo 2^32 (barrier_open), so an arrival is one atomic and a wait one
// polled word.  False when the wait gave up (status -4).
__device__ __forceinline__ bool arrive_and_wait(unsigned int* ctr, unsigned int nth,
                                                long long spin_limit, int* status) {
  const unsigned int target = nth * gridDim.x;
  unsigned int c;
  asm volatile("atom.add.acq_rel.gpu.u32 %0, [%1], 1;" : "=r"(c) : "l"(ctr) : "memory");
  bool ok = true;
  if (c + 1 != target) {
    long long spins = 0;
    for (;;) {
      asm volatile("ld.acquire.gpu.u32 %0, [%1];" : "=r"(c) : "l"(ctr) : "memory");
      if (barrier_open(c, target)) break;
      if (++spins > spin_limit || spin_limit <= 0) {
        ok = false;
        atomicExch(status, -4);
        break;
      }
    }
  }
  return ok;
}

// Sweeps of a pass when `left` more are expected: as few passes as blk allows, evenly.
__device__ __forceinline__ int even_pass(int left, int blk) {
  const int np = (left + blk - 1) / blk;
  return np > 0 ? (left + np - 1) / np : blk;
}

// What a pass's outcome means for a system.  n: its cells; sum: the pass's residual
// sums; hint: sweeps of the same substep's previous solve, or 0; out: the destination, or
// b where a pass must not write it directly.
template <int FORM>
__device__ __forceinline__ void sys_decide(SysState& S, double n, int maxiter, double thresh,
                                           const double* b, double* xa, double* xb, double* out,
                                           const double* sum, int hint, int blk) {
  if (S.rollback) {  // the redone pass delivered the final iterate
    S.active = 0;
    S.xin = S.xout;
    return;
  }
  if (FORM != kSysRecip && !S.safe && !(sum[1] < 0.5 * kBadSum)) {
    S.safe = 1;  // an operand the fast divisions do not take: the same pass again
    return;
  }
  if (FORM == kSysCsr && S.safe && sum[1] >= 0.5 * kBadSum) {
    S.exact = 1;  // a centre slot
    S.active = 0;
    return;
  }
  if (S.first) {
    const int d = stop_decision(sum[0], thresh, n);
    if (d != 0) {
      S.active = 0;
      if (d > 0)
        S.zero = 1;
      else
        S.exact = 1;
      return;
    }
  }
  int stop = 0;
  for (int t = 1; t <= S.Tp && stop == 0; ++t) {
    const int d = stop_decision(sum[t], thresh, n);
    if (d < 0) {
      S.exact = 1;
      S.active = 0;
      return;
    }
    if (d > 0) stop = t;
  }
  S.first = 0;
  if (stop > 0) {
    S.k += stop;
    if (stop < S.Tp) {  // the stop falls inside the pass: redo it with `stop` sweeps
      S.rollback = 1;
      S.Tp = stop;
    } else {
      S.active = 0;
      S.xin = S.xout;
    }
    return;
  }
  S.k += S.Tp;
  if (S.k >= maxiter) {
    S.active = 0;
    S.maxhit = 1;
    S.xin = S.xout;
    return;
  }
  // Sweeps still needed: from the hint while it holds, else from the decay of the last
  // two sweeps.  Only pass lengths depend on it.
  const float rT = (float)sum[S.Tp];
  const float rP = S.Tp >= 2 ? (float)sum[S.Tp - 1] : S.r_prev;
  S.r_prev = rT;
  int left = blk + 1;  // unknown: a full pass
  if (hint > S.k) {
    left = hint - S.k;
  } else if (rP > 0.f && rT > 0.f && rT < rP && thresh > 0.) {
    const float need = __log2f((float)thresh / rT) / __log2f(rT / rP);
    if (need > 0.f && need < 1000.f) left = (int)ceilf(need);
  }
  if (left < 1) left = 1;
  int Tp = left > blk ? blk : left;
  if (hint > S.k) Tp = even_pass(left, blk);
  if (maxiter - S.k < Tp) Tp = maxiter - S.k;
  S.Tp = Tp;
  // the next pass writes the other ping-pong buffer or, when it is expected to be the
  // last, the destination (unless that is the rhs or the pass's input)
  S.xin = S.xout;
  S.xout = (S.xin == xa) ? xb : xa;
  if (left <= Tp && out != b && out != S.xin) S.xout = out;
}


// A system's first pass.
__device__ __forceinline__ SysState sys_start(int maxiter, const double* b, double* xa, double* out,
                                              int hint, int blk) {
  SysState S;
  S.Tp = hint > 0 ? even_pass(hint, blk) : blk;
  if (S.Tp > maxiter) S.Tp = maxiter;
  S.xin = b;
  S.xout = (hint > 0 && hint <= S.Tp && out != b) ? out : xa;
  S.k = 0;
  S.active = 1;
  S.first = 1;
  S.rollback = S.zero = S.maxhit = S.exact = S.safe = 0;
  S.r_prev = -1.f;
  return S;
}

// Work split of a pass over `nact` systems: chunks per strip so that the slowest warp's
// rows (its chunks, each with 2 Tp rows of overlap) are fewest, for one to four chunks a
// warp.  Called by a whole warp.
__device__ __forceinline__ int strip_chunks(int nact, int strips, int ny, int Tp, int warps) {
  const unsigned r = 1 + (threadIdx.x & 3), per = (unsigned)nact * strips;
  const unsigned most = (ny + 3) / 4;
  unsigned ch = r * warps / per;
  ch = ch < 1 ? 1 : (ch > most ? most : ch);
  const unsigned cost = ((per * ch + warps - 1) / warps) * ((ny + ch - 1) / ch + 2 * Tp);
  unsigned best = cost, pick = ch;
#pragma unroll
  for (int o = 1; o < 4; o <<= 1) {
    const unsigned c2 = __shfl_xor_sync(0xffffffffu, best, o);
    const unsigned h2 = __shfl_xor_sync(0xffffffffu, pick, o);
    if (c2 < best || (c2 == best && h2 < pick)) {
      best = c2;
      pick = h2;
    }
  }
  return (int)pick;
}

// What solve_exact needs of a grid and its system's arrays.
struct ExactGrid {
  int nx, ny, pitch, maxiter;
  const unsigned long long* thresh;
  const int* rowstart;  // CSR pattern, 1-based
  const int* cols;
  unsigned long long (*acc)[2][3];  // ring of limb sums, zero between solves' passes
  unsigned int* bar;
  int* status;
  long long spin_limit;
};

// One cell of a system, the CSR rows through the pattern.
template <int FORM, typename Sys>
__device__ __forceinline__ double cell_update(const ExactGrid& g, const Sys& y, const double* xin,
                                              int i, int j) {
  double p = 0.;
  if constexpr (FORM == kSysCsr) {
    [[maybe_unused]] const int n = g.nx * g.ny;  // (the checked build's bound)
    const int row = j * g.nx + i;
    for (int sp = g.rowstart[row]; sp <= g.rowstart[row + 1] - 1; ++sp)
      if (SWM_IN_RANGE(sp - 1, 5LL * n, kChkCsr) && SWM_IN_RANGE(g.cols[sp - 1] - 1, n, kChkCsr))
        p = __dadd_rn(p, __dmul_rn(y.mass[sp - 1], __ldcg(&xin[g.cols[sp - 1] - 1])));
    return __ddiv_rn(__dsub_rn(y.b[row], p), y.diag[row]);
  } else {
    const int im = i == 0 ? g.nx - 1 : i - 1, ip = i == g.nx - 1 ? 0 : i + 1;
    const int jm = j == 0 ? g.ny - 1 : j - 1, jp = j == g.ny - 1 ? 0 : j + 1;
    if (!SWM_IN_RANGE(im, g.nx, kChkJacExact) || !SWM_IN_RANGE(ip, g.nx, kChkJacExact) ||
        !SWM_IN_RANGE(jm, g.ny, kChkJacExact) || !SWM_IN_RANGE(jp, g.ny, kChkJacExact))
      return 0.;
    const size_t r = (size_t)j * g.pitch, c = r + i;
    p = __dmul_rn(y.cS[c], __ldcg(&xin[(size_t)jm * g.pitch + i]));
    p = __dadd_rn(p, __dmul_rn(y.cW[c], __ldcg(&xin[r + im])));
    p = __dadd_rn(p, __dmul_rn(y.cE[c], __ldcg(&xin[r + ip])));
    p = __dadd_rn(p, __dmul_rn(y.cN[c], __ldcg(&xin[(size_t)jp * g.pitch + i])));
    if constexpr (FORM == kSysRecip)
      return __dsub_rn(y.cD[c], p);
    else
      return __ddiv_rn(__dsub_rn(y.b[c], p), y.cD[c]);
  }
}

// The rest of a solve one sweep at a time with IEEE divisions, residuals summed exactly
// in integer limbs; every block of the grid takes part.  pass, nbar: the block's position
// in the ring of limb sums and its count of grid barriers (shared memory).  Returns false
// when a barrier wait gave up.
template <int FORM, typename Sys>
__device__ __noinline__ bool solve_exact(const ExactGrid& g, const Sys& y, SysState& S, int* pass,
                                         unsigned int* nbar) {
  __shared__ unsigned long long s_acc[2][3];
  __shared__ unsigned long long s_tot[2][3];
  __shared__ int s_ok;
  const int n = g.nx * g.ny, stride = gridDim.x * blockDim.x;
  const double* xin = S.xin;
  int k = S.k, stop = -1;
  bool first = S.first != 0;
  for (;;) {
    double* xout = (xin == y.xa) ? y.xb : y.xa;
    if (threadIdx.x < 6) (&s_acc[0][0])[threadIdx.x] = 0ull;
    __syncthreads();
    Acc acc;
    acc_zero(acc);
    int since = 0;
    for (int base = blockIdx.x * blockDim.x; base < n; base += stride) {
      if (++since > kAccFlushCells) {  // block-uniform
        acc_reduce<1>(acc, s_acc);
        since = 1;
      }
      const int cell = base + threadIdx.x;
      if (cell < n) {
        const int i = cell % g.nx, j = cell / g.nx;
        const size_t c = (size_t)j * g.pitch + i;
        const double v = cell_update<FORM>(g, y, xin, i, j);
        xout[c] = v;
        acc_put<1>(acc, fabs(__dsub_rn(v, __ldcg(&xin[c]))));
        if (first) acc_put<0>(acc, fabs(0. - y.b[c]));
      }
    }
    acc_reduce<1>(acc, s_acc);
    __syncthreads();
    const int slot = *pass;
    if (threadIdx.x < 6) {
      const unsigned long long v = (&s_acc[0][0])[threadIdx.x];
      if (v) atomicAdd(&(&g.acc[slot][0][0])[threadIdx.x], v);
    }
    __syncthreads();
    if (threadIdx.x == 0) s_ok = arrive_and_wait(g.bar, ++*nbar, g.spin_limit, g.status);
    __syncthreads();
    if (!s_ok) return false;
    if (threadIdx.x < 6) (&s_tot[0][0])[threadIdx.x] = __ldcg(&(&g.acc[slot][0][0])[threadIdx.x]);
    if (blockIdx.x == 0 && threadIdx.x < 6) {
      (&g.acc[ring_at(slot, 2, kResSlots)][0][0])[threadIdx.x] = 0ull;
      __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) *pass = ring_at(slot, 1, kResSlots);
    if (first && limbs_le(s_tot[0][0], s_tot[0][1], s_tot[0][2], g.thresh)) {
      stop = 0;
      break;
    }
    first = false;
    ++k;
    xin = xout;
    if (limbs_le(s_tot[1][0], s_tot[1][1], s_tot[1][2], g.thresh)) {
      stop = k;
      break;
    }
    if (k >= g.maxiter) break;
    __syncthreads();
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    S.k = stop == 0 ? 0 : k;
    S.xin = xin;
    S.zero = stop == 0;
    S.maxhit = stop < 0;
  }
  __syncthreads();
  return true;
}

// TILES: a block per tile and passes of up to TILES sweeps (small grids); 0: a warp per
// chunk of a strip, passes of up to kPassT.
template <int TILES>
struct PassShared {
  static constexpr int T = TILES ? TILES : kPassT, NW = TILES ? kTileWarps : kStripWarps;
  static_assert(T <= kMaxBlock, "residual sums of a pass");
  SysState st[kMaxSys];
  double sum[NW][kMaxSys][T + 1], tot[kMaxSys][T + 1];
  int ok, slot, xpass, nact, ch, act[kMaxSys], hint[kMaxSys];  // slot, xpass: ring positions
  unsigned int nbar;
};

// Passes over the active systems until none is left, or a barrier wait gave up (sh.ok).
template <int FORM, int TILES, bool SAFE>
__device__ __forceinline__ void solve_passes(const JacobiGroup& a, PassShared<TILES>& sh) {
  extern __shared__ __align__(16) unsigned char jring[];
  using G = Strip<FORM>;
  constexpr int T = PassShared<TILES>::T, NW = PassShared<TILES>::NW;
  using TG = Tile<FORM, T>;
  JacobiCtl* ctl = a.ctl;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int blk = a.block < 1 ? 1 : (a.block > T ? T : a.block);
  const double thresh = limbs_value(a.thresh[0], a.thresh[1], a.thresh[2]);
  const int strips = (a.nx + TG::UX - 1) / TG::UX, warps = gridDim.x * kStripWarps;
  const int tiles = TILES ? strips * ((a.ny + TG::UY - 1) / TG::UY) : 0;
  static_assert(TILES || G::U == TG::UX, "strips deliver as many columns as tiles");
  double2* ring = reinterpret_cast<double2*>(jring + (TILES ? 0 : warp * G::warp_bytes));
  // the systems still iterating and the pass's split, by warp 0
  auto plan = [&]() {
    int na = 0, most = 0;
    for (int q = 0; q < a.nsys; ++q)
      if (sh.st[q].active) {
        if (lane == 0) sh.act[na] = q;
        ++na;
        most = max(most, sh.st[q].Tp);
      }
    const int ch = !TILES && na ? strip_chunks(na, strips, a.ny, most, warps) : 1;
    if (lane == 0) {
      sh.nact = na;
      sh.ch = ch;
    }
  };
  if (warp == 0) plan();
  __syncthreads();
  StripRow<FORM> cf[TILES ? TG::RW : 1];  // tiles: the rows held, of tile `held`
  int held = -1;
  bool held_bad = false;
  while (sh.nact > 0) {
    for (int q = lane; q < kMaxSys * (T + 1); q += 32) (&sh.sum[warp][0][0])[q] = 0.;
    __syncwarp();
    const int nact = sh.nact;
    auto aligned = [&](const JacobiSys& y, const SysState& S) {
      unsigned long long al = (unsigned long long)S.xin | (unsigned long long)S.xout |
                              (unsigned long long)y.b;
      if constexpr (FORM == kSysCsr)
        al |= (unsigned long long)y.mass | (unsigned long long)y.diag;
      else
        al |= (unsigned long long)y.cS | (unsigned long long)y.cW | (unsigned long long)y.cE |
              (unsigned long long)y.cN | (unsigned long long)y.cD;
      return (al & 15ull) == 0;
    };
    if constexpr (TILES) {
      for (int it = blockIdx.x; it < nact * tiles; it += gridDim.x) {
        const int q = sh.act[it / tiles], tile = it % tiles;
        const JacobiSys& y = a.sys[q];
        const SysState& S = sh.st[q];
        const int Tp = S.Tp, strip = tile % strips, j0 = (tile / strips) * TG::UY;
        const StripLane L = strip_lane<T>(a.nx, a.nx, strip, aligned(y, S));
        if (held != q * tiles + tile) {  // a block with one tile keeps its rows of the system
          held = q * tiles + tile;
          held_bad = false;
          tile_rows<FORM, SAFE>(y, a.nx, a.ny, a.nx, wrap(j0 + warp * TG::RW - T, a.ny), L, cf,
                                held_bad);
        }
        tile_pass<FORM, T, SAFE>(S.xin, S.xout, a.nx, a.ny, a.nx, Tp, S.first != 0, j0, L, cf,
                                 held_bad, ring, sh.sum[warp][q]);
        __syncthreads();  // the edge rows are read
      }
    } else {
      const int ch = sh.ch, R = (a.ny + ch - 1) / ch, items = nact * strips * ch;
      // items in (system, chunk, strip) order over all CTAs first, so that few items
      // spread over many SMs and neighbouring strips stream together
      for (int it = warp * gridDim.x + blockIdx.x; it < items; it += warps) {
        const int strip = it % strips, rest = it / strips;
        const int q = sh.act[rest / ch], j0 = (rest % ch) * R, rows = min(R, a.ny - j0);
        if (rows <= 0) continue;
        const JacobiSys& y = a.sys[q];
        const SysState& S = sh.st[q];
        const int Tp = S.Tp;
        double sum[T + 1];
        strip_pass<FORM, SAFE>(y, S.xin, S.xout, a.nx, a.ny, a.nx, a.nx, Tp, S.first != 0, strip,
                               j0, rows, aligned(y, S), ring, sum);
#pragma unroll
        for (int t = 0; t <= T; ++t) {
          if (t > Tp) break;
          const double v = warp_sum(sum[t]);
          if (lane == 0) sh.sum[warp][q][t] += v;
        }
      }
    }
    __syncthreads();
    if (warp == 0) {
      // the block's sums, the grid barrier, then every block's decisions from the totals
      static_assert(kMaxSys * (T + 1) <= 32, "a lane per sum");
      const int slot = sh.slot, q = lane / (T + 1), t = lane % (T + 1);
      const bool mine = q < a.nsys && sh.st[q < kMaxSys ? q : 0].active;
      if (mine) {
        double v = sh.sum[0][q][t];
        for (int w = 1; w < NW; ++w) v += sh.sum[w][q][t];
        if (v != 0.) atomicAdd(&ctl->sum[slot][q][t], v);
      }
      __syncwarp();
      if (lane == 0)
        sh.ok = arrive_and_wait(&ctl->bar[a.sys[0].solve_idx], ++sh.nbar, a.spin_limit,
                                &ctl->status);
      __syncwarp();
      if (sh.ok) {
        if (mine) sh.tot[q][t] = __ldcg(&ctl->sum[slot][q][t]);
        if (blockIdx.x == 0) {  // recycle the slot of the pass before this one
          for (int z = lane; z < kMaxSys * (kMaxBlock + 1); z += 32)
            (&ctl->sum[ring_at(slot, 2, kResSlots)][0][0])[z] = 0.;
          __threadfence();
        }
        __syncwarp();
        if (lane < a.nsys && sh.st[lane].active) {
          const JacobiSys& y = a.sys[lane];
          sys_decide<FORM>(sh.st[lane], (double)a.nx * a.ny, a.maxiter, thresh, y.b, y.xa, y.xb,
                           y.out, sh.tot[lane], sh.hint[lane], blk);
          // its passes come after the fast ones'
          if (!SAFE && sh.st[lane].safe) sh.st[lane].active = 0;
        }
        __syncwarp();
        plan();
        if (lane == 0) sh.slot = ring_at(slot, 1, kResSlots);
      }
    }
    __syncthreads();
    if (!sh.ok) return;
  }
}

// The systems left to single sweeps.  False when a barrier wait gave up.
template <int FORM, int TILES>
__device__ __forceinline__ bool solve_singly(const JacobiGroup& a, PassShared<TILES>& sh) {
  JacobiCtl* ctl = a.ctl;
  const ExactGrid eg{a.nx,   a.ny,     a.nx,       a.maxiter, a.thresh, a.rowstart, a.cols,
                     ctl->acc, &ctl->bar[a.sys[0].solve_idx], &ctl->status, a.spin_limit};
  for (int q = 0; q < a.nsys; ++q)
    if (sh.st[q].exact && !solve_exact<FORM>(eg, a.sys[q], sh.st[q], &sh.xpass, &sh.nbar))
      return false;
  return true;
}

// The systems that the fast passes left: by passes with IEEE divisions, then by single
// sweeps.  One call out of line: what it needs must not come out of the fast passes'
// registers.  (The divided rows have no such passes: a call like this one cost their strips
// 4% at 2048^2, 1766 against 1696 us a step.)
template <int FORM, int TILES>
__device__ __noinline__ bool solve_rest(const JacobiGroup& a, PassShared<TILES>& sh) {
  if (threadIdx.x < a.nsys) sh.st[threadIdx.x].active = sh.st[threadIdx.x].safe;
  __syncwarp();  // (warp 0 reads them first)
  solve_passes<FORM, TILES, true>(a, sh);
  return sh.ok && solve_singly<FORM, TILES>(a, sh);
}

template <int FORM, int TILES>
__global__ void __launch_bounds__(TILES ? kTileNT : kStripNT,
                                  TILES ? 1 : (FORM == kSysRecip ? 3 : 2))
    jacobi_kernel(const __grid_constant__ JacobiGroup a) {
  constexpr int T = PassShared<TILES>::T;
  __shared__ PassShared<TILES> sh;
  JacobiCtl* ctl = a.ctl;
  if (threadIdx.x < 32) {
    if (threadIdx.x < a.nsys) {
      const JacobiSys& y = a.sys[threadIdx.x];
      const int blk = a.block < 1 ? 1 : (a.block > T ? T : a.block);
      const int hint = y.hint_idx >= 0 ? __ldcg(&ctl->iters[y.hint_idx]) : 0;
      sh.hint[threadIdx.x] = hint;
      sh.st[threadIdx.x] = sys_start(a.maxiter, y.b, y.xa, y.out, hint, blk);
    }
    if (threadIdx.x == 0) {
      sh.slot = *((volatile int*)&ctl->pass_next);
      sh.xpass = *((volatile int*)&ctl->exact_next);
      sh.nbar = 0;
      sh.ok = 1;
    }
    __syncwarp();
  }
  solve_passes<FORM, TILES, false>(a, sh);
  if (!sh.ok) return;
  bool rest = false;
  for (int q = 0; q < a.nsys; ++q) rest = rest || sh.st[q].safe || sh.st[q].exact;
  if (rest) {
    __syncthreads();
    if constexpr (FORM == kSysRecip) {
      if (!solve_singly<FORM, TILES>(a, sh)) return;
    } else {
      if (!solve_rest<FORM, TILES>(a, sh)) return;
    }
  }
  // deliver the final iterates (haVec of the reference) to their destinations
  const int n = a.nx * a.ny;
  for (int q = 0; q < a.nsys; ++q) {
    const JacobiSys& y = a.sys[q];
    if (!sh.st[q].zero && sh.st[q].xin == y.out) continue;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x)
      y.out[c] = sh.st[q].zero ? 0. : __ldcg(&sh.st[q].xin[c]);
  }
  if (blockIdx.x == 0 && threadIdx.x < a.nsys) {
    const SysState& S = sh.st[threadIdx.x];
    ctl->iters[a.sys[threadIdx.x].solve_idx] = S.zero ? 0 : S.k;
    if (S.maxhit) atomicCAS(&ctl->status, 0, 1);
    if (threadIdx.x == 0) {
      *((volatile int*)&ctl->pass_next) = sh.slot;
      *((volatile int*)&ctl->exact_next) = sh.xpass;
    }
  }
}

struct JacobiLaunch {
  const void* fn;
  int threads, width, height;  // cells one block (tiles) or one chunk of a strip delivers
  size_t smem;
};

template <int FORM, int T>
static JacobiLaunch jacobi_tiles() {
  using G = Tile<FORM, T>;
  return {reinterpret_cast<const void*>(&jacobi_kernel<FORM, T>), kTileNT, G::UX, G::UY, G::bytes};
}

template <int FORM>
static JacobiLaunch jacobi_launch_of(int tiles) {
  if (tiles) return tiles == 8 ? jacobi_tiles<FORM, 8>() : jacobi_tiles<FORM, 4>();
  return {reinterpret_cast<const void*>(&jacobi_kernel<FORM, 0>), kStripNT, Strip<FORM>::U, 8,
          Strip<FORM>::bytes};
}

static JacobiLaunch jacobi_pick(int form, int tiles) {
  if (form == kSysRecip) return jacobi_launch_of<kSysRecip>(tiles);
  return form == kSysDiv ? jacobi_launch_of<kSysDiv>(tiles) : jacobi_launch_of<kSysCsr>(tiles);
}

int jacobi_grid_blocks(int form, int tiles, int device) {
  const JacobiLaunch l = jacobi_pick(form, tiles);
  int per_sm = 0, sms = 0;
  cudaFuncSetAttribute(l.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)l.smem);
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, l.fn, l.threads, l.smem) !=
      cudaSuccess)
    return -1;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  return per_sm < 1 ? -1 : per_sm * sms;
}

JacobiGrid jacobi_grid(int form, int device) {
  const int t8 = jacobi_grid_blocks(form, 8, device), t4 = jacobi_grid_blocks(form, 4, device);
  const JacobiGrid g{t8 < t4 ? t8 : t4, jacobi_grid_blocks(form, 0, device)};
  return g.tile_blocks < 1 || g.strip_blocks < 1 ? JacobiGrid{0, 0} : g;
}

// Which pieces a solve is cut into, by how many rounds they make over the resident blocks.
// Measured per step (13 solves of 8 to 11 sweeps, B200), 8-sweep tiles / 4-sweep tiles /
// strips: split 50^2 136 / 152 / 201 us, 320^2 (168 and 126 tiles of a launch's three
// systems over 148 blocks) 190 / 174 / 292, 512^2 (396 and 300) 252 / 295 / 332, 768^2 (864
// and 630) 414 / 457 / 421, 1024^2 721 / 746 / 555; FP64 400^2 (351 and 240) 287 / 280 / 355,
// 512^2 (528 and 390) 397 / 358 / 434, 600^2 (741 and 495) 479 / 449 / 430; CSR 600^2 559 / 537
// / 510; mPDeC2 257^2 (54 and 35) 69 / 88 / 148.  One round of either length beats two (a block
// keeps its rows of the system for the whole solve), the longer passes win up to three
// rounds (within 5% everywhere), strips beyond.
constexpr int kTileWaves = 3;

cudaError_t launch_jacobi(const JacobiGroup& a, const JacobiGrid& g, cudaStream_t s) {
  auto pieces = [&](const JacobiLaunch& l) {  // tiles, or chunks of at least 8 rows
    return (long long)a.nsys * ((a.nx + l.width - 1) / l.width) * ((a.ny + l.height - 1) / l.height);
  };
  const long long t8 = pieces(jacobi_pick(a.form, 8)), t4 = pieces(jacobi_pick(a.form, 4));
  const long long round = g.tile_blocks;
  const bool long_pass = a.block > 4;  // else 8-sweep tiles would carry halo for nothing
  const int tiles = long_pass && t8 <= round ? 8
                    : t4 <= round ? 4
                    : long_pass && t8 <= kTileWaves * round ? 8
                    : t4 <= kTileWaves * round ? 4 : 0;
  const JacobiLaunch l = jacobi_pick(a.form, tiles);
  long long blocks = tiles == 8 ? t8 : t4, most = round;
  if (tiles == 0) {
    blocks = (pieces(l) + kStripWarps - 1) / kStripWarps;
    most = g.strip_blocks;
  }
  if (blocks > most) blocks = most;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(blocks < 1 ? 1 : blocks));
  cfg.blockDim = dim3(l.threads);
  cfg.dynamicSmemBytes = l.smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  void* args[] = {const_cast<JacobiGroup*>(&a)};
  return cudaLaunchKernelExC(&cfg, l.fn, args);
}

// Ensembles: one cooperative launch solves a.nsets x a.nprob systems of any sizes, each
// with its own stop rule, by strips.  A pass visits the chunks of every system still
// iterating (a warp takes its first by its number, the others from a counter whose next
// value it fetches while it works); then each block decides for its share of the systems.
template <int FORM>
__global__ void __launch_bounds__(kStripNT, FORM == kSysRecip ? 3 : 2)
    jacobi_batch_kernel(const StripBatchArgs a) {
  constexpr int T = kPassT;
  static_assert(T + 1 <= kBatchSums, "sums of a pass");
  constexpr bool RECIP = FORM == kSysRecip;
  extern __shared__ __align__(16) unsigned char jring[];
  __shared__ int s_ok, s_xpass, s_nact, s_nexact;
  __shared__ unsigned int s_nbar;
  __shared__ SysState s_st;
  __shared__ __align__(16) JacobiArgs s_d;
  StripBatchCtl* ctl = a.ctl;
  unsigned int* bar = &ctl->bar[a.correction];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int blk = a.block < 1 ? 1 : (a.block > T ? T : a.block);
  const int warps = gridDim.x * kStripWarps, me = warp * gridDim.x + blockIdx.x;
  const int nsys = a.nsets * a.nprob, nwork = a.nsets * a.nitems;
  double2* ring = reinterpret_cast<double2*>(jring + warp * Strip<FORM>::warp_bytes);
  if (threadIdx.x == 0) {
    s_nbar = 0;
    s_xpass = *((volatile int*)&ctl->exact_next);
  }
  auto direct = [](const JacobiArgs& d) {  // where a pass may write the destination
    return d.pitch == d.nx ? d.out : const_cast<double*>(d.b);
  };
  auto start = [&](const JacobiArgs& d, int sys) {
    return sys_start(d.maxiter, d.b, d.xa, direct(d), a.hint ? __ldg(&a.hint[sys]) : 0, blk);
  };
  __syncthreads();
  bool begun = false;  // the systems' states are in memory
  for (int slot = 0;; slot = ring_at(slot, 1, 3), begun = true) {
    for (int w = me; w < nwork;) {
      unsigned int nw = 0;
      if (lane == 0) nw = (unsigned int)warps + atomicAdd(&ctl->work, 1u);
      const int set = w / a.nitems;
      const int4 it = a.items[w - set * a.nitems];
      const int sys = set * a.nprob + it.x;
      const JacobiArgs& d = a.descs[sys];
      int Tp, first, active = 1, safe = 0;
      const double* xin;
      double* xout;
      if (!begun) {  // the states are written by the first decisions
        const SysState S = start(d, sys);
        Tp = S.Tp;
        first = 1;
        xin = S.xin;
        xout = S.xout;
      } else {
        const SysState* S = &a.st[sys].s;
        active = __ldcg(&S->active);
        Tp = __ldcg(&S->Tp);
        first = __ldcg(&S->first);
        safe = __ldcg(&S->safe);
        xin = reinterpret_cast<const double*>(__ldcg(reinterpret_cast<const unsigned long long*>(&S->xin)));
        xout = reinterpret_cast<double*>(__ldcg(reinterpret_cast<const unsigned long long*>(&S->xout)));
      }
      if (active && SWM_IN_RANGE(it.x, a.nprob, kChkEnsItem)) {
        const int nx = d.nx, ny = d.ny, pitch = d.pitch;
        const unsigned long long al =
            (unsigned long long)xin | (unsigned long long)xout | (unsigned long long)d.b |
            (unsigned long long)d.cS | (unsigned long long)d.cW | (unsigned long long)d.cE |
            (unsigned long long)d.cN | (unsigned long long)d.cD;
        auto add = [&](const double (&sum)[T + 1]) {
#pragma unroll
          for (int t = 0; t <= T; ++t) {
            if (t > Tp) break;
            const double v = warp_sum(sum[t]);
            if (lane == t && v != 0.) atomicAdd(&a.st[sys].sum[t], v);
          }
        };
        if (!RECIP && safe) {  // (its sums are in local memory)
          double sum[T + 1];
          strip_pass_safe<FORM>(d, xin, xout, nx, ny, pitch, pitch, Tp, first != 0, it.y, it.z,
                                it.w, (al & 15ull) == 0, ring, sum);
          add(sum);
        } else {
          double sum[T + 1];
          strip_pass<FORM, false>(d, xin, xout, nx, ny, pitch, pitch, Tp, first != 0, it.y, it.z,
                                  it.w, (al & 15ull) == 0, ring, sum);
          add(sum);
        }
      }
      w = (int)__shfl_sync(0xffffffffu, nw, 0);
    }
    __syncthreads();
    if (threadIdx.x == 0) s_ok = arrive_and_wait(bar, ++s_nbar, a.spin_limit, &ctl->status);
    __syncthreads();
    if (!s_ok) return;
    // decisions: system p by thread p / gridDim.x of block p % gridDim.x
    for (int p = blockIdx.x + gridDim.x * threadIdx.x; p < nsys; p += gridDim.x * blockDim.x) {
      const JacobiArgs& d = a.descs[p];
      StripBatchState& B = a.st[p];
      SysState S = begun ? B.s : start(d, p);
      if (!S.active) continue;
      double sum[T + 1];
#pragma unroll
      for (int t = 0; t <= T; ++t) {
        sum[t] = __ldcg(&B.sum[t]);
        B.sum[t] = 0.;
      }
      const double thresh = limbs_value(d.thresh[0], d.thresh[1], d.thresh[2]);
      sys_decide<FORM>(S, (double)d.nx * d.ny, d.maxiter, thresh, d.b, d.xa, d.xb, direct(d), sum,
                        a.hint ? __ldg(&a.hint[p]) : 0, blk);
      B.s = S;
      if (S.active) atomicAdd(&ctl->nact[slot], 1);
      if (S.exact) atomicAdd(&ctl->nexact, 1);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      ctl->work = 0u;
      ctl->nact[ring_at(slot, 1, 3)] = 0;  // read by everyone before the barrier above
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      s_ok = arrive_and_wait(bar, ++s_nbar, a.spin_limit, &ctl->status);
      s_nact = __ldcg(&ctl->nact[slot]);
      s_nexact = __ldcg(&ctl->nexact);
    }
    __syncthreads();
    if (!s_ok) return;
    if (s_nact == 0) break;
  }
  if (blockIdx.x == 0 && threadIdx.x < 3) ctl->nact[threadIdx.x] = 0;  // the next launch's
  if (s_nexact > 0) {
    for (int p = 0; p < nsys; ++p) {
      if (!__ldcg(&a.st[p].s.exact)) continue;
      if (threadIdx.x == 0) {
        s_st = a.st[p].s;
        s_d = a.descs[p];
      }
      __syncthreads();
      const ExactGrid eg{s_d.nx,  s_d.ny,  s_d.pitch, s_d.maxiter,  s_d.thresh,   nullptr,
                         nullptr, ctl->acc, bar,       &ctl->status, a.spin_limit};
      if (!solve_exact<FORM>(eg, s_d, s_st, &s_xpass, &s_nbar)) return;
      if (blockIdx.x == 0 && threadIdx.x == 0) {
        s_st.exact = 0;
        a.st[p].s = s_st;
      }
      __syncthreads();
    }
    if (threadIdx.x == 0) s_ok = arrive_and_wait(bar, ++s_nbar, a.spin_limit, &ctl->status);
    __syncthreads();
    if (!s_ok) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      ctl->nexact = 0;
      *((volatile int*)&ctl->exact_next) = s_xpass;
    }
  }
  // deliver the iterates that the last pass did not write to their destinations, chunk by
  // chunk, and the sweep counts
  for (int w = me; w < nwork; w += warps) {
    const int set = w / a.nitems;
    const int4 it = a.items[w - set * a.nitems];
    const int sys = set * a.nprob + it.x;
    const JacobiArgs& d = a.descs[sys];
    const SysState* S = &a.st[sys].s;
    const double* x =
        reinterpret_cast<const double*>(__ldcg(reinterpret_cast<const unsigned long long*>(&S->xin)));
    const int zero = __ldcg(&S->zero);
    if (!zero && x == d.out) continue;
    const int i0 = it.y * Strip<FORM>::U, i1 = min(i0 + Strip<FORM>::U, d.nx);
    for (int j = it.z; j < it.z + it.w; ++j)
      for (int i = i0 + lane; i < i1; i += 32)
        d.out[(size_t)j * d.nx + i] = zero ? 0. : __ldcg(&x[(size_t)j * d.pitch + i]);
  }
  for (int p = blockIdx.x + gridDim.x * threadIdx.x; p < nsys; p += gridDim.x * blockDim.x) {
    const SysState* S = &a.st[p].s;
    a.iters[p] = __ldcg(&S->zero) ? 0 : __ldcg(&S->k);
    if (__ldcg(&S->maxhit)) atomicCAS(&ctl->status, 0, 1);
  }
}

static const void* batch_fn(bool recip) {
  return recip ? reinterpret_cast<const void*>(&jacobi_batch_kernel<kSysRecip>)
               : reinterpret_cast<const void*>(&jacobi_batch_kernel<kSysDiv>);
}

int jacobi_batch_strips(int nx) { return (nx + Strip<kSysDiv>::U - 1) / Strip<kSysDiv>::U; }

int jacobi_batch_grid_blocks(int device, bool recip) {
  const size_t smem = recip ? Strip<kSysRecip>::bytes : Strip<kSysDiv>::bytes;
  const void* fn = batch_fn(recip);
  int per_sm = 0, sms = 0;
  cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kStripNT, smem) != cudaSuccess)
    return -1;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  return per_sm < 1 ? -1 : per_sm * sms;
}

cudaError_t launch_jacobi_batch(const StripBatchArgs& a, int grid_blocks, bool recip,
                                cudaStream_t s) {
  const long long need = ((long long)a.nsets * a.nitems + kStripWarps - 1) / kStripWarps;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(need < grid_blocks ? (need < 1 ? 1 : need) : grid_blocks));
  cfg.blockDim = dim3(kStripNT);
  cfg.dynamicSmemBytes = recip ? Strip<kSysRecip>::bytes : Strip<kSysDiv>::bytes;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  void* args[] = {const_cast<StripBatchArgs*>(&a)};
  return cudaLaunchKernelExC(&cfg, batch_fn(recip), args);
}

// Batched TimeStep: block b covers 128 cells of problem blk[b].x from blk[b].y.
__global__ void __launch_bounds__(128)
    dt_batch_kernel(const DtBatchDesc* __restrict__ d, const int2* __restrict__ blk,
                    unsigned long long* lam, int* bad) {
  const int2 w = blk[blockIdx.x];
  const DtBatchDesc& q = d[w.x];
  const int c = w.y + threadIdx.x;
  double lx = 0.0, ly = 0.0;
  int b = 0;
  if (c < q.nx * q.ny) {
    double h = q.h[c], hu = q.hu[c], hv = q.hv[c], u, v;
    if (!(h >= 0.0) || !isfinite(h) || !isfinite(hu) || !isfinite(hv)) b = 1;
    cons_to_prim<true>(h, hu, hv, u, v);
    double cc = sqrt(q.g * h);
    lx = fabs(u + cc);
    ly = fabs(v + cc);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lx = dmax(lx, __shfl_down_sync(0xffffffffu, lx, o));
    ly = dmax(ly, __shfl_down_sync(0xffffffffu, ly, o));
  }
  b = __any_sync(0xffffffffu, b);
  // block maxima first: one pair of atomics per block, not per warp (the atomics of a
  // problem's blocks all go to the same two words)
  __shared__ double s_lx[4], s_ly[4];
  __shared__ int s_b[4];
  static_assert(128 / 32 == 4, "four warps per block");
  if ((threadIdx.x & 31) == 0) {
    s_lx[threadIdx.x >> 5] = lx;
    s_ly[threadIdx.x >> 5] = ly;
    s_b[threadIdx.x >> 5] = b;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int q = 1; q < 4; ++q) {
      lx = dmax(lx, s_lx[q]);
      ly = dmax(ly, s_ly[q]);
      b |= s_b[q];
    }
    atomicMax(&lam[2 * w.x], (unsigned long long)__double_as_longlong(lx));
    atomicMax(&lam[2 * w.x + 1], (unsigned long long)__double_as_longlong(ly));
    if (b) atomicOr(&bad[w.x], 1);
  }
}

// dt = CFL * min(HUGE, dx/LambdaMaxX, dy/LambdaMaxY), floored (equation.f90:818-834)
__global__ void dt_finalize_kernel(const DtBatchDesc* d, int nprob, const unsigned long long* lam,
                                   double* dt) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= nprob) return;
  const double LX = __longlong_as_double((long long)lam[2 * p]);
  const double LY = __longlong_as_double((long long)lam[2 * p + 1]);
  double ts = 1.7976931348623157e308;
  const double a1 = d[p].dx / LX, b1 = d[p].dy / LY;
  if (a1 < ts) ts = a1;
  if (b1 < ts) ts = b1;
  ts = d[p].cfl * ts;
  if (ts < 1.0e-30) ts = 1.0e-30;
  dt[p] = ts;
}

size_t ensemble_smem_bytes(int tb, int precision) {
  const size_t rhs = precision == SWM_PREC_SPLIT ? RhsSmem<float>::bytes : RhsSmem<double>::bytes;
  const size_t jac = tb <= 2 ? JTile<2>::bytes : (tb <= 4 ? JTile<4>::bytes : JTile<8>::bytes);
  return rhs > jac ? rhs : jac;
}

cudaError_t launch_dt_batch(const DtBatchDesc* d, const int2* blk, int nblk, int nprob,
                            unsigned long long* lam, int* bad, double* dt, cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(lam, 0, sizeof(unsigned long long) * 2 * nprob, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(bad, 0, sizeof(int) * nprob, s);
  if (e != cudaSuccess) return e;
  dt_batch_kernel<<<nblk, 128, 0, s>>>(d, blk, lam, bad);
  dt_finalize_kernel<<<(nprob + 127) / 128, 128, 0, s>>>(d, nprob, lam, dt);
  return cudaGetLastError();
}

}  // namespace swm
