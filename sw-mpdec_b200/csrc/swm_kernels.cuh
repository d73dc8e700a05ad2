// swm_kernels.cuh -- declarations shared by the host orchestration and the
// memory-bound kernels (dt, layouts, Patankar assembly, Jacobi).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "swm_device.cuh"
#include "swm_rhs.cuh"
#include "swm_rules.h"

namespace swm {

// Residual accumulator: |dx| in units of 2^-100 split into three 40-bit limbs.
// Integer addition is associative, so the residual sum (and with it the Jacobi
// stop index) does not depend on tiling, launch shape or atomic ordering.
constexpr int kResSlots = 3;    // ring of pass slots (see jacobi kernels)
constexpr int kMaxBlock = 8;    // max Jacobi sweeps per stencil pass
constexpr int kMaxSolves = 16;  // solves recorded per step
// Polls of a grid-barrier wait before it gives up (status -4); ~1 s at 40 ns a poll.
// A limit <= 0 makes every wait that is not already open give up at once.
constexpr long long kDefaultSpinLimit = 1LL << 26;

// Independent systems of one grid solved together by one launch: the three substeps of a
// correction iteration.
constexpr int kMaxSys = 3;

// How a system is stored: planes holding the row divided by its Diagonal and b/Diagonal
// (split and FMA forms), planes and Diagonal (FP64 form), or the reference's CSR values
// Mass[5N] in slot order S, W, C, E, N (finitevolume.f90:234-261) and Diagonal.
enum { kSysRecip = 0, kSysDiv = 1, kSysCsr = 2 };

struct JacobiCtl {
  // ring of passes: residual sums of every system, [0] initial, [1..] per sweep
  double sum[kResSlots][kMaxSys][kMaxBlock + 1];
  // ring of exact passes (one sweep each): limbs of the initial residual and the sweep's
  unsigned long long acc[kResSlots][2][3];
  unsigned int bar[kMaxSolves];  // barrier arrivals of the launch whose first solve it is
  int iters[kMaxSolves];  // iterations of each solve of the current step
  int status;             // 0 ok, 1 maxiter, -4 watchdog
  int pass_next;          // the next pass's position in the ring of sums, across solves
  int exact_next;         // the next exact pass's position in the ring of limbs
};

struct AssembleArgs {
  int nx, ny;
  double dx, dy;
  int m;                  // substep 2..4 (1-based, as in the reference)
  int msteps;             // 4 (mPDeC5) or 2 (mPDeC2)
  int compat2;            // mPDeC2 sequence-association read of hp
  int jpitch;             // row pitch of the stencil planes and rhs_out (<= 0: nx)
  double theta[4];        // thetaDeC(m, 1:4)
  const double* dt;       // device scalar
  const double* hu_n;     // Ua(1, 2:3) = U^n momentum
  const double* hv_n;
  const double* fu[4];    // FUp(r, 2) planes
  const double* fv[4];    // FUp(r, 3)
  const double* fxm[4];   // mass fluxes of stage r [ny][nx+1] (over dx unless fast)
  const double* fym[4];   // [ny+1][nx] (over dy unless fast)
  const double* hp[4];    // Up(r, 1) for r = 1..msteps (hp(m,.) is hp[m-1])
  double* hu_out;         // Ua(m, 2:3)
  double* hv_out;
  // stencil layout: 5 planes (S, W, E, N, Diag); CSR layout: mass[5N], diag[N]
  double* cS;
  double* cW;
  double* cE;
  double* cN;
  double* cD;
  double* csr_mass;
  double* csr_diag;
  double* rhs_out;        // nullable: rhs = hp(1,.) (needed when hp is read through compat2)
  // split form: PATANKAR_DIV from one reciprocal per depth, P/D by 1/dx, and the
  // stencil planes holding the row divided by its Diagonal, the D plane b/Diagonal
  // (not bit-identical to the reference order)
  int fast;
  double inv_dx, inv_dy;
};

// Substeps m of one mPDeC5 correction iteration assembled in one launch (stencil
// layout): `base` carries the shared inputs (stage RHS slots, face fluxes, hp, U^n
// momentum, dt, grid); per substep its number, weights and output planes.
constexpr int kMaxFusedStages = 3;
struct AssembleMultiArgs {
  AssembleArgs base;
  int nm;
  int m[kMaxFusedStages];  // 1-based substeps
  double theta[kMaxFusedStages][4];
  double* hu_out[kMaxFusedStages];
  double* hv_out[kMaxFusedStages];
  double* cS[kMaxFusedStages];
  double* cW[kMaxFusedStages];
  double* cE[kMaxFusedStages];
  double* cN[kMaxFusedStages];
  double* cD[kMaxFusedStages];
  double* csr_mass[kMaxFusedStages];  // CSR solver
  double* csr_diag[kMaxFusedStages];
};

struct JacobiArgs {
  int nx, ny;
  int maxiter;
  int pitch;              // stencil: row pitch of b, the coefficient planes and xa/xb
                          // (<= 0: nx); out is unpadded
  unsigned long long thresh[3];  // tol * n in residual units (limbs)
  const double* b;        // rhs (= hp(1) = h^n)
  // stencil coefficients
  const double* cS;
  const double* cW;
  const double* cE;
  const double* cN;
  const double* cD;
  double* xa;             // ping-pong buffers
  double* xb;
  double* out;            // final iterate destination
};

// One system of a JacobiGroup.
struct JacobiSys {
  const double* b;        // rhs (= hp(1) = h^n)
  const double* cS;       // stencil planes (see JacobiArgs)
  const double* cW;
  const double* cE;
  const double* cN;
  const double* cD;
  const double* mass;     // CSR values, Mass[5N] and Diagonal
  const double* diag;
  double* xa;             // ping-pong buffers
  double* xb;
  double* out;            // final iterate destination
  int solve_idx;          // slot in ctl->iters
  int hint_idx;           // slot of an earlier solve of this step whose sweep count plans
                          // the passes (the same substep's previous correction); < 0 none
};
struct JacobiGroup {
  int nx, ny, nsys;
  int maxiter;
  int block;              // sweeps per pass at most
  int form;               // kSysRecip, kSysDiv, kSysCsr (swm_strip.cuh)
  unsigned long long thresh[3];  // tol * n in residual units (limbs)
  const int* rowstart;    // CSR pattern, 1-based (finitevolume.f90:230,267)
  const int* cols;
  JacobiCtl* ctl;
  long long spin_limit;   // grid-barrier watchdog
  JacobiSys sys[kMaxSys];
};

struct DtArgs {
  int nx, ny;
  double g;
  const double* h;
  const double* hu;
  const double* hv;
  unsigned long long* lam;  // [2] bit patterns of LambdaMaxX/Y (non-negative doubles)
  int* bad;                 // non-finite or negative depth seen
};

// ---- ensembles: one launch covers every problem ----
// Jacobi state of one problem during a batched solve (global memory).
struct JacBatchState {
  int active;    // still iterating
  int k;         // sweeps done
  int Tp;        // sweeps of the coming pass
  int rollback;  // the coming pass redoes the last one with Tp sweeps
  int first;     // the coming pass is the first (initial residual checked)
  int cur;       // buffer holding x^k: 0 = b, 1 = xa, 2 = xb, 3 = the destination
  int result;    // final iterate: 0 = zero vector, 1 = xa, 2 = xb, 3 = the destination
  int final_k;
  int maxhit;
  int xnext;     // buffer the coming pass writes: 1 = xa, 2 = xb, 3 = the destination
  double r_prev;  // residual sum of the last sweep of the previous pass (pass planning)
  unsigned long long acc[kMaxBlock + 1][3];
};
struct JacBatchCtl {
  unsigned int bar_count, bar_gen;
  int n_active;
  int status;  // 0 ok, 1 some problem hit maxIter, -4 watchdog
};
struct JacobiBatchArgs {
  // per system (set q, problem p -> q * nprob + p): nx, ny, b, stencil planes, xa, xb,
  // out, thresh, maxiter
  const JacobiArgs* descs;
  const int2* tiles;        // (problem, tile index) of every tile of every problem
  int ntiles, nprob;
  int nsets;                // independent systems per problem solved together (>= 1)
  JacBatchState* st;        // [nsets * nprob]
  JacBatchCtl* ctl;
  int* iters;               // [nsets * nprob] sweeps of each system's solve
  int block;
  long long spin_limit;
  // nullable: work-item counter; when set, CTAs take a pass's tiles one at a time from
  // it (reset to 0 before every pass) instead of striding by CTA
  unsigned int* work;
};
// ---- the same solves by strips (the per-phase form; swm_strip.cuh) ----
// State of one system between passes.
struct SysState {
  const double* xin;
  double* xout;
  int k;            // sweeps done
  int Tp;           // sweeps of the coming pass
  int active;       // still iterating
  int first;        // the coming pass is the first
  int rollback;     // the coming pass redoes the last one with Tp sweeps
  int zero;         // converged before the first sweep: the reference returns 0
  int maxhit;
  int exact;        // left to solve_exact, which goes on from xin
  int safe;         // its passes divide by IEEE divisions
  float r_prev;     // residual sum of the last sweep of the previous pass (planning)
};
constexpr int kPassT = 4;  // sweeps per pass of the strips at most
constexpr int kJacobiBatchWarps = 4;  // warps per block of the batched solve
constexpr int kBatchSums = 8;  // residual sums of a pass, padded
struct StripBatchState {
  SysState s;
  double sum[kBatchSums];  // zero between passes
};
struct StripBatchCtl {
  unsigned int bar[5];          // barrier arrivals of each correction's launch
  int nact[3];                  // systems still iterating after a pass (ring)
  int nexact;                   // systems left to solve_exact in this launch
  int status;                   // 0 ok, 1 some problem hit maxIter, -4 watchdog
  int exact_next;
  unsigned int work;            // next work item of the pass
  unsigned long long acc[kResSlots][2][3];  // solve_exact's limbs
};
struct StripBatchArgs {
  const JacobiArgs* descs;  // [nsets * nprob], as JacobiBatchArgs
  const int4* items;        // (problem, strip, first row, rows) of every chunk of a set
  int nitems, nprob, nsets;
  int correction;           // 0..4: which barrier counter
  StripBatchState* st;      // [nsets * nprob], zeroed before the step
  StripBatchCtl* ctl;       // zeroed before the step
  int* iters;               // [nsets * nprob] sweeps of each system's solve
  const int* hint;          // nullable: sweeps of the same substeps' previous solves
  int block;                // sweeps per pass at most
  long long spin_limit;
};
struct DtBatchDesc {
  int nx, ny;
  double g, cfl, dx, dy;
  const double* h;
  const double* hu;
  const double* hv;
};

// ---- ensembles in one persistent launch per mPDeC5 step ----
constexpr int kEnsCells = 256;  // cells of one TimeStep / assembly work item (= CTA size)

struct EnsembleArgs {
  int nprob;
  int precision;             // SWM_PREC_*: which RHS tile function runs
  // TimeStep (equation.f90:791-837) of every problem
  const DtBatchDesc* dtd;
  const int2* cells;         // (problem, first cell) of every kEnsCells-cell block
  int ncells;
  unsigned long long* lam;   // [2 nprob] LambdaMax bit patterns, zeroed before the launch
  int* bad;                  // [nprob] non-finite / negative depth, zeroed before the launch
  double* dt;                // [nprob]
  // RHS: descriptors [set][nprob] (set 0: U^n; 1 + 3 par + m - 2: Ua(m) of correction
  // parity par) and the (problem, i0, j0) tiles of one set
  const RhsArgs* rhs;
  const int4* rtiles;
  int nrtiles;
  // combination + assembly: per (solve, problem) [13][nprob]; the fast forms' three
  // substeps of corrections 1..4 fused per cell [4][nprob]
  const AssembleArgs* asmd;
  const AssembleMultiArgs* asmm;
  // Jacobi: the systems of correction k = 1..5, [5][3 nprob]: set q = substep m - 2
  // (the last correction's one system is set 0)
  const JacobiArgs* jac;
  const int2* jtiles;        // (problem, tile) of every problem's Jacobi tiles
  int njtiles;
  JacBatchState* st;         // [3 nprob]
  JacBatchCtl* ctl;          // grid barrier and status, zeroed before the launch
  int* iters;                // [13][nprob] sweeps of every solve
  int block;                 // Jacobi sweeps per pass
  long long spin_limit;      // grid-barrier watchdog
  // nullable: the global timer (ns) when CTA 0 starts and leaves each phase's
  // closing barrier, kEnsMarks entries (measurement only)
  unsigned long long* clock;
  // work-item counters, zeroed before the launch: [0..4] RHS phases (U^n, k = 1..4),
  // [5..9] assembly phases (k = 1..5), [10] the Jacobi passes
  unsigned int* work;
};
constexpr int kEnsCounters = 11;
// start, TimeStep, RHS of U^n, then per correction assembly, Jacobi and (k < 5) RHS
constexpr int kEnsMarks = 3 + 5 * 3 - 1;
// The ensemble step kernel (swm_ensemble.cuh) of a precision form and a Jacobi
// temporal block tb (2, 4 or 8), as instantiated in the RHS units: split and FP64-FMA
// forms in swm_rhs_fast.cu, the FP64 form in swm_rhs_exact.cu.
const void* ensemble_kernel_fast(int mode, int tb);  // mode 1 split, 0 FP64-FMA
const void* ensemble_kernel_exact(int tb);
// dynamic shared memory of that kernel: the larger of the RHS tile's and the Jacobi
// tile's (swm_kernels.cu)
size_t ensemble_smem_bytes(int tb, int precision);

// Checked-build records of the three units with device-side index checks (see
// SWM_IN_RANGE): read and cleared; site -1 when the unit was built without them.
int check_record_kernels(int* site, unsigned long long* count);
int check_record_rhs_fast(int* site, unsigned long long* count);
int check_record_rhs_exact(int* site, unsigned long long* count);
int check_record_kernels_sites(unsigned int* seen);
int check_record_rhs_fast_sites(unsigned int* seen);
int check_record_rhs_exact_sites(unsigned int* seen);

// Host launchers (swm_kernels.cu, swm_rhs_*.cu)
cudaError_t launch_rhs_batch_fast(int mode, const RhsArgs* descs, const int4* work, int nwork,
                                  cudaStream_t s);
cudaError_t launch_rhs_batch_exact(const RhsArgs* descs, const int4* work, int nwork,
                                   cudaStream_t s);
cudaError_t launch_assemble_multi_batch(const AssembleMultiArgs* descs, const int2* blk, int nblk,
                                        cudaStream_t s);
cudaError_t launch_assemble_batch(const AssembleArgs* descs, const int2* blk, int nblk, bool fast,
                                  cudaStream_t s);
cudaError_t launch_jacobi_batch(const StripBatchArgs& a, int grid_blocks, bool recip,
                                cudaStream_t s);
int jacobi_batch_grid_blocks(int device, bool recip);
int jacobi_batch_strips(int nx);  // strips of a grid nx cells wide
cudaError_t launch_dt_batch(const DtBatchDesc* d, const int2* blk, int nblk, int nprob,
                            unsigned long long* lam, int* bad, double* dt, cudaStream_t s);
cudaError_t launch_rhs_fast(int mode, const RhsArgs& a, const RhsTma& tm, cudaStream_t s);
cudaError_t launch_rhs_exact(const RhsArgs& a, const RhsTma& tm, cudaStream_t s);
// n states of one grid in one launch; small: 8 x 8 tiles
cudaError_t launch_rhs_group_fast(int mode, const RhsGroup& g, int n, bool small, cudaStream_t s);
cudaError_t launch_rhs_group_exact(const RhsGroup& g, int n, bool small, cudaStream_t s);
size_t rhs_smem_bytes(int mode);

cudaError_t launch_dt(const DtArgs& a, cudaStream_t s);
cudaError_t launch_assemble(const AssembleArgs& a, bool csr, cudaStream_t s);
cudaError_t launch_assemble_multi(const AssembleMultiArgs& a, bool csr, cudaStream_t s);
// Resident blocks of the Jacobi kernel's two forms (swm_strip.cuh).
struct JacobiGrid {
  int tile_blocks, strip_blocks;  // tiles: the fewer of the two pass lengths' kernels
};
cudaError_t launch_jacobi(const JacobiGroup& a, const JacobiGrid& g, cudaStream_t s);
int jacobi_grid_blocks(int form, int tiles, int device);  // tiles: 8 or 4, 0 for strips
// both, or {0, 0} when a kernel cannot be resident
JacobiGrid jacobi_grid(int form, int device);
cudaError_t launch_ghosted_to_planes(const double* G, int nx, int ny, double* h, double* hu,
                                     double* hv, cudaStream_t s);
cudaError_t launch_planes_to_ghosted(const double* h, const double* hu, const double* hv, int nx,
                                     int ny, double* G, double* Vg, cudaStream_t s);
cudaError_t launch_summary(const double* h, int n, double* out /*[2]*/, cudaStream_t s);

// Stage combinations of the explicit schemes, out[v] for v = h, hu, hv (FP64, each
// product and sum rounded in the reference's order; out may alias X[0]):
//  kComboSsp  sum_i c_i X_i + sum_j (d_j Y_j) dt      SSPRK(5,4), forward Euler
//  kComboRk   X_0 + (sum_j d_j Y_j) dt                RK65
//  kComboDec  X_0 + sum_j (dt d_j) Y_j                DeC5
enum { kComboSsp = 0, kComboRk = 1, kComboDec = 2 };
constexpr int kComboMax = 6;
struct ComboArgs {
  int n;        // cells
  int form;
  int nx, ny;   // terms in X and Y
  double c[kComboMax], d[kComboMax];
  const double* dt;  // device scalar
  const double* X[kComboMax][3];
  const double* Y[kComboMax][3];
  double* out[3];
};
cudaError_t launch_combo(const ComboArgs& a, cudaStream_t s);

// Formatted output (swm_output.cu): one fixed-width line per cell.
struct OutLines {
  int nx, ny;
  int ncoord;      // 0 or 2: the barycentre coordinates first
  int nval;        // values per line after the coordinates (<= 4)
  int sep;         // spaces after every field (2X)
  int zero_small;  // print |v| < 1e-70 as 0
  double x0, y0, dx, dy;
  const double* val[4];  // planes [ny][nx]; null prints 0
  char* out;             // nx*ny lines of out_line_width() bytes
};
size_t out_line_width(const OutLines& a);
cudaError_t launch_out_lines(const OutLines& a, cudaStream_t s);
cudaError_t launch_prim(const double* h, const double* hu, const double* hv, double* u, double* v,
                        int n, cudaStream_t s);
// n values as 21-character (SP,ES21.14E2) fields, back to back
cudaError_t launch_format_values(const double* x, int n, char* out, cudaStream_t s);

// Initial conditions and the L1 error on the device (swm_ic.cu).
struct IcArgs {
  Grid gr;
  int ic;            // ExactFunction case: 1..6 (equation.f90:109-206), 101..105
  double par[8];     // parameters of cases 101..105
  double t;          // time of the exact solution (case 1 is advected)
  double sx[2];      // domain extents |x1 - x0| (MESH_SX)
  double* h;         // planes [ny][nx]: written by the fill, read by the L1 error
  double* hu;
  double* hv;
};
constexpr int kIcMaxBlocks = 148 * 8;
bool ic_supported(int ic);
int ic_blocks(int ncells);
cudaError_t launch_ic_fill(const IcArgs& a, cudaStream_t s);
// partial: 3 * ic_blocks(nx*ny) doubles of scratch; out: 3 doubles (device)
cudaError_t launch_l1_error(const IcArgs& a, double* partial, double* out, cudaStream_t s);
// Error(1:3) = U - Uexact(ic, t) into e[3] planes (output.f90:76-85; U read from a.h/hu/hv)
cudaError_t launch_error_planes(const IcArgs& a, double* const e[3], cudaStream_t s);
// Bath = 4x4 Gauss average of Bathymetry (finitevolume.f90:323-325) into b[N]
cudaError_t launch_bath_average(const IcArgs& a, double* b, cudaStream_t s);
void residual_limbs_host(double v, unsigned long long out[3]);

}  // namespace swm
