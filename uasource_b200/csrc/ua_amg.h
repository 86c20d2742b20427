// Aggregation AMG preconditioner of the uv tangent (internal interface).
#pragma once
#include "ua_internal.h"

namespace ua {

struct Amg;

// Values of the collapsed cycle to fill after a numeric set-up.
struct CycFillReq {
  bool lo;   // BF16 copy of the finest level
  void* dw;  // receives the finest level's damped l1 diagonal per node (value precision)
};

// Fine-level view of one preconditioner application z = M^-1 r inside PCG.
// x0 holds the pre-smoothed fine vector (l1-Jacobi of r, written by the
// caller with amg_invd0); z receives the result (and pcopy, if set, a copy);
// part_rz the row-block partials of r.z.
struct AmgPcgView {
  const int *rowptr0, *colind0;
  const void* K0;
  const void* r;
  const void* x0;
  void* z;
  void* pcopy;
  double* part_rz;
  const unsigned char* cmask;
  const int *sel, *done;
  const int *rb_start0, *rb_sys0;
  int nrb0;
  int lpr;     // lanes per fine row (8 or 16)
  void* tmp;   // a free fine-level vector (residual, then corrected iterate)
  // optional timing hook around the fine-level launches (kind 0 restriction, 1 prolongation;
  // phase 0 before, 1 after)
  void (*mark)(void* ctx, int kind, int phase) = nullptr;
  void* mark_ctx = nullptr;
  // optional BF16 copy of K0 for the finest-level residual and smoothing (mixed precision)
  const void* K0lo = nullptr;
  // loop the row-block and node-block kernels over the active-block lists (amg_act_compact)
  bool act = false;
  // finest-level residual and smoothing over the node slices (amg_sell_fill done for this
  // tangent); sell_lo: read their BF16 values
  bool sell = false, sell_lo = false;
};

// Active-block lists.  After every convergence check the row blocks (and, for the smoothed
// transfers, the node blocks) of the systems still iterating are compacted on the device,
// in ascending order; list-driven kernels run a grid of about one wave that loops over the
// list, so converged systems of a batch cost no blocks.
struct ActList {
  const int* map = nullptr;  // list entry -> block id
  const int* cnt = nullptr;  // number of entries (device scalar)
  int cap = 0;               // blocks of the full structure
};
// Build the lists of a uv handle's hierarchy (level 0 uses the handle's row blocks,
// sys_rb_off0 = per-system prefix of those blocks); no-op when built.
int amg_act_init(ua_mesh* m, const std::vector<int>& sys_rb_off0);
// Recompute every list from sel/done (one launch).
void amg_act_compact(ua_mesh* m, const int* sel, const int* done, long long* launches);
ActList amg_act_rows0(const ua_mesh* m);
// grid of a list-driven kernel over at most nblocks blocks of 256 threads
int act_grid(int nblocks, int nsm);

// Build the hierarchy of every system of the handle (host aggregation,
// device structures; smoothed = smoothed-aggregation prolongators, else
// piecewise constant); no-op when built (the first call fixes the kind).  Returns UA_OK or an error code
// (the handle then keeps point-Jacobi).
int amg_setup(ua_mesh* m, bool smoothed);
void amg_free(Amg* a);
int amg_levels(const ua_mesh* m);
// l1-Jacobi inverse row sums of the fine level (VT-typed, valid after amg_numeric)
const void* amg_invd0(const ua_mesh* m);
// Numeric phase for a new tangent K0 (Galerkin products, smoother, coarsest inverses).
// sel (device): the systems of this Newton step (others keep their hierarchies); h_sel (host copy)
// and p_refresh > 1: each system's prolongators are recomputed on the first set-up of its solve
// (amg_restart_P) and then every p_refresh-th set-up, the coarse operators every time.
// graph: run the set-up's launches as a captured CUDA graph (captured once per kind of call).
// cyc: also fill the values of the collapsed cycle (cycle_init and cycle_alloc_values done).
int amg_numeric(ua_mesh* m, const int* rowptr0, const int* colind0, const void* K0, bool fp32,
                const unsigned char* cmask, long long* launches, const int* sel = nullptr,
                const std::vector<int>* h_sel = nullptr, int p_refresh = 1, bool graph = false,
                const CycFillReq* cyc = nullptr);
// the systems of `run` start a solve: their next set-up recomputes the prolongators
void amg_restart_P(ua_mesh* m, const std::vector<int>& run);
// uvh handles: extract the velocity block of the 3-dof tangent K3 (and its
// constraint mask) into the hierarchy's own finest level, then the numeric
// phase (FP64).
int amg_numeric_uvh(ua_mesh* m, const double* K3, const unsigned char* cmask3, long long* launches,
                    const CycFillReq* cyc = nullptr, bool graph = false);
// out3 = V-cycle(p3) on the velocity rows of 3-dof vectors (other rows untouched).
int amg_apply_uvh(ua_mesh* m, const double* p3, double* out3, const int* sel, const int* done, int lpr,
                  long long* launches);
// Node slices of a uv handle's finest level (structure once per handle; call before
// amg_act_init so that the slice blocks get an active list).  sys_rb_off0 is the handle's
// per-system row-block prefix; its row blocks must split at the u/v boundary.  UA_OK, else an
// error code and the CSR kernels stay in use.
int amg_sell_init(ua_mesh* m, const std::vector<int>& sys_rb_off0);
// Slice values of a new tangent K0 (KT = float if fp32, else double); lo: also the BF16 copy.
int amg_sell_fill(ua_mesh* m, const void* K0, bool fp32, bool lo, long long* launches, const int* sel = nullptr);
// Per-slice partials of the node-slice SpMV (p.q) and smoothing (r.z), and the per-system
// slice prefix (the PCG reductions sum these instead of the row-block partials).
void amg_sell_partials(const ua_mesh* m, const double** spart, const int** sys_sl_off);
// PCG SpMV over the node slices: q = mask(K p), partials p.q per slice (amg_sell_partials).
int amg_sell_spmv(ua_mesh* m, bool fp32, bool act, const int* sel, const int* done, const void* p,
                  const unsigned char* cmask, void* q, long long* launches);
// Refresh the BF16 copy of an FP32 finest-level tangent (allocated on first use;
// nullptr if that fails).
const void* amg_bf16_copy(ua_mesh* m, const float* K0, long long nnz, long long* launches);
// One V(1,1) cycle.  The finest level runs as row-block kernels (residual,
// aggregation, correction, smoothing); coarser levels use one thread per aggregate.
int amg_vcycle(ua_mesh* m, bool fp32, const AmgPcgView& v, long long* launches);

// ---- resident Krylov solves on the collapsed V-cycle (ua_pcg.cu) ----
bool cycle_supported(const ua_mesh* m);
int cycle_init(ua_mesh* m);
int cycle_alloc_values(ua_mesh* m, bool fp32, bool lo);
// values of the collapsed cycle: the finest level's slices (after its diagonal), and the coarse levels'
// operators and every Q (after the last A P)
void cycle_fill_fine(ua_mesh* m, const int* colind0, const void* K0, bool fp32, bool lo, const int* sel,
                     cudaStream_t st, long long* launches);
void cycle_fill_levels(ua_mesh* m, bool fp32, bool lo, const int* sel, cudaStream_t st, long long* launches);
struct PcgSolve {
  bool fp32, lo, prof;
  const int* sel;
  const int* colind;
  const void* K;
  const double* f;        // right-hand side (dofs)
  const int* dof_con;     // dof -> single-dof constraint or -1, with right-hand sides con_rhs at X + dX
  const double *con_rhs, *X;
  double *dX, *grhs;      // out: the solution; con_rhs - X
  void *r, *z, *p, *q;    // work, one pair per node in the value precision
  double* x;              // work, one FP64 pair per node
  const void* dw;
  double* tol2;           // [nsys]
  int *done, *its, *status;
  int maxit;
};
// sel: systems to solve; steps: expected iterations (the schedule's weights)
int pcg_resident(ua_mesh* m, const PcgSolve& v, const std::vector<int>& sel, const std::vector<int>& steps, int nsm,
                 long long* launches);
// l1-Jacobi sweeps on the thickness block by default.  A sweep is a pass with a barrier; five take the time of
// eight or less in steps that converge well, and their few more iterations do not move the step at which GMRES
// stalls (milliseconds a step and iterations, five against eight: P1 141x71 0.1 a 19 and 303, 21 and 300; 0.3 a
// 34 and 552, 37 and 529; P2 101x51 0.1 a 28 and 315, 29 and 280; 0.3 a 53 and 601, 53 and 518).  The sweeps are
// not weighted: l1 scaling bounds the modulus of the spectrum, but the block is an advection, its eigenvalues
// leave the real axis with the step, and Chebyshev weights, which are small on the axis alone, amplify there
// (0.5 a: P1 61x43 533 -> 2514 iterations, P1 281x141 2746 -> no convergence).
constexpr int kHSweepDefault = 5;
struct GmSolve {
  const int* rowptr;      // 3-dof CSR
  const double* K;
  const unsigned char* cmask;
  const int* sel;
  const double* f;
  double* dX;             // in: the particular solution on the constrained dofs; out: the solution
  const double* tol;      // [nsys] relative tolerances
  int *done, *its;
  int mr, maxit, max_cycles;
  int hsw;                // sweeps on the thickness block
};
// restarted GMRES of the uvh system (ua_gmres.cu), restart up to gmres_resident_max_restart()
int gmres_resident_max_restart();
int gmres_resident(ua_mesh* m, const GmSolve& v, const std::vector<int>& sel, const std::vector<int>& steps, int nsm,
                   long long* launches);
// device flag set by a resident solve whose team did not meet
const int* resident_error_flag(const ua_mesh* m);
int resident_error(int flag);  // UA_OK, or the error of a set flag
// pass classes of a profiled resident solve: operator, finest restriction, finest up pass, rest
int pcg_resident_status(ua_mesh* m, bool prof, double* ms, int* cnt);

}  // namespace ua
