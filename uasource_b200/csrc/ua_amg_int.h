// Device structures of the AMG hierarchy and small device helpers, shared by the set-up and
// launch-per-pass cycle (ua_amg.cu) and the resident Krylov kernels (ua_cycle.cuh).
#pragma once
#include <cmath>
#include <vector>
#include <cuda_bf16.h>
#include "ua_amg.h"

namespace ua {

constexpr int kAmgCoarseNodes = 48;   // a system stops coarsening at this many nodes
constexpr int kAmgMaxRow = 32;        // longest coarse dof row (2 x coarse node degree)
constexpr int kSaMaxDeg = 256;        // largest coarse node degree of a smoothed hierarchy (shared-memory rows)
constexpr int kAmgMaxDense = 2 * kAmgCoarseNodes;
constexpr int kAmgRB = 256;           // rows per row block of a coarse level
constexpr int kSaRB = 128, kSaLPR = 2;
constexpr int kAmgNB = 32;            // nodes per node block of the smoothed transfers (one warp's worth)  // smoothed hierarchies (longer coarse rows): rows per block, lanes per row

// Damping of the prolongator smoother (l1 diagonal: rho(D^-1 A) <= 1).  4/3 is the textbook value for
// a diagonal with rho = 1; the l1 diagonal overestimates rho, and the iteration counts fall until
// about 1.7 (B200, summed Krylov iterations of a Newton solve, 4/3 -> 1.7: P1 229x113 mixed 187 ->
// 169, P2 401x201 FP64 353 -> 324, uvh P1 141x71 329 -> 309, C adjoint 75 -> 68).
constexpr double kSaOmega = 1.7;
// Damping of the smoother, folded into its inverse diagonal.  With the l1 row sums the spectrum of
// D^-1 A lies in (0, 1], so any factor below 2 keeps the sweep convergent and the cycle positive
// definite (0.5% of room covers the BF16 values of the mixed form), and the plain sweep (factor 1)
// leaves the whole lower half of the spectrum barely damped.
constexpr double kSmoothOmega = 1.8;

struct AmgLevel {
  int nn = 0, ndof = 0;
  long long nnz = 0;
  std::vector<int> node_off, dof_off, knz_off, nnzn;  // per system (0-sized when the system has no such level)
  // dof-level CSR of a coarse level, same layout rule as the finest level
  int *rowptr = nullptr, *colind = nullptr;
  int* dof_sys = nullptr;
  int* d_dof_off = nullptr;               // per-system dof offsets on the device
  int* d_knz_off = nullptr;               // per-system non-zero offsets (uvh finest level)
  int *rb_start = nullptr, *rb_sys = nullptr;
  int nrb = 0;
  int* cmap = nullptr;                    // this level's dof -> next level's dof
  int *mptr = nullptr, *mlist = nullptr;  // per dof of this (coarse) level: member dofs of the finer level
  void* A = nullptr;                      // coarse values (KT)
  void* invd = nullptr;                   // l1-Jacobi inverse row sums (VT)
  void *b = nullptr, *x = nullptr, *x2 = nullptr;  // rhs, pre-smoothed, post-smoothed (VT)
  int* d_node_off = nullptr;              // per-system node offsets on the device
  int* node_sys = nullptr;                // node -> system (smoothed hierarchies)
  std::vector<int> h_sys_rb_off;          // per-system prefix of the row blocks
  // node blocks (kAmgNB nodes, never straddling two systems) for the smoothed transfers
  int *nb_start = nullptr, *nb_sys = nullptr;
  int nnb = 0;
  std::vector<int> h_sys_nb_off;
  // smoothed aggregation, transfer from this level to the next (node-level lists, global ids):
  // pn: fine node -> coarse nodes of its neighbours' aggregates (the prolongator's node pattern);
  // apn: fine node -> coarse nodes of A P; ptn: coarse node -> (fine node, position in pn)
  // interpolation weights in pn order and the corner nodes (the finest level of a quadratic mesh), else null
  double* pn_w = nullptr;
  int* pn_f = nullptr;
  int *sa_agg = nullptr, *pn_ptr = nullptr, *pn_col = nullptr, *apn_ptr = nullptr, *apn_col = nullptr;
  int *ptn_ptr = nullptr, *ptn_fine = nullptr, *ptn_k = nullptr;
  // lists of the set-up (sa_lists): per node {first entry of its u row, of its v row, degree, system};
  // per entry of A P its fine node, its entry of P (-1: none) and its products (neighbour position,
  // entry of P); per entry of the next level's operator its node and its products (entry of P, entry
  // of A P)
  int4* nrow = nullptr;
  int *ap_node = nullptr, *ap_p = nullptr, *ac_node = nullptr;
  unsigned *ap_lptr = nullptr, *ac_lptr = nullptr;
  int2 *ap_l = nullptr, *ac_l = nullptr;
  int* gptr = nullptr;       // node graph of a coarse level
  long long nap = 0, ng = 0;  // entries of A P, of the node graph (coarse levels)
  void* sa_ap = nullptr;      // A P, one quad per entry (value type of the form)
  // P in the transfer layout, one quad per node-level entry: pn order (sa_q*) and ptn order
  // (sa_qt*); BF16 quads for the mixed form, FP64 quads for the FP64 form (allocated on first use)
  long long np = 0;  // node-level prolongator entries of the level (all systems)
  void *sa_qh = nullptr, *sa_qth = nullptr, *sa_qd = nullptr, *sa_qtd = nullptr;
};

// one active-block list to compact: blocks blk_off[s] .. blk_off[s+1] of every system s with
// sel, !done and depth > lmin, in ascending order
struct ActSpec {
  const int* blk_off;
  int lmin;
  int* map;
  int* cnt;
};

// Finest-level node slices of a uv handle (sliced ELL over nodes).  A slice block is the set of
// nodes of one u-row block of the handle's Krylov rows (at most kSellNodes nodes of one system);
// inside it the nodes are ordered by decreasing degree and cut into slices of 32, one warp each.
// Slice j holds width W_j = its largest degree; its slots are 32 * W_j, entry k of lane t at slot
// off_j + 32 k + t.  Per slot: the u column (global u dof of the k-th neighbour; v column = u column
// + the system's node count) and four values (blocks uu, uv, vu, vv at value offsets
// 4 off_j + b 32 W_j + 32 k + t).  Padding slots hold zeros and the node's own column.  One column
// index then serves four values, and a warp's loads of one k are contiguous.
constexpr int kSellNodes = 256;  // nodes per slice block (= rows per row block)
constexpr int kSellSlices = kSellNodes / 32;

struct Sell {
  bool ready = false, failed = false;
  int nsb = 0;
  long long slots = 0;
  std::vector<int> h_sys_sb_off;  // per-system prefix of the slice blocks
  std::vector<int> h_perm;
  std::vector<long long> h_sl_off;
  int *sb_sys = nullptr, *sb_n0 = nullptr, *sb_cnt = nullptr;
  int* perm = nullptr;             // [nn_total]: per block, its global node ids in slice order
  long long* sl_off = nullptr;     // [nsb * kSellSlices + 1] slot offsets of the slices
  int* cols = nullptr;             // [slots]
  float* v32 = nullptr;            // [4 slots] FP32 values (mixed-precision PCG operator)
  double* v64 = nullptr;           // [4 slots] FP64 values
  __nv_bfloat16* vlo = nullptr;    // [4 slots] BF16 values (mixed-precision V-cycle)
  double* spart = nullptr;         // [nsb * kSellSlices] per-slice partials (p.q, r.z)
  int* sys_sl_off = nullptr;       // [nsys + 1] per-system slice prefix
  ActList act;                     // slice blocks of the systems still iterating
};

// Collapsed cycle (ua_cycle.cuh): device pointers of one level.  A quad is the four values of a
// node pair; the types of the quads are the form's.
constexpr int kCycMaxLev = 12;
struct CycLev {
  const int *aptr, *acol;   // node rows of the level's operator (levels >= 1)
  void* aval;               // scaled operator, aptr order
  const int* qptr;          // node rows of Q (the A P pattern), levels >= 1
  const long long* qoff;    // slices of Q, finest level
  const int* qcol;
  void* qval;
  const int *tptr, *tfine;  // rows of Q' by coarse node
  void* tval;
  void *b, *z;              // right-hand side and result, one pair per node (levels >= 1)
};
// one system of the handle: first node and node count on every level, slices, dense inverse
// solo: first level that every CTA of a team works through for itself (depth: none)
struct CycSys {
  int depth, solo, dn, doff, sl0, nsl;
  int n0[kCycMaxLev + 1], nn[kCycMaxLev + 1];
};
// node slices of the finest level; columns are slice positions
struct CycFine {
  const int* perm;           // position -> node
  const long long* sl_off;
  const int* cols;
};
struct CycArgs {
  CycLev lev[kCycMaxLev];
  CycFine fine;
  const CycSys* sys;
  const double* dense;
  const int4* cta;     // per CTA: queue begin, end, rank in its team, team size
  const int *team, *queue;
  unsigned* bar;       // arrival counter of team k at 32 k
  int* err;
  unsigned long long* prof;
  double* part;        // [3][nslices]
  long long nslices;
  unsigned long long* dbg;  // bounds-checked build
};
// Value types of a form: FP64; the mixed form with the finest level in BF16; the mixed form all in FP32.
// Q holds the smoothing of the operator beside it, so it has that operator's type: FP32 on the coarse levels
// of the mixed form, BF16 on the finest only where the operator there is.  (BF16 everywhere was no faster:
// 16 meshes mixed 44.3 ms against 44.1, P2 101x51 7.87 against 7.59.)
enum CycForm { CF_FP64 = 0, CF_LO, CF_FP32, CF_COUNT };
inline CycForm cyc_form(bool fp32, bool lo) { return !fp32 ? CF_FP64 : lo ? CF_LO : CF_FP32; }
// Set-up data of the collapsed cycle: structure once per handle, values per tangent.
struct Cycle {
  bool ready = false, failed = false;
  std::vector<CycSys> sys;
  CycSys* d_sys = nullptr;
  struct Lev {
    int* ncol = nullptr;                                       // node graph (levels >= 1)
    long long nq = 0;                                          // node-level entries of Q
    // Q: the A P lists on levels >= 1; on the finest level node slices (qoff, padding slots zero),
    // qslot the slot of an A P entry
    long long* qoff = nullptr;
    int *qcol = nullptr, *qslot = nullptr;
    int *tptr = nullptr, *tfine = nullptr, *tpos = nullptr;    // Q' lists; tpos: A P entry -> entry of Q'
    double2* sc = nullptr;                                     // D^-1/2 per node (u, v)
    void *a32 = nullptr, *a64 = nullptr;                       // scaled operator quads (levels >= 1)
    // Q and Q' quads: BF16 on the finest level beside the BF16 operator, else FP32 or FP64 (CycForm)
    void *qh = nullptr, *qf = nullptr, *qd = nullptr, *th = nullptr, *tf = nullptr, *td = nullptr;
    void* q(int form, int l) const { return form == CF_FP64 ? qd : form == CF_LO && l == 0 ? qh : qf; }
    void* t(int form, int l) const { return form == CF_FP64 ? td : form == CF_LO && l == 0 ? th : tf; }
  };
  std::vector<Lev> lev;
  // resident kernel: schedule (one int4 per CTA: queue begin, end, team rank, team size), queue,
  // team counters, per-slice partials, profile clocks
  int last_grid = 0;
  // one block uploaded per solve: error flag, per-CTA entries, teams, queue, barrier counters (zeros)
  int* d_sched = nullptr;
  int at_team = 0, at_queue = 0, at_bar = 0;
  double* d_part = nullptr;   // [3][slices]
  unsigned long long* d_prof = nullptr;
  int *d_ipos = nullptr, *d_pcol = nullptr;  // node -> slice position; slot columns as positions
  // uvh: basis and work vectors, partials, 3-dof tangent and inverse thickness l1 sums (slice order)
  double *gm_buf = nullptr, *gm_part = nullptr, *gm_v3 = nullptr, *gm_hinv = nullptr;
  int gm_mr = 0;  // restart that they are for (0: none)
  void* d_r2 = nullptr;       // second residual buffer
  std::vector<double> h_solo[CF_COUNT];   // per system: bytes of its solo levels
  std::vector<double> h_bytes[CF_COUNT];  // per system: bytes of the matrices a step reads
  int* h_stage = nullptr;     // pinned staging of the schedule
  long long nslices = 0;
  ~Cycle() {
    if (h_stage) cudaFreeHost(h_stage);
  }
};

struct Amg {
  int nsys = 0, nlev = 0, maxdn = 0;
  Sell sell;
  Cycle cyc;
  // host node graphs and A P lists of the levels, kept until the cycle's structure is built
  std::vector<std::vector<int>> h_gptr, h_gcol, h_apnp, h_apnc;
  // node slices of the coarse levels 1 .. nlev-2 (smoothed hierarchies): BF16 copies of the
  // coarse operators for the mixed-precision V-cycle's residual and smoothing there
  std::vector<Sell> csell;
  bool csell_tried = false;
  // active-block lists: rows[l] (level-l row blocks, depth > l; level 0 = the handle's blocks),
  // fnodes[l] (level-l node blocks, depth > l), cnodes[l] (level-(l+1) node blocks, depth > l)
  bool act_ready = false;
  int nsm = 148;
  std::vector<ActList> rows, fnodes, cnodes;
  ActSpec* d_specs = nullptr;
  int nspecs = 0;
  bool sa = false;            // smoothed aggregation (else plain)
  std::vector<AmgLevel> lev;  // lev[0] = the handle's own system
  std::vector<int> depth;     // per system: its coarsest level (>= 1)
  std::vector<int> h_dn, h_doff;
  int *d_depth = nullptr, *d_dn = nullptr, *d_doff = nullptr;
  double* dense = nullptr;    // per system dn x dn inverse (row-major)
  void **d_lev_b = nullptr, **d_lev_x2 = nullptr, **d_lev_A = nullptr;
  int **d_lev_rowptr = nullptr, **d_lev_colind = nullptr, **d_lev_dofoff = nullptr;
  size_t bytes = 0;
  __nv_bfloat16* k0lo = nullptr;  // mixed precision: BF16 copy of the finest-level tangent
  // uvh handles: constraint mask and vectors of the velocity rows (2-dof layout)
  unsigned char* uvh_mask = nullptr;
  double *uvh_r = nullptr, *uvh_x0 = nullptr, *uvh_z = nullptr, *uvh_t = nullptr;
  // per system: numeric set-ups since its solve started (prolongator refresh), and the systems
  // whose prolongators the current set-up recomputes
  std::vector<int> p_age, h_prefresh;
  int* d_prefresh = nullptr;
  int* h_pin = nullptr;  // pinned, two alternating copies of the refresh selection
  int pin_at = 0;
  bool lists = false;  // the levels' set-up lists are built
  // side branch of the captured set-up: the finest level's slice values beside the coarse levels
  cudaStream_t side = nullptr;
  cudaEvent_t fork = nullptr, join = nullptr;
  // the numeric set-up of a Newton step captured as one CUDA graph per (precision, selection
  // kind) and replayed: every argument is a fixed device buffer of the handle
  cudaGraphExec_t setup_exec[32] = {};
  long long setup_nodes[32] = {};
  ~Amg() {
    if (h_pin) cudaFreeHost(h_pin);
    if (side) cudaStreamDestroy(side);
    if (fork) cudaEventDestroy(fork);
    if (join) cudaEventDestroy(join);
    for (auto& e : setup_exec)
      if (e) cudaGraphExecDestroy(e);
  }
};

template <class T>
inline T* upload(ua_mesh* m, Amg* a, const std::vector<T>& v, bool& ok) {
  T* d = (T*)dev_alloc(m, std::max<size_t>(1, v.size()) * sizeof(T));
  if (!d) { ok = false; return nullptr; }
  if (!v.empty() && dev_write(m, d, v.data(), v.size() * sizeof(T)) != cudaSuccess) ok = false;
  a->bytes += v.size() * sizeof(T);
  return d;
}

inline void* dalloc(ua_mesh* m, Amg* a, size_t bytes, bool& ok) {
  void* d = dev_alloc(m, std::max<size_t>(bytes, 16));
  if (!d) ok = false;
  a->bytes += bytes;
  return d;
}

// quads of the set-up (A P): four values of a node pair
__device__ __forceinline__ void quad_put(double* base, long long e, double a, double b, double c, double d) {
  double2* p = reinterpret_cast<double2*>(base) + 2 * e;
  p[0] = make_double2(a, b);
  p[1] = make_double2(c, d);
}
__device__ __forceinline__ void quad_put(float* base, long long e, float a, float b, float c, float d) {
  reinterpret_cast<float4*>(base)[e] = make_float4(a, b, c, d);
}
__device__ __forceinline__ void quad_at(const double* base, long long e, double* v) {
  const double2* p = reinterpret_cast<const double2*>(base) + 2 * e;
  const double2 a = p[0], b = p[1];
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
__device__ __forceinline__ void quad_at(const float* base, long long e, double* v) {
  const float4 a = reinterpret_cast<const float4*>(base)[e];
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
}

__device__ __forceinline__ double to_d(double v) { return v; }
__device__ __forceinline__ double to_d(float v) { return (double)v; }
__device__ __forceinline__ double to_d(__nv_bfloat16 v) { return (double)__bfloat162float(v); }

// The four values of a slot (blocks uu, uv, vu, vv) are adjacent, so a lane reads them with one
// vector load: 8 bytes (BF16), 16 (FP32) or 32 (FP64, two loads).
template <typename KT> struct Quad;
template <> struct Quad<float> {
  static __device__ __forceinline__ void get(const float* p, double (&e)[4]) {
    const float4 q = __ldg(reinterpret_cast<const float4*>(p));
    e[0] = q.x; e[1] = q.y; e[2] = q.z; e[3] = q.w;
  }
};
template <> struct Quad<double> {
  static __device__ __forceinline__ void get(const double* p, double (&e)[4]) {
    const double2 q0 = __ldg(reinterpret_cast<const double2*>(p)), q1 = __ldg(reinterpret_cast<const double2*>(p) + 1);
    e[0] = q0.x; e[1] = q0.y; e[2] = q1.x; e[3] = q1.y;
  }
};
template <> struct Quad<__nv_bfloat16> {
  static __device__ __forceinline__ void get(const __nv_bfloat16* p, double (&e)[4]) {
    const uint2 q = __ldg(reinterpret_cast<const uint2*>(p));
    // a BF16 value is the upper half of the FP32 value with the same bits
    e[0] = __uint_as_float(q.x << 16); e[1] = __uint_as_float(q.x & 0xffff0000u);
    e[2] = __uint_as_float(q.y << 16); e[3] = __uint_as_float(q.y & 0xffff0000u);
  }
};

// P in the transfer layout: per node-level entry (fine node g, coarse node K) one quad of
// P((c,g),(c2,K)) in the order (c,c2) = (0,0), (0,1), (1,0), (1,1), read with one load.  The mixed
// form keeps BF16 quads (its set-up then reads the same rounded values, so the coarse operator is
// the Galerkin product of the prolongator the V-cycle applies), the FP64 form FP64 quads.
struct alignas(8) PQuadH {
  __nv_bfloat162 r0, r1;
};
struct alignas(16) PQuadD {
  double2 r0, r1;
};
template <typename VT>
struct PQuadOf {
  using T = PQuadD;
};
template <>
struct PQuadOf<float> {
  using T = PQuadH;
};
__device__ __forceinline__ void pq_get(const PQuadH* q, double (&v)[4]) {
  const uint2 u = __ldg(reinterpret_cast<const uint2*>(q));
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
  const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
__device__ __forceinline__ void pq_get(const PQuadH* q, float (&v)[4]) {
  const uint2 u = __ldg(reinterpret_cast<const uint2*>(q));
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
  const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
__device__ __forceinline__ void pq_get(const PQuadD* q, double (&v)[4]) {
  const double2 a = __ldg(&q->r0), b = __ldg(&q->r1);
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
__device__ __forceinline__ void pq_set(PQuadH* q, double v0, double v1, double v2, double v3) {
  PQuadH h;
  h.r0 = __floats2bfloat162_rn((float)v0, (float)v1);
  h.r1 = __floats2bfloat162_rn((float)v2, (float)v3);
  *q = h;
}
__device__ __forceinline__ void pq_set(PQuadD* q, double v0, double v1, double v2, double v3) {
  q->r0 = make_double2(v0, v1);
  q->r1 = make_double2(v2, v3);
}

}  // namespace ua
