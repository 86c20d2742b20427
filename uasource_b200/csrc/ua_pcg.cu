// Resident PCG of the uv Newton system: one cooperative launch runs the whole preconditioned
// conjugate-gradient solve of every selected system (ua_cycle.cuh: collapsed V-cycle, teams).
//
// What bounds the inner solve of a mesh up to some 100,000 nodes is not memory but the chain of
// short passes: with one launch per pass a PCG step of the 141x71 mesh took 72 us in 19 launches
// of about 3.8 us.  Here a step is 1 + 2 L passes for the L levels above the dense one and the solo
// ones (22 us on that mesh), a team barrier costs 1.25 us whatever the team's size, nothing is
// launched inside the solve, the systems of a batch do not wait for one another and the host neither
// checks nor over-runs the convergence.  With a launch per pass and with the resident kernel as it
// was first built, one B200: uv P1 141x71 FP64 25.8 and 12.9 ms, P2 101x51 mixed 41.6 and 21.6 ms, P2
// 401x201 FP64 180 and 125 ms, 16 meshes of 2k-200k elements mixed 84 and 58 ms.
#include <algorithm>
#include <cstring>
#include "ua_cycle.cuh"

namespace ua {

// ---------------------------------------------------------------------------
// set-up: values of the collapsed cycle for a new tangent
// ---------------------------------------------------------------------------

constexpr int kCycArena = 208 * 1024;       // with the kernel's static tables below 227 KB
constexpr int kCycArenaSmall = 64 * 1024;
constexpr int kSplitSlices = 12;

template <typename T> struct QuadSet;
template <> struct QuadSet<double> {
  static __device__ __forceinline__ void set(void* base, long long e, double a, double b, double c, double d) {
    double2* p = reinterpret_cast<double2*>(base) + 2 * e;
    p[0] = make_double2(a, b);
    p[1] = make_double2(c, d);
  }
};
template <> struct QuadSet<float> {
  static __device__ __forceinline__ void set(void* base, long long e, double a, double b, double c, double d) {
    reinterpret_cast<float4*>(base)[e] = make_float4((float)a, (float)b, (float)c, (float)d);
  }
};
template <> struct QuadSet<__nv_bfloat16> {
  static __device__ __forceinline__ void set(void* base, long long e, double a, double b, double c, double d) {
    pq_set(reinterpret_cast<PQuadH*>(base) + e, a, b, c, d);
  }
};

// Columns of the node slices as slice positions, once per handle (padding slots: the lane's own).
__global__ void __launch_bounds__(256) k_cyc_cols(CycFine F, const int* sb_n0, const int* sb_cnt, const int* nodeptr,
                                                  const int* nodecol, const int* ipos, int* cols) {
  const int sb = blockIdx.x, w = threadIdx.x >> 5, t = threadIdx.x & 31, pos = w * 32 + t, sl = sb * kSellSlices + w;
  const long long o0 = F.sl_off[sl];
  const int W = (int)((F.sl_off[sl + 1] - o0) >> 5);
  const int at = sb_n0[sb] + min(pos, sb_cnt[sb] - 1);
  const int p0 = nodeptr[F.perm[at]], deg = pos < sb_cnt[sb] ? nodeptr[F.perm[at] + 1] - p0 : 0;
  for (int k = 0; k < W; ++k) cols[o0 + 32LL * k + t] = k < deg ? ipos[nodecol[p0 + k]] : at;
}

// Scaled values of the finest level in its node slices (SliceQuad layouts), from the dof CSR (row
// (c, g): the u block then the v block of deg(g) entries).  One warp per kFillN nodes of a slice: 8
// neighbours at a time, a load covering both rows and both blocks of one node in 64-byte segments;
// turned in shared memory and written as kFillN nodes of the slice row (whole sectors).  Bound by
// memory: P2 401x201 moves 0.26 GB in 81 us (a lane per row, each with four streams: 116 us).
constexpr int kFillWarps = 4, kFillN = 8;
template <typename KT>
__global__ void __launch_bounds__(32 * kFillWarps) k_cyc_fill0(
    CycFine F, int nsl, const int* sb_n0, const int* sb_cnt, const int* sb_sys, const int* node_off,
    const int* dof_off, const int4* nrow, const int* colind, const KT* K, const double2* sc, KT* vk,
    __nv_bfloat16* vlo, const int* sel) {
  static_assert(kFillN == 8, "lane = 16 row + 8 block + neighbour");
  __shared__ KT sv[kFillWarps][4][8][kFillN + 1];
  __shared__ int4 hr[kFillWarps][kFillN];
  __shared__ double hs[kFillWarps][kFillN][2];
  const int wid = threadIdx.x >> 5, t = threadIdx.x & 31;
  const int sub = blockIdx.x * kFillWarps + wid, sl = sub / (32 / kFillN), n0 = (sub % (32 / kFillN)) * kFillN;
  if (sl >= nsl) return;  // whole warps
  const int sb = sl / kSellSlices, s = sb_sys[sb];
  if (sel && !sel[s]) return;
  const long long o0 = F.sl_off[sl];
  const int W = (int)((F.sl_off[sl + 1] - o0) >> 5);
  if (W == 0) return;
  const int no = node_off[s], shift = no - dof_off[s];
  if (t < kFillN) {
    const int pos = (sl % kSellSlices) * 32 + n0 + t;
    int4 r = make_int4(0, 0, 0, 0);
    double2 si = make_double2(0, 0);
    if (pos < sb_cnt[sb]) {
      const int g = F.perm[sb_n0[sb] + pos];
      r = nrow[g];
      si = sc[g];
    }
    hr[wid][t] = r;
    hs[wid][t][0] = si.x;
    hs[wid][t][1] = si.y;
  }
  const int row = t >> 4, blk = (t >> 3) & 1, kl = t & 7;
  for (int k0 = 0; k0 < W; k0 += 8) {
    __syncwarp();
    const int k = k0 + kl;
    int c[kFillN];
    double v[kFillN];
#pragma unroll
    for (int n = 0; n < kFillN; ++n) {
      const int4 r = hr[wid][n];
      c[n] = k < r.z ? colind[r.x + k] + shift : -1;
      v[n] = k < r.z ? (double)K[(row ? r.y : r.x) + (blk ? r.z : 0) + k] : 0.0;
    }
#pragma unroll
    for (int n = 0; n < kFillN; ++n) {
      const double sj = c[n] >= 0 ? reinterpret_cast<const double*>(sc)[2 * (size_t)c[n] + blk] : 0.0;
      sv[wid][2 * row + blk][kl][n] = (KT)(hs[wid][n][row] * v[n] * sj);
    }
    __syncwarp();
    if (sizeof(KT) == 8) {  // two blocks of 32 pairs (SliceQuad)
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int u = q * 32 + t, n = u & 7, half = (u >> 3) & 1, kk = u >> 4;
        if (k0 + kk < W)
          reinterpret_cast<double2*>(vk)[2 * (o0 + 32LL * (k0 + kk)) + 32 * half + n0 + n] =
              make_double2((double)sv[wid][2 * half][kk][n], (double)sv[wid][2 * half + 1][kk][n]);
      }
    } else {
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int u = q * 32 + t, n = u & 7, kk = u >> 3;
        if (k0 + kk >= W) break;
        const long long d = o0 + 32LL * (k0 + kk) + n0 + n;
        const KT e0 = sv[wid][0][kk][n], e1 = sv[wid][1][kk][n], e2 = sv[wid][2][kk][n], e3 = sv[wid][3][kk][n];
        QuadSet<KT>::set(vk, d, e0, e1, e2, e3);
        if (vlo) QuadSet<__nv_bfloat16>::set(vlo, d, e0, e1, e2, e3);
      }
    }
  }
}

// Scaled values of the coarse levels' operators (node-row order) and of Q = D^1/2 (P - D^-1 A P)
// D_c^-1/2 (A P pattern, in row order and in the order of Q'; coarse nodes on a system's coarsest level
// are not scaled), every level in one launch: a lane per entry, the blocks dealt out by segment.
struct CycSeg {
  int b0;          // first block
  int lev;         // level of Q, or -1: an operator
  long long n;     // entries
  const int *node, *col, *ptr;  // entry -> node, its column, node -> first entry
  const int4* nrow;
  const double2 *sc, *scc;
  const void* val;  // A P quads, or the operator's dof CSR values
  const void* P;
  const int *own, *qslot, *tpos;
  void *out, *outT;
};
struct CycSegs {
  int n;
  CycSeg s[2 * kCycMaxLev];
};
// QT: Q of the finest level, QC: of the others
template <typename KT, typename PT, typename QT, typename QC>
__global__ void __launch_bounds__(256) k_cyc_levels(const CycSegs S, const int* depth, const int* sel) {
  int k = 0;
  while (k + 1 < S.n && blockIdx.x >= S.s[k + 1].b0) ++k;
  const CycSeg& G = S.s[k];
  const long long e = (blockIdx.x - G.b0) * 256LL + threadIdx.x;
  if (e >= G.n) return;
  const int g = G.node[e];
  const int4 r = G.nrow[g];
  if (sel && !sel[r.w]) return;
  const double2 si = G.sc[g];
  if (G.lev < 0) {
    const int t = (int)(e - G.ptr[g]);
    const KT* A = (const KT*)G.val;
    const double2 sj = G.sc[G.col[e]];
    QuadSet<KT>::set(G.out, e, si.x * (double)A[r.x + t] * sj.x, si.x * (double)A[r.x + r.z + t] * sj.y,
                     si.y * (double)A[r.y + t] * sj.x, si.y * (double)A[r.y + r.z + t] * sj.y);
    return;
  }
  const int J = G.col[e], own = G.own[e];
  double a[4], p[4] = {0, 0, 0, 0};
  quad_at((const KT*)G.val, e, a);
  if (own >= 0) pq_get((const PT*)G.P + own, p);
  const double iu = si.x > 0 ? 1.0 / si.x : 0.0, iv = si.y > 0 ? 1.0 / si.y : 0.0;
  const double2 sj = depth[r.w] > G.lev + 1 ? G.scc[J] : make_double2(1.0, 1.0);
  const double q0 = (iu * p[0] - si.x * a[0]) * sj.x, q1 = (iu * p[1] - si.x * a[1]) * sj.y;
  const double q2 = (iv * p[2] - si.y * a[2]) * sj.x, q3 = (iv * p[3] - si.y * a[3]) * sj.y;
  if (G.qslot && sizeof(QT) == 8) {  // two blocks of 32 pairs (SliceQuad)
    const int o = G.qslot[e];
    double2* q = reinterpret_cast<double2*>(G.out) + 2 * (long long)(o & ~31) + (o & 31);
    q[0] = make_double2(q0, q1);
    q[32] = make_double2(q2, q3);
  } else if (G.qslot) {
    QuadSet<QT>::set(G.out, G.qslot[e], q0, q1, q2, q3);
  } else {
    QuadSet<QC>::set(G.out, e, q0, q1, q2, q3);
  }
  if (G.lev == 0) QuadSet<QT>::set(G.outT, G.tpos[e], q0, q1, q2, q3);
  else QuadSet<QC>::set(G.outT, G.tpos[e], q0, q1, q2, q3);
}

// ---------------------------------------------------------------------------
// host: structure
// ---------------------------------------------------------------------------

bool cycle_supported(const ua_mesh* m) {
  const Amg* a = m->amg;
  if (!a || !a->sa || a->nlev > kCycMaxLev || a->cyc.failed) return false;
  static thread_local int dev = -1, coop = 0;
  if (dev != m->device) {
    coop = 0;
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, m->device);
    dev = m->device;
  }
  return coop != 0;
}

// Shared memory for a schedule's copies: what its CTAs' rows need, and their solo levels as far as the
// maximum allows; rows that do not fit are left to L1 and L2.
void arena_size(const Cycle& C, const CycSchedule& sch, CycForm form, int most, int small, int& bytes, bool& room) {
  double need = 0, solo = 0;
  for (const int4& ct : sch.cta)
    for (int k = ct.x; k < ct.y; ++k) {
      const int s = sch.queue[k];
      const CycSys& y = C.sys[s];
      need = std::max(need, (C.h_bytes[form][s] + (ct.w == 1 ? C.h_solo[form][s] : 0.0)) / ct.w + 8.0 * y.dn * y.dn);
      if (ct.w > 1) solo = std::max(solo, C.h_solo[form][s] + 8192);
    }
  need = 1.15 * need + 8192;
  room = need <= most;
  bytes = room ? std::max(16384, (int)std::min((double)most, need + solo)) & ~15 : small;
}

// the schedule's block for up to 1024 CTAs
static size_t sched_ints(int nsys) { return 4 + 5 * 1024 + (size_t)nsys + 32 + 32 * 1024; }

// Lists and buffers of the collapsed cycle, once per handle (the node slices of the finest level
// must be there).
int cycle_init(ua_mesh* m) {
  Amg* a = m->amg;
  Cycle& C = a->cyc;
  if (C.ready) return UA_OK;
  if (!cycle_supported(m) || !a->sell.ready) return UA_ERR_INVALID;
  const int nsys = a->nsys, nl = a->nlev;
  bool ok = true;
  C.lev.resize(nl);
  const Sell& SL = a->sell;
  std::vector<int> ipos(std::max(a->lev[0].nn, 1), 0);
  for (int k = 0; k < a->lev[0].nn; ++k) ipos[SL.h_perm[k]] = k;
  C.d_ipos = upload(m, a, ipos, ok);
  C.d_pcol = (int*)dalloc(m, a, sizeof(int) * (size_t)SL.slots, ok);
  C.d_r2 = dalloc(m, a, 2 * sizeof(double) * (size_t)std::max(a->lev[0].nn, 1), ok);
  for (int l = 0; l < nl; ++l) {
    AmgLevel& L = a->lev[l];
    Cycle::Lev& D = C.lev[l];
    D.sc = (double2*)dalloc(m, a, sizeof(double2) * (size_t)std::max(L.nn, 1), ok);
    if (l > 0) D.ncol = upload(m, a, a->h_gcol[l], ok);
    if (l + 1 < nl) {
      // Q: the A P pattern, on the finest level in node slices; Q': by coarse node,
      // the fine nodes (positions) ascending
      const std::vector<int>&ap = a->h_apnp[l], &ac = a->h_apnc[l];
      const int nc = a->lev[l + 1].nn;
      std::vector<int> qc;
      D.nq = (long long)ac.size();
      std::vector<int> tp(nc + 1, 0), tf(ac.size()), tpos(ac.size());
      if (l == 0) {
        std::vector<long long> qo(kSellSlices * (size_t)SL.nsb + 1, 0);
        std::vector<int> qs(ac.size());
        for (int s = 0; s < nsys; ++s) {
          const int n0 = L.node_off[s], n1 = L.node_off[s + 1], c0 = a->lev[1].node_off[s];
          const size_t s0 = kSellSlices * (size_t)SL.h_sys_sb_off[s], s1 = kSellSlices * (size_t)SL.h_sys_sb_off[s + 1];
          for (size_t i = s0; i < s1; ++i) {
            const int k0 = n0 + 32 * (int)(i - s0), k1 = std::min(k0 + 32, n1);
            int wd = 0;
            for (int k = k0; k < k1; ++k) wd = std::max(wd, ap[SL.h_perm[k] + 1] - ap[SL.h_perm[k]]);
            qo[i + 1] = qo[i] + 32LL * wd;
            qc.resize(qo[i + 1], c0);
            for (int k = k0; k < k1; ++k)
              for (int e = ap[SL.h_perm[k]], t = 0; e < ap[SL.h_perm[k] + 1]; ++e, ++t) {
                qs[e] = (int)(qo[i] + 32 * t + (k - k0));
                qc[qs[e]] = ac[e];
              }
          }
        }
        D.nq = qo.back();
        if (D.nq > INT_MAX) ok = false;
        D.qoff = upload(m, a, qo, ok);
        D.qcol = upload(m, a, qc, ok);
        D.qslot = upload(m, a, qs, ok);
      } else {
        D.qcol = L.apn_col;
      }
      for (int J : ac) tp[J + 1]++;
      for (int J = 0; J < nc; ++J) tp[J + 1] += tp[J];
      std::vector<int> nx(tp.begin(), tp.end() - 1);
      for (int k = 0; k < L.nn; ++k) {
        const int g = l == 0 ? SL.h_perm[k] : k;
        for (int e = ap[g]; e < ap[g + 1]; ++e) {
          const int u = nx[ac[e]]++;
          tf[u] = k;
          tpos[e] = u;
        }
      }
      D.tptr = upload(m, a, tp, ok);
      D.tfine = upload(m, a, tf, ok);
      D.tpos = upload(m, a, tpos, ok);
      for (int w = 0; w < CF_COUNT; ++w) {  // bytes a step reads of this level
        const int qe = 4 + (w == CF_FP64 ? 32 : w == CF_LO && l == 0 ? 8 : 16);
        C.h_bytes[w].resize(nsys, 0.0);
        C.h_solo[w].resize(nsys, 0.0);
        for (int s = 0; s < nsys; ++s) {
          const int g0 = L.node_off[s], g1 = L.node_off[s + 1];
          if (g1 == g0) continue;
          double b = 2.0 * (ap[g1] - ap[g0]) * qe;
          if (l == 0)
            b += (double)(SL.h_sl_off[kSellSlices * SL.h_sys_sb_off[s + 1]] - SL.h_sl_off[kSellSlices * SL.h_sys_sb_off[s]]) *
                 (w == CF_FP64 ? 36 : w == CF_LO ? 28 : 20);
          else
            b += (double)(a->h_gptr[l][g1] - a->h_gptr[l][g0]) * (w ? 20 : 36);
          (l > 0 && g1 - g0 <= kSoloNodes ? C.h_solo : C.h_bytes)[w][s] += b + 8.0 * (g1 - g0);
        }
      }
    }
  }
  C.sys.resize(nsys);
  for (int s = 0; s < nsys; ++s) {
    CycSys& S = C.sys[s];
    std::memset(&S, 0, sizeof(S));
    S.depth = S.solo = a->depth[s];
    S.dn = a->h_dn[s];
    S.doff = a->h_doff[s];
    S.sl0 = kSellSlices * a->sell.h_sys_sb_off[s];
    for (int l = 0; l <= S.depth; ++l) {
      S.n0[l] = a->lev[l].node_off[s];
      S.nn[l] = a->lev[l].node_off[s + 1] - S.n0[l];
    }
    S.nsl = (S.nn[0] + 31) / 32;
    for (int b = S.nn[S.depth]; S.solo > 1 && S.nn[S.solo - 1] <= kSoloNodes; --S.solo) {
      b += 2 * S.nn[S.solo - 1];
      if (b > kSoloBuf) break;
    }
  }
  C.d_sys = upload(m, a, C.sys, ok);
  C.nslices = (long long)kSellSlices * a->sell.nsb;
  C.d_part = (double*)dalloc(m, a, sizeof(double) * 3 * (size_t)std::max(C.nslices, 1LL), ok);
  C.d_sched = (int*)dalloc(m, a, sizeof(int) * sched_ints(nsys), ok);
  C.d_prof = (unsigned long long*)dalloc(m, a, sizeof(unsigned long long) * 2 * CP_COUNT, ok);
  if (ok && cudaMallocHost(&C.h_stage, sizeof(int) * sched_ints(nsys)) != cudaSuccess) ok = false;
  if (!ok) {
    C.failed = true;
    return set_error(UA_ERR_OOM, "collapsed cycle: allocation failed");
  }
  if (SL.nsb)
    k_cyc_cols<<<SL.nsb, 256, 0, m->stream>>>(CycFine{SL.perm, SL.sl_off, nullptr}, SL.sb_n0, SL.sb_cnt,
                                              m->dm.nodeptr, m->dm.nodecol, C.d_ipos, C.d_pcol);
  if (cudaGetLastError() != cudaSuccess) {
    C.failed = true;
    return set_error(UA_ERR_CUDA, "collapsed cycle: launch failed");
  }
  // the host lists served their purpose
  for (auto* v : {&a->h_gptr, &a->h_gcol, &a->h_apnp, &a->h_apnc}) std::vector<std::vector<int>>().swap(*v);
  C.ready = true;
  return UA_OK;
}

// Buffers of the values in this precision (before any capture).
int cycle_alloc_values(ua_mesh* m, bool fp32, bool lo) {
  Amg* a = m->amg;
  Cycle& C = a->cyc;
  Sell& S = a->sell;
  bool ok = true;
  auto need = [&](void** p, size_t bytes, bool zero = false) {
    if (*p) return;
    *p = dalloc(m, a, std::max<size_t>(bytes, 32), ok);
    if (*p && zero && cudaMemsetAsync(*p, 0, std::max<size_t>(bytes, 32), m->stream) != cudaSuccess) ok = false;
  };
  const size_t nv = 4 * (size_t)S.slots;
  if (fp32) need((void**)&S.v32, sizeof(float) * nv);
  else need((void**)&S.v64, sizeof(double) * nv);
  if (lo) need((void**)&S.vlo, sizeof(__nv_bfloat16) * nv);
  for (int l = 0; l < a->nlev; ++l) {
    Cycle::Lev& D = C.lev[l];
    // levels 1 .. nlev-2 hold an operator; node entries = dof entries / 4
    if (l > 0 && l + 1 < a->nlev) need(fp32 ? &D.a32 : &D.a64, (fp32 ? 16 : 32) * (size_t)(a->lev[l].nnz / 4));
    if (l + 1 < a->nlev) {
      const bool half = lo && l == 0;
      need(half ? &D.qh : fp32 ? &D.qf : &D.qd, (half ? 8 : fp32 ? 16 : 32) * (size_t)D.nq, l == 0);  // padding slots stay zero
      need(half ? &D.th : fp32 ? &D.tf : &D.td, (half ? 8 : fp32 ? 16 : 32) * (size_t)a->lev[l].nap);
    }
  }
  return ok ? UA_OK : set_error(UA_ERR_OOM, "collapsed cycle: device allocation of the values failed");
}

// Values of the collapsed cycle from the numeric set-up just enqueued (launches only, capturable).
// dw: the finest level's D per node, for the residual norm.
template <typename KT>
static void fill_fine_t(ua_mesh* m, const int* colind0, const KT* K0, bool lo, const int* sel,
                        cudaStream_t st, long long* launches) {
  Amg* a = m->amg;
  Cycle& C = a->cyc;
  Sell& S = a->sell;
  if (!S.nsb) return;
  const CycFine F{S.perm, S.sl_off, C.d_pcol};
  KT* vk = sizeof(KT) == 4 ? (KT*)S.v32 : (KT*)S.v64;
  const int nsl = S.nsb * kSellSlices;
  const int nsub = nsl * (32 / kFillN);
  k_cyc_fill0<KT><<<(nsub + kFillWarps - 1) / kFillWarps, 32 * kFillWarps, 0, st>>>(
      F, nsl, S.sb_n0, S.sb_cnt, S.sb_sys, a->lev[0].d_node_off, a->lev[0].d_dof_off, a->lev[0].nrow, colind0, K0,
      C.lev[0].sc, vk, lo ? S.vlo : nullptr, sel), ++*launches;
}
void cycle_fill_fine(ua_mesh* m, const int* colind0, const void* K0, bool fp32, bool lo,
                     const int* sel, cudaStream_t st, long long* launches) {
  if (fp32) fill_fine_t<float>(m, colind0, (const float*)K0, lo, sel, st, launches);
  else fill_fine_t<double>(m, colind0, (const double*)K0, lo, sel, st, launches);
}

template <typename KT, typename QT>
static void fill_levels_t(ua_mesh* m, CycForm form, const int* sel, cudaStream_t st, long long* launches) {
  using PT = typename PQuadOf<KT>::T;
  constexpr bool f = sizeof(KT) == 4;
  Amg* a = m->amg;
  Cycle& C = a->cyc;
  CycSegs S{};
  long long nb = 0;
  auto add = [&](CycSeg g) {
    if (!g.n) return;
    g.b0 = (int)nb;
    S.s[S.n++] = g;
    nb += (g.n + 255) / 256;
  };
  for (int l = 0; l + 1 < a->nlev; ++l) {
    AmgLevel& L = a->lev[l];
    Cycle::Lev& D = C.lev[l];
    add(CycSeg{0, l, L.nap, L.ap_node, L.apn_col, L.apn_ptr, L.nrow, D.sc, C.lev[l + 1].sc, L.sa_ap,
               f ? L.sa_qh : L.sa_qd, L.ap_p, D.qslot, D.tpos, D.q(form, l), D.t(form, l)});
    if (l > 0)
      add(CycSeg{0, -1, L.ng, a->lev[l - 1].ac_node, D.ncol, L.gptr, L.nrow, D.sc, nullptr, L.A, nullptr, nullptr,
                 nullptr, nullptr, f ? D.a32 : D.a64, nullptr});
  }
  if (nb) k_cyc_levels<KT, PT, QT, KT><<<(unsigned)nb, 256, 0, st>>>(S, a->d_depth, sel), ++*launches;
}
void cycle_fill_levels(ua_mesh* m, bool fp32, bool lo, const int* sel, cudaStream_t st, long long* launches) {
  if (!fp32) fill_levels_t<double, double>(m, CF_FP64, sel, st, launches);
  else if (lo) fill_levels_t<float, __nv_bfloat16>(m, CF_LO, sel, st, launches);
  else fill_levels_t<float, float>(m, CF_FP32, sel, st, launches);
}

// ---------------------------------------------------------------------------
// schedule: CTAs -> teams, systems -> queues
// ---------------------------------------------------------------------------

// Up to half as many systems as CTAs: every system gets a team of its own and the CTAs go, one by
// one, to the team that would finish last.  More systems than that: equal teams, the systems dealt
// out largest first to the team with the least work.  The time of a system on T CTAs is modelled
// as steps x (a + nodes / (b T)): a the passes' latency, b the nodes a CTA streams per microsecond.
void cycle_schedule(const std::vector<CycSys>& sys, const std::vector<int>& sel, const std::vector<int>& steps,
                    int nsm, CycSchedule& out) {
  constexpr double kLatency = 16.0, kNodesPerUs = 90.0;
  constexpr int kSlicesPerCta = 4;  // a team grows while each of its CTAs has at least this many slices
  // up to so many slices one CTA with a slice a warp and no team barrier is as fast or faster (FP64, us a
  // step, one CTA against a team: 8 slices 12.3 and 14.7, 12: 15.1 and 15.0, 16: 17.9 and 16.0)
  constexpr int kOneCta = 12;
  std::vector<int> list;
  for (int s = 0; s < (int)sys.size(); ++s)
    if (sel[s]) list.push_back(s);
  const int n = (int)list.size();
  out.cta.clear();
  out.team.clear();
  out.queue.clear();
  if (!n) return;
  auto time = [&](int s, int T) {
    return std::max(1, steps[s]) * (kLatency + sys[s].nn[0] / (kNodesPerUs * T));
  };
  auto cap = [&](int s) { return sys[s].nsl <= kOneCta ? 1 : std::max(1, std::min(nsm, (sys[s].nsl + kSlicesPerCta - 1) / kSlicesPerCta)); };
  if (2 * n <= nsm) {
    std::vector<int> T(n, 1);
    for (int left = nsm - n; left > 0; --left) {
      int best = -1;
      double tb = -1;
      for (int i = 0; i < n; ++i) {
        const double t = time(list[i], T[i]);
        if (t > tb && T[i] < cap(list[i])) {
          tb = t;
          best = i;
        }
      }
      if (best < 0) break;
      T[best]++;
    }
    for (int i = 0; i < n; ++i) {
      for (int r = 0; r < T[i]; ++r) {
        out.cta.push_back(make_int4(i, i + 1, r, T[i]));
        out.team.push_back(i);
      }
      out.queue.push_back(list[i]);
    }
    return;
  }
  const int T = n <= nsm ? 2 : 4, nt = std::max(1, nsm / T);
  std::sort(list.begin(), list.end(), [&](int p, int q) {
    const double a = time(p, T), b = time(q, T);
    return a != b ? a > b : p < q;
  });
  std::vector<std::vector<int>> q(nt);
  std::vector<double> load(nt, 0.0);
  for (int s : list) {
    const int k = (int)(std::min_element(load.begin(), load.end()) - load.begin());
    q[k].push_back(s);
    load[k] += time(s, T);
  }
  for (int k = 0; k < nt; ++k) {
    const int b = (int)out.queue.size();
    out.queue.insert(out.queue.end(), q[k].begin(), q[k].end());
    for (int r = 0; r < T; ++r) {
      out.cta.push_back(make_int4(b, (int)out.queue.size(), r, T));
      out.team.push_back(k);
    }
  }
}

// Uploads the schedule and clears the team counters (the stream has drained: the pinned staging
// is free).
int upload_schedule(ua_mesh* m, const CycSchedule& s) {
  Cycle& C = m->amg->cyc;
  const int nc = (int)s.cta.size(), nq = (int)s.queue.size();
  if (nc > 1024) return set_error(UA_ERR_INVALID, "resident solve: schedule of %d CTAs", nc);
  C.at_team = 4 + 4 * nc;
  C.at_queue = C.at_team + nc;
  C.at_bar = (C.at_queue + nq + 31) & ~31;
  const int n = C.at_bar + 32 * (s.team.back() + 1);
  std::memset(C.h_stage, 0, sizeof(int) * n);
  std::memcpy(C.h_stage + 4, s.cta.data(), sizeof(int4) * nc);
  std::memcpy(C.h_stage + C.at_team, s.team.data(), sizeof(int) * nc);
  std::memcpy(C.h_stage + C.at_queue, s.queue.data(), sizeof(int) * nq);
  UA_CUDA_TRY(cudaMemcpyAsync(C.d_sched, C.h_stage, sizeof(int) * n, cudaMemcpyHostToDevice, m->stream));
  return UA_OK;
}

CycArgs cycle_args(const ua_mesh* m, CycForm form, bool prof) {
  const Amg* a = m->amg;
  const Cycle& C = a->cyc;
  CycArgs A{};
  for (int l = 0; l + 1 < a->nlev; ++l) {
    const AmgLevel& L = a->lev[l];
    const Cycle::Lev& D = C.lev[l];
    A.lev[l] = CycLev{L.gptr, D.ncol, form == CF_FP64 ? D.a64 : D.a32, l ? L.apn_ptr : nullptr, D.qoff, D.qcol,
                      D.q(form, l), D.tptr, D.tfine, D.t(form, l), L.b, L.x2};
  }
  A.lev[a->nlev - 1].b = a->lev[a->nlev - 1].b;
  A.fine = CycFine{a->sell.perm, a->sell.sl_off, C.d_pcol};
  A.sys = C.d_sys;
  A.dense = a->dense;
  A.cta = (const int4*)(C.d_sched + 4);
  A.team = C.d_sched + C.at_team;
  A.queue = C.d_sched + C.at_queue;
  A.bar = (unsigned*)(C.d_sched + C.at_bar);
  A.err = C.d_sched;
  A.prof = prof ? C.d_prof : nullptr;
  A.part = C.d_part;
  A.nslices = C.nslices;
  A.dbg = m->dm.dbg;
  return A;
}

// ---------------------------------------------------------------------------
// device: PCG
// ---------------------------------------------------------------------------

// Start of a solve, four lanes per node: the particular solution on the constrained dofs (x0 = rhs - X
// there, else zero) into dX and grhs, and the first residual in scaled form, r = D^-1/2 mask(f - K x0).
// The neighbours' x0 are worked out anew from their constraints, so that zeroing dX, the particular
// solution and the residual are one launch; a row's entries of K are read only beside a constrained dof
// that moves.  Bound by the loads' latency: P1 141x71 7.4 us (three launches: 23 us), P2 401x201
// 36 us (60 us).
template <typename KT, typename VT>
__global__ void __launch_bounds__(256) k_cyc_r0(int n, const int4* nrow, const int* node_off, const int* dof_off,
                                                const int* colind, const KT* K, const int* dof_con,
                                                const double* con_rhs, const double* X, const double* f,
                                                const double2* sc, const int* ipos, VT* r, double* dX, double* grhs,
                                                const int* sel) {
  const int g = (blockIdx.x * blockDim.x + threadIdx.x) >> 2, lane = threadIdx.x & 3;
  if (g >= n) return;  // whole groups
  const int4 q = nrow[g];
  if (!sel[q.w]) return;
  const int no = node_off[q.w], nn = node_off[q.w + 1] - no, i0 = dof_off[q.w] + (g - no), i1 = i0 + nn;
  auto x0 = [&](int d) {
    const int c = dof_con[d];
    return c >= 0 ? con_rhs[c] - X[d] : 0.0;
  };
  double a0 = 0, a1 = 0;
  for (int k = lane; k < q.z; k += 4) {
    const int j = colind[q.x + k];
    const double xu = x0(j), xv = x0(j + nn);
    if (xu != 0) {
      a0 += (double)K[q.x + k] * xu;
      a1 += (double)K[q.y + k] * xu;
    }
    if (xv != 0) {
      a0 += (double)K[q.x + q.z + k] * xv;
      a1 += (double)K[q.y + q.z + k] * xv;
    }
  }
  const unsigned gmask = 0xfu << (threadIdx.x & 28);
#pragma unroll
  for (int o = 2; o > 0; o >>= 1) {
    a0 += __shfl_xor_sync(gmask, a0, o, 4);
    a1 += __shfl_xor_sync(gmask, a1, o, 4);
  }
  if (lane < 2) {
    const int i = lane ? i1 : i0, c = dof_con[i];
    const double x = c >= 0 ? con_rhs[c] - X[i] : 0.0;
    dX[i] = x;
    if (c >= 0) grhs[c] = x;
    const double2 d = sc[g];
    const double w = lane ? d.y : d.x;
    r[2 * (size_t)ipos[g] + lane] = (VT)(w > 0 ? w * (f[i] - (lane ? a1 : a0)) : 0.0);
  }
}

#define UA_TEAM_SYNC(t)                                               \
  do {                                                                \
    if (!team_sync(t)) {                                              \
      if (threadIdx.x == 0) *a.cyc.err = 1;                           \
      return;                                                         \
    }                                                                 \
  } while (0)

struct PcgArgs {
  CycArgs cyc;
  const void *kv, *lv;       // finest level: PCG operator, V-cycle operator (scaled, node slices)
  void *r, *r2, *z, *p, *q;  // pairs per node in slice order (VT)
  double2* x;                // FP64 pairs
  const void* dw;            // D per node in slice order (VT pairs): |r|^2 = sum D r^2
  const double2* sc;
  double* dX;
  const int* dof_off;
  double* sysv_tol2;         // [nsys] squared relative tolerance
  int *done, *its, *status;
  int maxit;
  int arena;                 // dynamic shared memory for copies of the matrices
  bool room;                 // it holds every system's rows (solo levels apart)
};

// The whole PCG of the systems in the team's queue.  The passes of a step, a team barrier after
// each:  the levels down (but the finest), the dense level (by every CTA for itself, no barrier),
// the levels up, the finest up pass with the partials of r.z, the operator pass (p and q are
// updated in it: q = A z + beta q, partials p.q), and the vector update together with the finest
// restriction, which forms r - alpha q as it gathers (the new residual goes to a second buffer).
// All scalars are computed by every CTA from the per-slice partials, so nothing but vectors and
// partials crosses CTAs.
// 512 threads of up to 128 registers, one CTA per SM: few warps, each with up to ten slots of its
// slice in flight (1024 threads at 64 registers spilled 800 bytes a thread).
// QT, QC: Q of the finest level and of the coarse ones.
template <typename KT, typename LT, typename VT, typename QT, typename QC>
__global__ void __launch_bounds__(kCycThreads, 1) k_pcg_team(const PcgArgs a) {
  static_assert(sizeof(QT) >= sizeof(LT) && sizeof(QC) >= sizeof(KT),
                "Q holds the smoothing of its level's operator and is no narrower than it");
  using V2 = typename Vec2<VT>::T;
  extern __shared__ __align__(16) char arena_mem[];
  __shared__ CycSys S;
  __shared__ LevS lev[kCycMaxLev];
  __shared__ FineS fine;
  __shared__ double red[3][32];
  __shared__ DenseSh dsh;
  __shared__ V2 zcs[kAmgMaxDense / 2], sbuf[kSoloBuf];
  __shared__ int ok;
  const int4 c = a.cyc.cta[blockIdx.x];
  TeamCtx t{c.z, c.w, a.cyc.bar + 32 * a.cyc.team[blockIdx.x], 0u, &ok, a.cyc.dbg};
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  V2 *z = (V2*)a.z, *p = (V2*)a.p, *q = (V2*)a.q;
  const V2* dw = (const V2*)a.dw;
  double *part_pq = a.cyc.part, *part_rz = part_pq + a.cyc.nslices, *part_rr = part_rz + a.cyc.nslices;
  const bool clk = a.cyc.prof && t.rank == 0 && threadIdx.x == 0;
  unsigned long long tick = clk ? cyc_now() : 0;
  auto mark = [&](int cls) {
    if (!clk) return;
    const unsigned long long now = cyc_now();
    atomicAdd(a.cyc.prof + 2 * cls, (now - tick) * (unsigned long long)t.size);
    atomicAdd(a.cyc.prof + 2 * cls + 1, 1ULL);
    tick = now;
  };
  for (int qi = c.x; qi < c.y; ++qi) {
    const int s = a.cyc.queue[qi];
    __syncthreads();  // the shared tables of the previous system are no longer read
    if (threadIdx.x < (int)(sizeof(CycSys) / sizeof(int)))
      reinterpret_cast<int*>(&S)[threadIdx.x] = reinterpret_cast<const int*>(a.cyc.sys + s)[threadIdx.x];
    __syncthreads();
    Arena ar{arena_mem, a.arena, 0};
    const double* dense;
    int lo, hi;
    team_share(t, S.nsl, lo, hi);
    cyc_stage<KT, LT, QT, QC>(a.cyc, a.kv, a.lv, S, t, lo, hi, ar, lev, &fine, 4 * sizeof(KT), dense, a.room);
    const int n0 = S.n0[0], nn = S.nn[0], dep = S.depth, solo = t.size > 1 ? S.solo : dep;
    const bool stream = fine.cols == a.cyc.fine.cols;  // rows read from global memory
    // restrict the updated residual after one more barrier, or b - alpha q from the two old vectors:
    // the second gather costs more than the barrier once a CTA has kSplitSlices slices
    const bool same = a.kv == a.lv;  // the cycle reads the method's operator
    const bool split = S.nsl >= kSplitSlices * t.size;
    const V2* bL = (const V2*)a.cyc.lev[dep].b;
    V2 *r = (V2*)a.r, *rn = (V2*)a.r2;
    for (int i = lo + warp; i < hi; i += kCycWarps) {
      double v = 0;
      if (32 * i + lane < nn) {
        const V2 rv = r[n0 + 32 * i + lane], d = dw[n0 + 32 * i + lane];
        v = (double)d.x * ((double)rv.x * (double)rv.x) + (double)d.y * ((double)rv.y * (double)rv.y);
      }
      v = lane_sum(v, 32);
      if (lane == 0) part_rr[S.sl0 + i] = v;
    }
    cyc_down<VT, QT>(lev[0], S, 0, t, r, (V2*)a.cyc.lev[1].b);
    UA_TEAM_SYNC(t);
    const double rr0 = team_sum(part_rr + S.sl0, S.nsl, red[2]);
    const double stop = a.sysv_tol2[s] * rr0;
    int its = 0, status = 0;
    double rz_old = 0;
    mark(CP_OTHER);
    while (rr0 != 0.0) {
      const bool odd = its & 1;
      // z = cycle(r), the finest restriction done
      for (int l = 1; l < solo; ++l) {
        cyc_down<VT, QC>(lev[l], S, l, t, (const V2*)a.cyc.lev[l].b, (V2*)a.cyc.lev[l + 1].b);
        UA_TEAM_SYNC(t);
      }
      const V2* zc = zcs - S.n0[dep];
      if (solo < dep) zc = cyc_solo<VT, KT, QC>(lev, S, a.cyc, dense, dsh, zcs, sbuf);
      else cyc_dense<VT>(S, dense, bL, dsh, zcs);
      for (int l = solo - 1; l > 0; --l) {
        cyc_up<VT, KT, QC>(lev[l], S, l, t, (const V2*)a.cyc.lev[l].b, (V2*)a.cyc.lev[l].z, zc);
        UA_TEAM_SYNC(t);
        zc = (const V2*)a.cyc.lev[l].z;
      }
      mark(CP_OTHER);
      for_slices(lo, hi, n0, nn, !same && odd, [&](int i, int g, bool in, int nx) {
        if (stream && lane == 0 && nx >= lo && nx < hi) {
          slice_prefetch<LT>(a.cyc.fine.sl_off, a.cyc.fine.cols, a.lv, S.sl0 + nx);
          slice_prefetch<QT>(a.cyc.lev[0].qoff, a.cyc.lev[0].qcol, a.cyc.lev[0].qval, S.sl0 + nx);
        }
        double v = 0;
        if (in) {
          const V2 bv = r[g];
          double z0, z1;
          cyc_up0_node<LT, VT, QT>(fine, lev[0], S, t, S.sl0 + i, lane, r, zc, 1.0, z0, z1);
          V2 o;
          o.x = (VT)(2.0 * (double)bv.x + z0);
          o.y = (VT)(2.0 * (double)bv.y + z1);
          z[g] = o;
          v = (double)bv.x * (double)o.x + (double)bv.y * (double)o.y;
        }
        v = lane_sum(v, 32);
        if (lane == 0) part_rz[S.sl0 + i] = v;
      });
      UA_TEAM_SYNC(t);
      const double rz = team_sum(part_rz + S.sl0, S.nsl, red[0]);
      mark(CP_UP0);
      const double beta = its ? rz / rz_old : 0.0;
      rz_old = rz;
      // p = z + beta p, q = A z + beta q, partials p.q
      for_slices(lo, hi, n0, nn, same || odd, [&](int i, int g, bool in, int nx) {
        if (stream && lane == 0 && nx >= lo && nx < hi) slice_prefetch<KT>(a.cyc.fine.sl_off, a.cyc.fine.cols, a.kv, S.sl0 + nx);
        double v = 0;
        if (in) {
          V2 pn = z[g], po, qo;
          if (its) {
            po = p[g];
            qo = q[g];
          }
          double a0, a1;
          slice_product<KT, VT>(fine.sl_off, fine.cols, fine.kv, S.sl0 + i, lane, z, UA_COL_RANGE(t.dbg, n0, nn), a0, a1);
          if (its) {
            pn.x = (VT)((double)pn.x + beta * (double)po.x);
            pn.y = (VT)((double)pn.y + beta * (double)po.y);
            a0 += beta * (double)qo.x;
            a1 += beta * (double)qo.y;
          }
          V2 qn;
          qn.x = (VT)a0;
          qn.y = (VT)a1;
          p[g] = pn;
          q[g] = qn;
          v = (double)pn.x * (double)qn.x + (double)pn.y * (double)qn.y;
        }
        v = lane_sum(v, 32);
        if (lane == 0) part_pq[S.sl0 + i] = v;
      });
      UA_TEAM_SYNC(t);
      const double pq = team_sum(part_pq + S.sl0, S.nsl, red[1]);
      mark(CP_SPMV);
      if (!(pq > 0)) {  // not positive definite on the free dofs, or breakdown
        status = 1;
        break;
      }
      const double alpha = rz / pq;
      // x += alpha p, r -= alpha q, partials |r|^2, and the restriction of the new residual
      for (int i = lo + warp; i < hi; i += kCycWarps) {
        double v = 0;
        const int g = n0 + 32 * i + lane;
        if (32 * i + lane < nn) {
          const V2 pv = p[g], qv = q[g], d = dw[g];
          V2 rv = r[g];
          double2 xv = its ? a.x[g] : make_double2(0.0, 0.0);
          xv.x += alpha * (double)pv.x;
          xv.y += alpha * (double)pv.y;
          rv.x = (VT)((double)rv.x - alpha * (double)qv.x);
          rv.y = (VT)((double)rv.y - alpha * (double)qv.y);
          a.x[g] = xv;
          rn[g] = rv;
          v = (double)d.x * ((double)rv.x * (double)rv.x) + (double)d.y * ((double)rv.y * (double)rv.y);
        }
        v = lane_sum(v, 32);
        if (lane == 0) part_rr[S.sl0 + i] = v;
      }
      if (split) {
        UA_TEAM_SYNC(t);
        cyc_down<VT, QT>(lev[0], S, 0, t, rn, (V2*)a.cyc.lev[1].b, nullptr, 0.0, 1.0, odd);
      } else {
        cyc_down<VT, QT>(lev[0], S, 0, t, r, (V2*)a.cyc.lev[1].b, q, alpha, 1.0, odd);
      }
      ++its;
      UA_TEAM_SYNC(t);
      const double rr = team_sum(part_rr + S.sl0, S.nsl, red[2]);
      mark(CP_DOWN0);
      V2* sw = r;
      r = rn;
      rn = sw;
      if (rr <= stop || its >= a.maxit || !(rr == rr)) break;
    }
    // dX += D^-1/2 x on the CTA's nodes (x written by this CTA)
    if (its)
      for (int i = 32 * lo + threadIdx.x; i < min(32 * hi, nn); i += kCycThreads) {
        const int g = a.cyc.fine.perm[n0 + i], j = a.dof_off[s] + (g - n0);
        const double2 xv = a.x[n0 + i], d = a.sc[g];
        if (d.x > 0) a.dX[j] += d.x * xv.x;
        if (d.y > 0) a.dX[j + nn] += d.y * xv.y;
      }
    if (t.rank == 0 && threadIdx.x == 0) {
      a.its[s] = its;
      a.status[s] = status;
      a.done[s] = 1;
    }
  }
}

template <typename KT, typename LT, typename VT, typename QT, typename QC>
static int launch_pcg(ua_mesh* m, const PcgArgs& a, int nctas) {
  UA_CUDA_TRY(cudaFuncSetAttribute(k_pcg_team<KT, LT, VT, QT, QC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   kCycArena));
  return launch_team(m, k_pcg_team<KT, LT, VT, QT, QC>, a, nctas, a.arena);
}

int pcg_resident(ua_mesh* m, const PcgSolve& v, const std::vector<int>& sel, const std::vector<int>& steps, int nsm,
                 long long* launches) {
  Amg* a = m->amg;
  Cycle& C = a->cyc;
  CycSchedule sch;
  cycle_schedule(C.sys, sel, steps, std::min(nsm, 1024), sch);
  if (sch.cta.empty()) return UA_OK;
  if (int rc = upload_schedule(m, sch)) return rc;
  if (v.prof) UA_CUDA_TRY(cudaMemsetAsync(C.d_prof, 0, sizeof(unsigned long long) * 2 * CP_COUNT, m->stream));
  const Sell& S = a->sell;
  PcgArgs A{};
  const CycForm form = cyc_form(v.fp32, v.lo);
  A.cyc = cycle_args(m, form, v.prof);
  A.kv = v.fp32 ? (const void*)S.v32 : (const void*)S.v64;
  A.lv = v.fp32 ? (v.lo ? (const void*)S.vlo : (const void*)S.v32) : (const void*)S.v64;
  A.r = v.r;
  A.r2 = C.d_r2;
  // shared memory for the copies: all of it where the largest share of a CTA fits, else what the
  // small levels take (the rest serves as L1 for the streamed rows)
  arena_size(C, sch, form, kCycArena, kCycArenaSmall, A.arena, A.room);
  A.z = v.z;
  A.p = v.p;
  A.q = v.q;
  A.x = (double2*)v.x;
  A.dw = v.dw;
  A.sc = C.lev[0].sc;
  A.dX = v.dX;
  A.dof_off = a->lev[0].d_dof_off;
  A.sysv_tol2 = v.tol2;
  A.done = v.done;
  A.its = v.its;
  A.status = v.status;
  A.maxit = v.maxit;
  const AmgLevel& L0 = a->lev[0];
  const int nb = std::max(1, (L0.nn + 63) / 64);
  if (v.fp32)
    k_cyc_r0<float, float><<<nb, 256, 0, m->stream>>>(L0.nn, L0.nrow, L0.d_node_off, L0.d_dof_off, v.colind,
                                                      (const float*)v.K, v.dof_con, v.con_rhs, v.X, v.f, C.lev[0].sc,
                                                      C.d_ipos, (float*)v.r, v.dX, v.grhs, v.sel);
  else
    k_cyc_r0<double, double><<<nb, 256, 0, m->stream>>>(L0.nn, L0.nrow, L0.d_node_off, L0.d_dof_off, v.colind,
                                                        (const double*)v.K, v.dof_con, v.con_rhs, v.X, v.f,
                                                        C.lev[0].sc, C.d_ipos, (double*)v.r, v.dX, v.grhs, v.sel);
  ++*launches;
  UA_CUDA_TRY(cudaGetLastError());
  const int nc = C.last_grid = (int)sch.cta.size();
  int rc;
  if (!v.fp32) rc = launch_pcg<double, double, double, double, double>(m, A, nc);
  else if (v.lo) rc = launch_pcg<float, __nv_bfloat16, float, __nv_bfloat16, float>(m, A, nc);
  else rc = launch_pcg<float, float, float, float, float>(m, A, nc);
  ++*launches;
  return rc;
}

#ifdef UA_BOUNDS_CHECK
// Two CTAs' barrier, met by as many as are launched, with a wait of some microseconds.
__global__ void k_team_probe(unsigned* bar, int* err) {
  __shared__ int ok;
  TeamCtx t{(int)blockIdx.x, 2, bar, 0u, &ok, nullptr};
  if (!team_sync<4096>(t, []() {}) && threadIdx.x == 0) *err = 1;
}
#endif

const int* resident_error_flag(const ua_mesh* m) { return m->amg->cyc.d_sched; }

int resident_error(int flag) {
  return flag ? set_error(UA_ERR_TIMEOUT, "resident solve: a team barrier was not met") : UA_OK;
}

// After the solve's stream has drained: whether every barrier was met, and the pass times (ms of
// the whole grid) and counts of a profiled solve.
int pcg_resident_status(ua_mesh* m, bool prof, double* ms, int* cnt) {
  Cycle& C = m->amg->cyc;
  int err = 0;
  UA_CUDA_TRY(dev_read(m, &err, C.d_sched, sizeof(int)));
  if (int rc = resident_error(err)) return rc;
  if (prof) {
    unsigned long long h[2 * CP_COUNT];
    UA_CUDA_TRY(dev_read(m, h, C.d_prof, sizeof(h)));
    for (int k = 0; k < CP_COUNT; ++k) {
      ms[k] += 1e-6 * (double)h[2 * k] / std::max(C.last_grid, 1);
      cnt[k] += (int)h[2 * k + 1];
    }
  }
  return UA_OK;
}

}  // namespace ua

extern "C" int ua_debug_team_wait(const ua_mesh* m, int32_t ctas) {
  using namespace ua;
  if (!m || ctas < 1 || ctas > 2) return set_error(UA_ERR_INVALID, "ua_debug_team_wait: bad argument");
#ifdef UA_BOUNDS_CHECK
  UA_CUDA_TRY(cudaSetDevice(m->device));
  int* d = nullptr;  // flag, barrier counter
  UA_CUDA_TRY(cudaMalloc(&d, 2 * sizeof(int)));
  int flag = 0;
  cudaError_t e = dev_clear(m, d, 2 * sizeof(int));
  unsigned* bar = (unsigned*)d + 1;
  void* args[] = {&bar, &d};
  if (e == cudaSuccess)
    e = cudaLaunchCooperativeKernel((const void*)k_team_probe, dim3(ctas), dim3(kCycThreads), args, 0, m->stream);
  if (e == cudaSuccess) e = dev_read(m, &flag, d, sizeof(int));
  cudaFree(d);
  UA_CUDA_TRY(e);
  return resident_error(flag);
#else
  return set_error(UA_ERR_INVALID, "ua_debug_team_wait: in the debug build only");
#endif
}
