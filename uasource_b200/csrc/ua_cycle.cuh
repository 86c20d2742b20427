// The V-cycle in collapsed form and the team primitives of the resident Krylov kernels.
//
// With one damped l1-Jacobi sweep before and after the coarse correction, a V(1,1) cycle from a
// zero guess is the sum
//     z = M b + P~ z_c,   z_c = cycle(P~' b),   M = 2 D^-1 - D^-1 A D^-1,   P~ = (I - D^-1 A) P
// (D the damped l1 diagonal): the pre-smoothed residual and the post-smoothing of the correction
// are folded into the transfer P~, whose entries the set-up has at hand (A P is formed for the
// coarse operator).  Scaled by D^1/2 on every level but a system's coarsest,
//     A^ = D^-1/2 A D^-1/2,  Q = D^1/2 P~ D_c^-1/2,  b^ = D^-1/2 b,  z^ = D^1/2 z,
// one level is  b^_c = Q' b^  on the way down and  z^ = 2 b^ - A^ b^ + Q z^_c  on the way up, one
// pass each, where the uncollapsed cycle makes a residual, a restriction, a prolongation and a
// smoothing pass in sequence.  The scaled operator has no diagonal, mask or weight to read.
//
// Teams.  A resident kernel runs one CTA of kCycThreads threads per SM.  The CTAs are split into
// teams; a team solves the systems of its queue one after another, its CTAs meeting at a counter
// in global memory after every pass (a __syncthreads for a team of one).  A system's sums have a
// fixed order that depends on the system alone (per-slice partials, summed by every CTA of the
// team), so its result does not depend on its team's size or on the other systems.
#pragma once
#include "ua_amg_int.h"

namespace ua {

constexpr int kCycThreads = 512;
constexpr int kCycWarps = kCycThreads / 32;

template <typename VT> struct Vec2;
template <> struct Vec2<float> { using T = float2; };
template <> struct Vec2<double> { using T = double2; };

// a quad as loaded, widened only at its use (registers)
template <typename KT> struct QuadRaw;
template <> struct QuadRaw<float> {
  using T = float4;
  static __device__ __forceinline__ T load(const char* p) { return *reinterpret_cast<const float4*>(p); }
  static __device__ __forceinline__ void get(const T& e, double (&q)[4]) { q[0] = e.x; q[1] = e.y; q[2] = e.z; q[3] = e.w; }
};
template <> struct QuadRaw<double> {
  struct T { double2 a, b; };
  static __device__ __forceinline__ T load(const char* p) {
    return T{reinterpret_cast<const double2*>(p)[0], reinterpret_cast<const double2*>(p)[1]};
  }
  static __device__ __forceinline__ void get(const T& e, double (&q)[4]) { q[0] = e.a.x; q[1] = e.a.y; q[2] = e.b.x; q[3] = e.b.y; }
};
template <> struct QuadRaw<__nv_bfloat16> {
  using T = uint2;
  static __device__ __forceinline__ T load(const char* p) { return *reinterpret_cast<const uint2*>(p); }
  static __device__ __forceinline__ void get(const T& e, double (&q)[4]) {
    q[0] = __uint_as_float(e.x << 16); q[1] = __uint_as_float(e.x & 0xffff0000u);
    q[2] = __uint_as_float(e.y << 16); q[3] = __uint_as_float(e.y & 0xffff0000u);
  }
};

// The quad of a lane in a slice's slot block (32 quads): FP64 quads are kept as two blocks of 32
// pairs, so that a warp's 16-byte loads are contiguous.
template <typename KT> struct SliceQuad {
  static __device__ __forceinline__ typename QuadRaw<KT>::T load(const char* blk, int lane) {
    return QuadRaw<KT>::load(blk + lane * (4 * sizeof(KT)));
  }
};
template <> struct SliceQuad<double> {
  static __device__ __forceinline__ QuadRaw<double>::T load(const char* blk, int lane) {
    return QuadRaw<double>::T{reinterpret_cast<const double2*>(blk)[lane], reinterpret_cast<const double2*>(blk + 512)[lane]};
  }
};

struct TeamCtx {
  int rank, size;        // this CTA in its team
  unsigned* bar;         // the team's arrival counter
  unsigned target;       // arrivals that end the next barrier
  int* ok;               // shared: the last barrier was met
  unsigned long long* dbg;  // bounds-checked build
};

// Arrive and wait.  The wait is bounded (some seconds): a team that does not meet returns false in
// every thread and the kernel ends with an error status.
constexpr unsigned kTeamSpinLimit = 1u << 24;
// f: run by one thread of another warp meanwhile.
template <unsigned LIMIT = kTeamSpinLimit, typename F>
__device__ __forceinline__ bool team_sync(TeamCtx& t, F f) {
  __syncthreads();
  if (threadIdx.x == 32) f();
  if (t.size == 1) {
    __syncthreads();
    return true;
  }
  if (threadIdx.x == 0) {
    t.target += t.size;
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(t.bar) : "memory");
    int ok = 0;
    for (unsigned i = 0; i < LIMIT; ++i) {
      unsigned v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(t.bar) : "memory");
      if ((int)(v - t.target) >= 0) {
        ok = 1;
        break;
      }
    }
    *t.ok = ok;
  }
  __syncthreads();
  return *t.ok != 0;
}
__device__ __forceinline__ bool team_sync(TeamCtx& t) {
  if (t.size == 1) {
    __syncthreads();
    return true;
  }
  return team_sync(t, []() {});
}

// Sum of n partials by the whole CTA, the same bits in every thread of every CTA: thread t adds
// the partials t, t + kCycThreads, ..., then a butterfly.  red: kCycWarps shared doubles that no
// thread of the CTA still reads.
__device__ __forceinline__ double team_sum(const double* part, int n, double* red) {
  double a = 0;
  for (int i = threadIdx.x; i < n; i += kCycThreads) a += __ldcg(part + i);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = a;
  __syncthreads();
  a = (threadIdx.x & 31) < kCycWarps ? red[threadIdx.x & 31] : 0.0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
  return a;
}

__device__ __forceinline__ double lane_sum(double v, int width) {
  for (int o = width >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// this CTA's share [lo, hi) of n items
__device__ __forceinline__ void team_share(const TeamCtx& t, int n, int& lo, int& hi) {
  lo = (int)((long long)n * t.rank / t.size);
  hi = (int)((long long)n * (t.rank + 1) / t.size);
}

// Lanes per node.  A row's entries are dealt to kDownW (restriction) or kUpW (coarse up pass) virtual
// lanes, each summed in order, the lanes' sums added by a butterfly: an order that does not depend on
// how many physical lanes work on it.  A CTA with few nodes takes one lane per virtual lane (a pass is
// then one round of dependent loads); one with more nodes than that fills gives every lane four of
// them, which keeps four times the nodes in flight (a warp per coarse node: 33 rounds of 1900 cycles
// for the 528 coarse nodes of a 4,753-node mesh on one CTA).
constexpr int kDownW = 32, kUpW = 8;

// What the passes read of one level and of the finest level's operator: global memory, or the
// copies of this CTA's rows in shared memory (cyc_stage).  Row pointers and entry numbers are the
// global ones in both, the bases are shifted.  The loads are generic on purpose.
struct LevS {
  const int *aptr, *acol;
  const char* aval;
  const int* qptr;        // rows of Q (levels >= 1)
  const long long* qoff;  // slices of Q (finest level)
  const int* qcol;
  const char* qval;
  const int *tptr, *tfine;
  const char* tval;
};
struct FineS {
  const long long* sl_off;
  const int* cols;
  const char *kv, *lv;  // operator of the Krylov method and of the cycle
};

// Shared memory left for copies.
struct Arena {
  char* base;
  int cap, used;
  __device__ __forceinline__ char* take(long long bytes) {  // uniform over the CTA
    const long long b = (bytes + 15) & ~15LL;
    if (used + b > cap) return nullptr;
    char* p = base + used;
    used += (int)b;
    return p;
  }
};
// Copies of global memory into the arena, asynchronous so that a stage waits once for all of them
// (stage_wait); in the widest pieces the addresses allow.
__device__ __forceinline__ void copy_in(void* d, const void* s, long long bytes) {
  const unsigned sd = (unsigned)__cvta_generic_to_shared(d);
  const char* p = (const char*)s;
  const unsigned long long al = (unsigned long long)p | (unsigned long long)sd | (unsigned long long)bytes;
  if (!(al & 15))
    for (long long i = 16LL * threadIdx.x; i < bytes; i += 16 * kCycThreads)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sd + (unsigned)i), "l"(p + i) : "memory");
  else if (!(al & 7))
    for (long long i = 8LL * threadIdx.x; i < bytes; i += 8 * kCycThreads)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(sd + (unsigned)i), "l"(p + i) : "memory");
  else
    for (long long i = 4LL * threadIdx.x; i < bytes; i += 4 * kCycThreads)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(sd + (unsigned)i), "l"(p + i) : "memory");
}
__device__ __forceinline__ void stage_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// rows [lo, hi) of a node-CSR matrix with quads of qb bytes
__device__ __forceinline__ void stage_csr(Arena& ar, int lo, int hi, int qb, const int*& ptr, const int*& col,
                                          const char*& val) {
  if (lo >= hi) return;
  const int e0 = ptr[lo], e1 = ptr[hi];
  char* p = ar.take((long long)(hi - lo + 1) * 4 + 12 + (long long)(e1 - e0) * (4 + qb) + 16);
  if (!p) return;
  char* pv = p;  // values first (16-byte aligned), then columns, then row pointers
  int* pc = reinterpret_cast<int*>(p + (((long long)(e1 - e0) * qb + 15) & ~15LL));
  int* pp = pc + (e1 - e0);
  copy_in(pv, val + (long long)e0 * qb, (long long)(e1 - e0) * qb);
  copy_in(pc, col + e0, 4LL * (e1 - e0));
  copy_in(pp, ptr + lo, 4LL * (hi - lo + 1));
  ptr = pp - lo;
  col = pc - e0;
  val = pv - (long long)e0 * qb;
}

// slices [lo, hi) of a sliced matrix with quads of qb bytes
__device__ __forceinline__ void stage_slices(Arena& ar, int lo, int hi, int qb, const long long*& off,
                                             const int*& col, const char*& val) {
  if (lo >= hi) return;
  const long long e0 = off[lo], ne = off[hi] - e0;
  char* p = ar.take(8LL * (hi - lo + 2) + ne * (4 + qb));
  if (!p) return;
  long long* po = reinterpret_cast<long long*>(p);
  char* pv = p + ((8LL * (hi - lo + 1) + 15) & ~15LL);  // slots come in blocks of 32: 16-byte aligned
  int* pc = reinterpret_cast<int*>(pv + ne * qb);
  copy_in(po, off + lo, 8LL * (hi - lo + 1));
  copy_in(pv, val + e0 * qb, ne * qb);
  copy_in(pc, col + e0, 4 * ne);
  off = po - lo;
  col = pc - e0;
  val = pv - e0 * qb;
}

// Reads the level tables into shared memory and copies this CTA's rows as far as they fit, the
// small levels first.  In a team with enough CTAs everything fits: a pass then waits for one
// gather of the vector instead of three dependent loads.  [slo, shi): the CTA's slices of the finest
// level (the passes of that level visit no others).  Every thread keeps the same pointers;
// thread 0 publishes them.  room: the arena holds everything but, perhaps, the solo levels.
// QT, QC: Q of the finest level and of the coarse ones.
template <typename KT, typename LT, typename QT, typename QC>
__device__ __forceinline__ void cyc_stage(const CycArgs& A, const void* kv, const void* lv, const CycSys& S,
                                          const TeamCtx& t, int slo, int shi, Arena& ar, LevS* lev, FineS* fine, int kslot,
                                          const double*& dense, bool room) {
  constexpr int q0 = 4 * sizeof(QT), qb = 4 * sizeof(QC), ab = 4 * sizeof(KT);
  int lo, hi;
  dense = A.dense + S.doff;
  if (char* p = ar.take(8LL * S.dn * S.dn)) {
    copy_in(p, dense, 8LL * S.dn * S.dn);
    dense = (const double*)p;
  }
  // the solo levels whole: ahead of the rest where the finest rows stay in global memory, else with
  // what room is left
  const int solo = t.size > 1 ? S.solo : S.depth;
  auto stage_solo = [&]() {
    for (int l = S.depth - 1; l >= solo; --l) {
      const CycLev& G = A.lev[l];
      LevS L{G.aptr, G.acol, (const char*)G.aval, G.qptr, G.qoff, G.qcol, (const char*)G.qval,
             G.tptr, G.tfine, (const char*)G.tval};
      stage_csr(ar, S.n0[l + 1], S.n0[l + 1] + S.nn[l + 1], qb, L.tptr, L.tfine, L.tval);
      stage_csr(ar, S.n0[l], S.n0[l] + S.nn[l], qb, L.qptr, L.qcol, L.qval);
      stage_csr(ar, S.n0[l], S.n0[l] + S.nn[l], ab, L.aptr, L.acol, L.aval);
      if (threadIdx.x == 0) lev[l] = L;
    }
  };
  if (!room) stage_solo();
  for (int l = solo - 1; l >= 0; --l) {
    const CycLev& G = A.lev[l];
    LevS L{G.aptr, G.acol, (const char*)G.aval, G.qptr, G.qoff, G.qcol, (const char*)G.qval,
           G.tptr, G.tfine, (const char*)G.tval};
    team_share(t, S.nn[l + 1], lo, hi);
    stage_csr(ar, S.n0[l + 1] + lo, S.n0[l + 1] + hi, l ? qb : q0, L.tptr, L.tfine, L.tval);
    if (l > 0) {
      team_share(t, S.nn[l], lo, hi);
      stage_csr(ar, S.n0[l] + lo, S.n0[l] + hi, qb, L.qptr, L.qcol, L.qval);
      stage_csr(ar, S.n0[l] + lo, S.n0[l] + hi, ab, L.aptr, L.acol, L.aval);
    } else {
      stage_slices(ar, S.sl0 + slo, S.sl0 + shi, q0, L.qoff, L.qcol, L.qval);
    }
    if (threadIdx.x == 0) lev[l] = L;
  }
  FineS F{A.fine.sl_off, A.fine.cols, (const char*)kv, (const char*)lv};
  lo = slo;
  hi = shi;
  if (lo < hi) {
    const int s0 = S.sl0 + lo, ns = hi - lo;
    const long long e0 = F.sl_off[s0], ne = F.sl_off[S.sl0 + hi] - e0;
    if (char* p = ar.take(ne * 4 + 8LL * (ns + 1))) {
      long long* po = reinterpret_cast<long long*>(p);
      int* pc = reinterpret_cast<int*>(po + ns + 1);
      copy_in(po, F.sl_off + s0, 8LL * (ns + 1));
      copy_in(pc, F.cols + e0, 4 * ne);
      F.sl_off = po - s0;
      F.cols = pc - e0;
      const int lb = 4 * sizeof(LT);
      if (char* q = ar.take(ne * lb)) {
        copy_in(q, F.lv + e0 * lb, ne * lb);
        const bool same = F.kv == F.lv;
        F.lv = q - e0 * lb;
        if (same) F.kv = F.lv;
      }
      if (kv != lv)
        if (char* q = ar.take(ne * kslot)) {
          copy_in(q, F.kv + e0 * kslot, ne * kslot);
          F.kv = q - e0 * kslot;
        }
    }
  }
  if (room) stage_solo();
  if (threadIdx.x == 0) *fine = F;
  stage_wait();
  __syncthreads();
}

// KC entries of each of a lane's NV virtual lanes from entry e on: their columns and values load
// together, then the vector's pairs get(column).  Entries past the row's end repeat its last one with a
// zero vector pair.
template <int W, int NV, int KC, bool TR, typename QT, typename G>
__device__ __forceinline__ void row_chunk(const int* col, const char* val, int e, int ee, int lane, double sign, G get,
                                          ColRange range, double (&a0)[NV], double (&a1)[NV]) {
  using V2 = decltype(get(0));
  constexpr int qb = 4 * sizeof(QT), CH = NV * KC;
  int c[CH];
  typename QuadRaw<QT>::T m[CH];
#pragma unroll
  for (int k = 0; k < CH; ++k) {
    const int u = min(e + W * (k / NV) + (W / NV) * (k % NV) + lane, ee - 1);
    c[k] = col[u];
    UA_CHECK_COL(range, c[k], BS_ROW_COL);
    m[k] = QuadRaw<QT>::load(val + (long long)u * qb);
  }
  V2 x[CH];
#pragma unroll
  for (int k = 0; k < CH; ++k) {
    x[k] = get(c[k]);
    if (e + W * (k / NV) + (W / NV) * (k % NV) + lane >= ee) x[k].x = x[k].y = 0;
  }
#pragma unroll
  for (int k = 0; k < CH; ++k) {
    double q[4];
    QuadRaw<QT>::get(m[k], q);
    const double xu = sign * (double)x[k].x, xv = sign * (double)x[k].y;
    a0[k % NV] = fma(q[TR ? 2 : 1], xv, fma(q[0], xu, a0[k % NV]));
    a1[k % NV] = fma(q[3], xv, fma(q[TR ? 1 : 2], xu, a1[k % NV]));
  }
}
// Entries [e, ee) of a row over W virtual lanes, NV of them per physical lane, in chunks of KC entries
// each (of one for a rest that W entries hold: a short row does not pay for a long chunk).  TR: the quad
// transposed (restriction).  a0, a1: the virtual lanes' sums.
template <int W, int NV, int KC, bool TR, typename QT, typename G>
__device__ __forceinline__ void row_sums(const int* col, const char* val, int e, int ee, int lane, double sign, G get,
                                         ColRange range, double (&a0)[NV], double (&a1)[NV]) {
  while (e < ee) {
    if (KC == 1 || ee - e <= W) {
      row_chunk<W, NV, 1, TR, QT>(col, val, e, ee, lane, sign, get, range, a0, a1);
      e += W;
    } else {
      row_chunk<W, NV, KC, TR, QT>(col, val, e, ee, lane, sign, get, range, a0, a1);
      e += W * KC;
    }
  }
}
// the butterfly of W virtual lanes, its first stages inside the physical lane
template <int W, int NV>
__device__ __forceinline__ double lanes_total(const double (&a)[NV]) {
  static_assert(NV == 1 || NV == 4, "one or four virtual lanes a lane");
  return lane_sum(NV == 1 ? a[0] : (a[0] + a[NV / 2]) + (a[NV / 4] + a[NV / 2 + NV / 4]), W / NV);
}

// b_c = Q' b for the coarse nodes of level l + 1; with a second vector, of b - alpha q (rounded as
// the update of the residual rounds it), scaled by w.
template <int NV, typename VT, typename QT>
__device__ __forceinline__ void cyc_down_nv(const LevS& L, int c0, int lo, int hi, const typename Vec2<VT>::T* b,
                                            typename Vec2<VT>::T* bc, const typename Vec2<VT>::T* q2, double alpha,
                                            double w, bool rev, ColRange range) {
  using V2 = typename Vec2<VT>::T;
  constexpr int lanes = kDownW / NV, nsub = kCycThreads / lanes, KC = sizeof(VT) == 4 ? (NV == 1 ? 4 : 2) : (NV == 1 ? 2 : 1);
  const int sub = threadIdx.x / lanes, lane = threadIdx.x & (lanes - 1);
  for (int j0 = lo; j0 < hi; j0 += nsub) {
    const int J = c0 + (rev ? lo + hi - 1 - (j0 + sub) : j0 + sub);
    const bool valid = j0 + sub < hi;
    double a0[NV] = {}, a1[NV] = {};
    if (valid)
      row_sums<kDownW, NV, KC, true, QT>(L.tfine, L.tval, L.tptr[J], L.tptr[J + 1], lane, 1.0, [&](int f) {
        V2 x = b[f];
        if (q2) {
          const V2 y = q2[f];
          x.x = (VT)((double)x.x - alpha * (double)y.x);
          x.y = (VT)((double)x.y - alpha * (double)y.y);
        }
        return x;
      }, range, a0, a1);
    const double s0 = lanes_total<kDownW, NV>(a0), s1 = lanes_total<kDownW, NV>(a1);
    if (valid && lane == 0) {
      V2 o;
      o.x = (VT)(w * s0);
      o.y = (VT)(w * s1);
      bc[J] = o;
    }
  }
}
template <typename VT, typename QT>
__device__ __forceinline__ void cyc_down(const LevS& L, const CycSys& S, int l, const TeamCtx& t,
                                         const typename Vec2<VT>::T* b, typename Vec2<VT>::T* bc,
                                         const typename Vec2<VT>::T* q2 = nullptr, double alpha = 0.0,
                                         double w = 1.0, bool rev = false) {
  int lo, hi;
  team_share(t, S.nn[l + 1], lo, hi);
  const ColRange range = UA_COL_RANGE(t.dbg, S.n0[l], S.nn[l]);
  if (hi - lo <= kCycThreads / kDownW)
    cyc_down_nv<1, VT, QT>(L, S.n0[l + 1], lo, hi, b, bc, q2, alpha, w, rev, range);
  else
    cyc_down_nv<4, VT, QT>(L, S.n0[l + 1], lo, hi, b, bc, q2, alpha, w, rev, range);
}

// z = 2 b - A b + Q z_c on level l >= 1 (zc: indexed by the coarse level's node numbers).
template <int NV, typename VT, typename AT, typename QT>
__device__ __forceinline__ void cyc_up_nv(const LevS& L, int n0, int lo, int hi, const typename Vec2<VT>::T* b,
                                          typename Vec2<VT>::T* z, const typename Vec2<VT>::T* zc,
                                          ColRange range, ColRange range_c) {
  using V2 = typename Vec2<VT>::T;
  constexpr int lanes = kUpW / NV, nsub = kCycThreads / lanes, KC = sizeof(VT) == 4 ? (NV == 1 ? 4 : 2) : (NV == 1 ? 2 : 1);
  const int sub = threadIdx.x / lanes, lane = threadIdx.x & (lanes - 1);
  for (int j0 = lo; j0 < hi; j0 += nsub) {
    const int g = n0 + j0 + sub;
    const bool valid = j0 + sub < hi;
    double a0[NV] = {}, a1[NV] = {};
    V2 bv;
    bv.x = bv.y = 0;
    if (valid) {
      bv = b[g];
      row_sums<kUpW, NV, KC, false, AT>(L.acol, L.aval, L.aptr[g], L.aptr[g + 1], lane, -1.0,
                                        [&](int c) { return b[c]; }, range, a0, a1);
      row_sums<kUpW, NV, KC, false, QT>(L.qcol, L.qval, L.qptr[g], L.qptr[g + 1], lane, 1.0,
                                        [&](int c) { return zc[c]; }, range_c, a0, a1);
    }
    const double s0 = lanes_total<kUpW, NV>(a0), s1 = lanes_total<kUpW, NV>(a1);
    if (valid && lane == 0) {
      V2 o;
      o.x = (VT)(2.0 * (double)bv.x + s0);
      o.y = (VT)(2.0 * (double)bv.y + s1);
      z[g] = o;
    }
  }
}
template <typename VT, typename AT, typename QT>
__device__ __forceinline__ void cyc_up(const LevS& L, const CycSys& S, int l, const TeamCtx& t,
                                       const typename Vec2<VT>::T* b, typename Vec2<VT>::T* z,
                                       const typename Vec2<VT>::T* zc) {
  int lo, hi;
  team_share(t, S.nn[l], lo, hi);
  const ColRange range = UA_COL_RANGE(t.dbg, S.n0[l], S.nn[l]), range_c = UA_COL_RANGE(t.dbg, S.n0[l + 1], S.nn[l + 1]);
  if (hi - lo <= kCycThreads / kUpW)
    cyc_up_nv<1, VT, AT, QT>(L, S.n0[l], lo, hi, b, z, zc, range, range_c);
  else
    cyc_up_nv<4, VT, AT, QT>(L, S.n0[l], lo, hi, b, z, zc, range, range_c);
}

// The coarsest level of the system by every CTA of the team for itself (no team barrier follows):
// zc = A_L^-1 b_L in shared memory, the dense inverse in the dof order [u; v].  Threads along the
// rows (the inverse is symmetric, so a row is read as a column: consecutive threads, consecutive
// words), the columns in as many segments as the CTA has threads for; sums in a fixed order.
struct DenseSh {
  double b[kAmgMaxDense];
  double part[kCycThreads];
};
template <typename VT>
__device__ __forceinline__ void cyc_dense(const CycSys& S, const double* M, const typename Vec2<VT>::T* bL,
                                          DenseSh& sh, typename Vec2<VT>::T* zc) {
  using V2 = typename Vec2<VT>::T;
  const int n = S.dn, nn = n >> 1, c0 = S.n0[S.depth], np = (n + 31) & ~31, seg = kCycThreads / np;
  for (int i = threadIdx.x; i < nn; i += kCycThreads) {
    const V2 v = bL[c0 + i];
    sh.b[i] = (double)v.x;
    sh.b[nn + i] = (double)v.y;
  }
  __syncthreads();
  const int k = threadIdx.x / np, r = threadIdx.x - k * np;
  if (k < seg) {
    double acc = 0;
    if (r < n) {
      const int lo = n * k / seg, hi = n * (k + 1) / seg;
#pragma unroll 8
      for (int c = lo; c < hi; ++c) acc = fma(M[c * n + r], sh.b[c], acc);
    }
    sh.part[threadIdx.x] = acc;
  }
  __syncthreads();
  if (threadIdx.x < n) {
    double acc = 0;
    for (int q = 0; q < seg; ++q) acc += sh.part[q * np + threadIdx.x];
    reinterpret_cast<VT*>(zc)[threadIdx.x < nn ? 2 * threadIdx.x : 2 * (threadIdx.x - nn) + 1] = (VT)acc;
  }
  __syncthreads();
}

// The levels from S.solo on by every CTA of the team for itself: from b (global, level S.solo) to z_c of
// that level in shared memory, without a team barrier.  Levels of at most kSoloNodes nodes: their rows are
// some tens of kilobytes, the passes a few hundred cycles between CTA barriers, where a team barrier and
// the hand-over of a level through L2 cost 2.2 us each (P1 141x71, levels of 10011, 1128, 80 and 7 nodes:
// 25.5 -> 23.0 us a PCG step).  Same sums in the same order as by the team.
// buf: twice the nodes of those levels and of the coarsest one.
constexpr int kSoloNodes = 128;
constexpr int kSoloBuf = 4 * kSoloNodes + kAmgCoarseNodes;  // cycle_init leaves out levels that do not fit
template <typename VT, typename KT, typename QT>
__device__ __forceinline__ const typename Vec2<VT>::T* cyc_solo(const LevS* lev, const CycSys& S, const CycArgs& A,
                                                                const double* dense, DenseSh& dsh,
                                                                typename Vec2<VT>::T* zcs,
                                                                typename Vec2<VT>::T* buf) {
  using V2 = typename Vec2<VT>::T;
  const TeamCtx one{0, 1, nullptr, 0u, nullptr, A.dbg};
  const int s0 = S.solo, dep = S.depth;
  const V2* b0 = (const V2*)A.lev[s0].b + S.n0[s0];
  for (int i = threadIdx.x; i < S.nn[s0]; i += kCycThreads) buf[i] = b0[i];
  __syncthreads();
  V2* b = buf;
  for (int l = s0; l < dep; ++l) {
    V2* bc = b + S.nn[l];
    cyc_down<VT, QT>(lev[l], S, l, one, b - S.n0[l], bc - S.n0[l + 1]);
    b = bc;
    __syncthreads();
  }
  cyc_dense<VT>(S, dense, b - S.n0[dep], dsh, zcs);
  V2* z = b + S.nn[dep];
  const V2* zc = zcs - S.n0[dep];
  for (int l = dep - 1; l >= s0; --l) {
    b -= S.nn[l];
    cyc_up<VT, KT, QT>(lev[l], S, l, one, b - S.n0[l], z - S.n0[l], zc);
    __syncthreads();
    zc = z - S.n0[l];
    z += S.nn[l];
  }
  return zc;
}

// CH slots k0 .. of a slice product of width k1: the columns and values load
// together, then the gathered pairs.  Slots past the end repeat the last one with a zero vector
// entry, so that nothing branches between the loads.
template <int CH, typename KT, typename VT>
__device__ __forceinline__ void slice_chunk(const int* cp, const char* vp, int lane, int k0, int k1,
                                            const typename Vec2<VT>::T* v, ColRange range, double& a0, double& a1) {
  using V2 = typename Vec2<VT>::T;
  int j[CH];
  typename QuadRaw<KT>::T e[CH];
#pragma unroll
  for (int k = 0; k < CH; ++k) {
    const int kk = min(k0 + k, k1 - 1);
    j[k] = cp[32 * kk + lane];
    UA_CHECK_COL(range, j[k], BS_SLICE_COL);
    e[k] = SliceQuad<KT>::load(vp + (long long)kk * (128 * sizeof(KT)), lane);
  }
  V2 x[CH];
#pragma unroll
  for (int k = 0; k < CH; ++k) {
    x[k] = v[j[k]];
    if (k0 + k >= k1) x[k].x = x[k].y = 0;
  }
#pragma unroll
  for (int k = 0; k < CH; ++k) {
    double q[4];
    QuadRaw<KT>::get(e[k], q);
    a0 = fma(q[0], (double)x[k].x, a0);
    a0 = fma(q[1], (double)x[k].y, a0);
    a1 = fma(q[2], (double)x[k].x, a1);
    a1 = fma(q[3], (double)x[k].y, a1);
  }
}

// (A^ v) at slice sl's lane (its node sits at position 32 sl + lane: the vectors of
// the finest level are kept in slice order), in chunks of ten slots (five for FP64 values and for
// what is left): a linear mesh's slice is one or two chunks, two dependent loads each, where a plain
// unrolled loop takes the slots of its remainder one by one.
template <typename KT, typename VT>
__device__ __forceinline__ void slice_product(const long long* sl_off, const int* cols, const char* vals, int sl,
                                              int lane, const typename Vec2<VT>::T* v, ColRange range, double& a0,
                                              double& a1) {
  const long long off = sl_off[sl];
  const int k1 = (int)((sl_off[sl + 1] - off) >> 5);
  const int* cp = cols + off;
  const char* vp = vals + off * (long long)(4 * sizeof(KT));
  a0 = a1 = 0;
  for (int k0 = 0; k0 < k1;) {  // the width is the same for the whole warp
    if (sizeof(KT) < 8 && k1 - k0 > 5) {
      slice_chunk<10, KT, VT>(cp, vp, lane, k0, k1, v, range, a0, a1);
      k0 += 10;
    } else if (k1 - k0 > 3) {
      slice_chunk<5, KT, VT>(cp, vp, lane, k0, k1, v, range, a0, a1);
      k0 += 5;
    } else {
      slice_chunk<3, KT, VT>(cp, vp, lane, k0, k1, v, range, a0, a1);
      k0 += 3;
    }
  }
}

// The slices' columns and values into L2 ahead of their use (one lane; sizes and addresses are
// multiples of 128 bytes): the demand loads then wait for L2 instead of DRAM.
__device__ __forceinline__ void prefetch_l2(const void* p, long long bytes) {
  if (bytes >= 16)
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"((unsigned)bytes) : "memory");
}
template <typename KT>
__device__ __forceinline__ void slice_prefetch(const long long* sl_off, const int* cols, const void* vals, int sl) {
  const long long off = sl_off[sl], n = sl_off[sl + 1] - off;
  prefetch_l2(cols + off, 4 * n);
  prefetch_l2((const char*)vals + off * (4 * sizeof(KT)), n * (4 * sizeof(KT)));
}

// Runs the slices [lo, hi) over the CTA's warps: f(i, lane's node, node is there, a slice of the next
// round, which may lie outside).  The slices of a
// block of eight are ordered by width (25 down to 9 slots on a quadratic mesh), so the warps rotate
// from round to round: with a plain stride of 16 a warp met the same place of a block every time,
// and a pass waited for the warps of the widest one (401x201 P2: CTAs of 52k and 110k cycles side
// by side).  (Splitting a slice's slots over two or four warps of a CTA that has few was slower
// at every size: the exchange through shared memory costs what the shorter chains save.)
//
// rev: from the last slice to the first.  A pass that reads what the pass before it (or the same pass of
// the step before) has read goes the other way, so that it meets in L2 what was read last.
template <typename F>
__device__ __forceinline__ void for_slices(int lo, int hi, int n0, int nn, bool rev, F f) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int b = lo, r = 0; b < hi; b += kCycWarps, r += 5) {
    const int k = b + ((warp + r) & (kCycWarps - 1)), i = rev ? hi - 1 - (k - lo) : k;
    if (k < hi) f(i, n0 + 32 * i + lane, 32 * i + lane < nn, rev ? i - kCycWarps : i + kCycWarps);
  }
}

// - w A^ b + Q z_c at the lane of slice sl, finest level (the caller adds 2 w b).
template <typename LT, typename VT, typename QT>
__device__ __forceinline__ void cyc_up0_node(const FineS& F, const LevS& L, const CycSys& S, const TeamCtx& t, int sl, int lane,
                                             const typename Vec2<VT>::T* b, const typename Vec2<VT>::T* zc, double w,
                                             double& z0, double& z1) {
  double a0, a1, q0, q1;
  slice_product<LT, VT>(F.sl_off, F.cols, F.lv, sl, lane, b, UA_COL_RANGE(t.dbg, S.n0[0], S.nn[0]), a0, a1);
  slice_product<QT, VT>(L.qoff, L.qcol, L.qval, sl, lane, zc, UA_COL_RANGE(t.dbg, S.n0[1], S.nn[1]), q0, q1);
  z0 = q0 - w * a0;
  z1 = q1 - w * a1;
}

// ---- host side of a resident launch (ua_pcg.cu) ----
struct CycSchedule {
  std::vector<int4> cta;
  std::vector<int> team, queue;
};
void cycle_schedule(const std::vector<CycSys>& sys, const std::vector<int>& sel, const std::vector<int>& steps,
                    int nsm, CycSchedule& out);
int upload_schedule(ua_mesh* m, const CycSchedule& s);
void arena_size(const Cycle& C, const CycSchedule& sch, CycForm form, int most, int small, int& bytes, bool& room);
CycArgs cycle_args(const ua_mesh* m, CycForm form, bool prof);
// cooperative launch of a team kernel, one CTA per SM
template <typename A>
inline int launch_team(ua_mesh* m, void (*k)(const A), const A& a, int nctas, int smem) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(nctas);
  cfg.blockDim = dim3(kCycThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = m->stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  UA_CUDA_TRY(cudaLaunchKernelEx(&cfg, k, a));
  return UA_OK;
}

// Per-thread phase clock of a profiled solve: the first thread of a team's first CTA adds the time
// since the last mark, weighted with the team's share of the grid, to the class of the pass.
enum { CP_SPMV = 0, CP_DOWN0, CP_UP0, CP_OTHER, CP_COUNT };
__device__ __forceinline__ unsigned long long cyc_now() {
  unsigned long long v;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(v));
  return v;
}

}  // namespace ua
