// Resident restarted GMRES of the implicit uvh Newton system: one cooperative launch runs the whole
// solve of every selected system (ua_cycle.cuh: teams, collapsed V-cycle of the velocity block).
//
// Launched pass by pass, an Arnoldi step was 34 launches and a host synchronisation for the
// rotations (250 us on the 101x51-vertex P2 mesh).  Here the step's passes are separated by team
// barriers and the Hessenberg column, the rotations and the convergence test are computed by one
// thread of every CTA for itself, so the host takes no part until the solve ends.
#include <algorithm>
#include <cstring>
#include "ua_alloc.h"
#include "ua_cycle.cuh"

namespace ua {

constexpr int kGmMaxRestart = 48;  // the triangular factor and the rotations live in shared memory
constexpr int kGmSlab = 64;        // slices whose dot products are combined at a time
constexpr int kGmArena = 180 * 1024, kGmArenaSmall = 64 * 1024;

// Slices per partial sum: at most 2048 partials of a dot product per system (every CTA of the team
// reads them all), a function of the system's size alone.
__host__ __device__ inline int gm_unit(int nsl) {
  int u = 1;
  while ((nsl + u - 1) / u > 2048 && u < kGmSlab) u <<= 1;
  return u;
}

// The 3-dof tangent in the node slices: nine values a slot, each of them contiguous over the lanes
// (entry (3 c + b) of slot k at 9 (off + 32 k) + 32 (3 c + b) + lane), rows of constrained dofs zero;
// and the inverse l1 row sums of the thickness block in slice order (0 on constrained rows).
__global__ void __launch_bounds__(256) k_gm_fill(CycFine F, const int* sb_n0, const int* sb_cnt, const int* sb_sys,
                                                 const int* node_off, const int* dof_off, const int* rowptr,
                                                 const double* K, const unsigned char* cmask, double* out,
                                                 double* hinv, const int* sel) {
  const int sb = blockIdx.x, s = sb_sys[sb];
  if (!sel[s]) return;
  const int w = threadIdx.x >> 5, t = threadIdx.x & 31, pos = w * 32 + t, sl = sb * kSellSlices + w;
  const long long o0 = F.sl_off[sl];
  const int W = (int)((F.sl_off[sl + 1] - o0) >> 5);
  if (W == 0) return;
  const int no = node_off[s], nn = node_off[s + 1] - no, d0 = dof_off[s];
  const bool has = pos < sb_cnt[sb];
  const int at = sb_n0[sb] + (has ? pos : 0);
  int r[3] = {0, 0, 0}, deg = 0;
  bool live[3] = {false, false, false};
  if (has) {
    const int i = d0 + (F.perm[at] - no);
    for (int c = 0; c < 3; ++c) {
      r[c] = rowptr[i + c * nn];
      live[c] = !cmask[i + c * nn];
    }
    deg = (rowptr[i + 1] - r[0]) / 3;
  }
  double l1 = 0;
  for (int k = 0; k < W; ++k) {
    double* o = out + 9 * (o0 + 32LL * k) + t;
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        const double v = (live[c] && k < deg) ? K[r[c] + b * deg + k] : 0.0;
        o[32 * (3 * c + b)] = v;
        if (c == 2 && b == 2) l1 += fabs(v);
      }
  }
  if (has) hinv[at] = live[2] ? (l1 > 0 ? 1.0 / l1 : 1.0) : 0.0;
}

struct GmVec {  // a vector in slice order: velocity pairs and thickness
  double2* uv;
  double* h;
};

struct GmArgs {
  CycArgs cyc;
  const void* lv;           // cycle operator of the velocity block (FP64)
  const double *v3, *hinv;
  const double *f;          // right-hand side (dofs)
  double* dX;               // in: the particular solution; out: the solution
  const unsigned char* cmask;
  const int* dof_off;
  const double2* sc;        // D^-1/2 of the velocity block per node
  double2* scp;             // the same in slice order
  double* V;                // mr + 1 basis vectors of 3 npad doubles
  GmVec w, z, x, fs;
  double2* ws;              // D^-1/2 w
  double *bh, *ht;          // thickness sweeps: right-hand side, ping-pong
  double *part1, *part2, *part3;  // partials of the two Gram-Schmidt passes and of the norms, [vector][part_ld]
  long long npad, part_ld, part_sys;  // part_sys: doubles per system
  int mr, maxit, max_cycles;
  int hsw;
  const double* tol;        // [nsys]
  int *done, *its;
  int arena;
  bool room;
};

__device__ __forceinline__ GmVec gm_basis(const GmArgs& a, int i) {
  double* b = a.V + (size_t)i * 3 * a.npad;
  return GmVec{reinterpret_cast<double2*>(b), b + 2 * a.npad};
}

// (K v) at the lane of slice sl
__device__ __forceinline__ void gm_product(const CycFine& F, const double* v3, int sl, int lane,
                                           const GmVec& v, ColRange range, double (&r)[3]) {
  const long long off = F.sl_off[sl];
  const int k1 = (int)((F.sl_off[sl + 1] - off) >> 5);
  const int* cp = F.cols + off + lane;
  const double* vp = v3 + 9 * off + lane;
  r[0] = r[1] = r[2] = 0;
  constexpr int CH = 5;
  for (int k0 = 0; k0 < k1; k0 += CH) {
    double2 xu[CH];
    double xh[CH];
#pragma unroll
    for (int k = 0; k < CH; ++k) {
      int j = __ldg(cp + 32 * min(k0 + k, k1 - 1));
      UA_CHECK_COL(range, j, BS_GM_COL);
      xu[k] = v.uv[j];
      xh[k] = v.h[j];
    }
#pragma unroll
    for (int k = 0; k < CH; ++k) {
      if (k0 + k >= k1) xu[k].x = xu[k].y = xh[k] = 0;
      const double* e = vp + 288 * min(k0 + k, k1 - 1);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        r[c] = fma(__ldg(e + 96 * c), xu[k].x, r[c]);
        r[c] = fma(__ldg(e + 96 * c + 32), xu[k].y, r[c]);
        r[c] = fma(__ldg(e + 96 * c + 64), xh[k], r[c]);
      }
    }
  }
}
// thickness row: B = 0: (K_hu v_u + K_hv v_v), B = 1: K_hh v_h
template <int B>
__device__ __forceinline__ double gm_hrow(const CycFine& F, const double* v3, int sl, int lane,
                                          const double2* uv, const double* h, ColRange range) {
  const long long off = F.sl_off[sl];
  const int k1 = (int)((F.sl_off[sl + 1] - off) >> 5);
  const int* cp = F.cols + off + lane;
  const double* vp = v3 + 9 * off + lane + (B ? 256 : 192);
  double acc = 0;
  constexpr int CH = B ? 10 : 7;
  for (int k0 = 0; k0 < k1; k0 += CH) {
    int j[CH];
    double e0[CH], e1[CH];
#pragma unroll
    for (int k = 0; k < CH; ++k) {
      const int kk = min(k0 + k, k1 - 1);
      j[k] = __ldg(cp + 32 * kk);
      UA_CHECK_COL(range, j[k], BS_GM_COL);
      e0[k] = __ldg(vp + 288 * kk);
      if (!B) e1[k] = __ldg(vp + 288 * kk + 32);
    }
#pragma unroll
    for (int k = 0; k < CH; ++k) {
      const bool in = k0 + k < k1;
      if (B) {
        const double x = h[j[k]];
        acc = fma(e0[k], in ? x : 0.0, acc);
      } else {
        const double2 x = uv[j[k]];
        acc = fma(e0[k], in ? x.x : 0.0, acc);
        acc = fma(e1[k], in ? x.y : 0.0, acc);
      }
    }
  }
  return acc;
}

// Sums of eight values over the warp: lane l returns the total of value l >> 2 (7 + 2 exchanges of
// doubles instead of 40).
__device__ __forceinline__ double warp_sum8(double (&v)[8], int lane) {
#pragma unroll
  for (int s = 0, n = 4, o = 16; s < 3; ++s, n >>= 1, o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (k < n) {
        const double send = up ? v[k] : v[k + n], keep = up ? v[k + n] : v[k];
        v[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
      }
  }
  v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
  v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
  return v[0];
}

constexpr int kGmUpd = 512;  // node partials of a split update: 4 x 128 or 2 x 256
struct GmShared {
  double R[kGmMaxRestart * (kGmMaxRestart + 1) / 2];  // packed columns of the triangular factor
  double cs[kGmMaxRestart], sn[kGmMaxRestart], g[kGmMaxRestart + 1], y[kGmMaxRestart];
  double h1[kGmMaxRestart + 1], h2[kGmMaxRestart + 1];
  double slab[8][kGmSlab];
  double upd[3 * kGmUpd];
  double scal[4];
  int flag;
};

// Dot products of w with the basis vectors 0 .. nv-1 (nv = 0: with itself) over the slices of the
// CTA's units; one partial per vector and unit.  w may have been written by other warps: the CTA meets
// first.  With one slice a unit the warps take pairs (slice, eight vectors), so that a CTA with four
// slices keeps all sixteen busy.
__device__ __forceinline__ double gm_dot8(const GmArgs& a, int g, bool in, int nv, int c, int lane) {
  double v[8];
  double2 wu = make_double2(0, 0);
  double wh = 0;
  if (in) {
    wu = a.w.uv[g];
    wh = a.w.h[g];
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    v[k] = 0;
    if (in && (nv ? 8 * c + k < nv : k == 0)) {
      const GmVec b = nv ? gm_basis(a, 8 * c + k) : a.w;
      const double2 bu = b.uv[g];
      v[k] = wu.x * bu.x + wu.y * bu.y + wh * b.h[g];
    }
  }
  return warp_sum8(v, lane);
}
__device__ __forceinline__ void gm_dots(const GmArgs& a, GmShared& sh, const CycSys& S, int U, int u0, int u1, int nv,
                                        double* part) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, n0 = S.n0[0], nn = S.nn[0];
  const int chunks = nv ? (nv + 7) >> 3 : 1, per = max(1, kGmSlab / U);
  __syncthreads();
  if (U == 1) {
    const int ns = u1 - u0;
    for (int q = warp; q < ns * chunks; q += kCycWarps) {
      const int c = q / ns, i = u0 + (q - c * ns);
      const double t = gm_dot8(a, n0 + 32 * i + lane, 32 * i + lane < nn, nv, c, lane);
      if ((lane & 3) == 0 && (nv ? 8 * c + (lane >> 2) < nv : lane == 0)) part[(8 * c + (lane >> 2)) * a.part_ld + i] = t;
    }
    return;
  }
  for (int ub = u0; ub < u1; ub += per) {
    const int ue = min(ub + per, u1), s0 = ub * U, s1 = min(ue * U, S.nsl);
    for (int c = 0; c < chunks; ++c) {
      for (int i = s0 + warp; i < s1; i += kCycWarps) {
        const double t = gm_dot8(a, n0 + 32 * i + lane, 32 * i + lane < nn, nv, c, lane);
        if ((lane & 3) == 0) sh.slab[lane >> 2][i - s0] = t;
      }
      __syncthreads();
      const int nu = ue - ub;
      for (int k = threadIdx.x; k < 8 * nu; k += kCycThreads) {
        const int q = k / nu, u = k - q * nu;
        if (!(nv ? 8 * c + q < nv : q == 0)) continue;
        double t = 0;
        for (int i = u * U; i < min((u + 1) * U, s1 - s0); ++i) t += sh.slab[q][i];
        part[(8 * c + q) * a.part_ld + ub + u] = t;
      }
      __syncthreads();
    }
  }
}
// totals of nv dot products: a warp takes three at a time, four partials of each in flight per lane
__device__ __forceinline__ void gm_totals(const GmArgs& a, const double* part, int units, int nv, double* out) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i0 = warp; i0 < nv; i0 += 3 * kCycWarps) {
    double t[3] = {0, 0, 0};
    for (int k0 = lane; k0 < units; k0 += 128) {
      double v[3][4];
#pragma unroll
      for (int q = 0; q < 3; ++q)
#pragma unroll
        for (int k = 0; k < 4; ++k)
          v[q][k] = i0 + q * kCycWarps < nv && k0 + 32 * k < units
                        ? __ldcg(part + (i0 + q * kCycWarps) * a.part_ld + k0 + 32 * k) : 0.0;
#pragma unroll
      for (int q = 0; q < 3; ++q)
#pragma unroll
        for (int k = 0; k < 4; ++k) t[q] += v[q][k];
    }
#pragma unroll
    for (int q = 0; q < 3; ++q)
      if (i0 + q * kCycWarps < nv) {  // uniform over the warp
        const double s = lane_sum(t[q], 32);
        if (lane == 0) out[i0 + q * kCycWarps] = s;
      }
  }
  __syncthreads();
}

// sum over the vectors q = r, r + 4, ... <= j of h[q] b_q at node k (class r of four)
__device__ __forceinline__ void gm_class_sum(const GmArgs& a, const double* h, int r, int j, int k, double (&o)[3]) {
  o[0] = o[1] = o[2] = 0;
#pragma unroll 5
  for (int q = r; q <= j; q += 4) {
    const GmVec b = gm_basis(a, q);
    const double2 bu = b.uv[k];
    o[0] = fma(h[q], bu.x, o[0]);
    o[1] = fma(h[q], bu.y, o[1]);
    o[2] = fma(h[q], b.h[k], o[2]);
  }
}
// w -= sum_q h[q] b_q on the slices [lo, hi) and, if asked for, ws = D^-1/2 w.  The vectors are summed in
// four classes q mod 4, added as (0 + 2) + (1 + 3).  A CTA with at most four (eight) slices gives a class
// (two) to a warp, so that a warp waits for ten basis vectors instead of forty one after the other.
__device__ __forceinline__ void gm_update(const GmArgs& a, GmShared& sh, const double* h, int j, int lo, int hi, int n0,
                                          int nn, bool scaled) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, ns = hi - lo;
  auto write = [&](int k, double s0, double s1, double s2) {
    double2 wu = a.w.uv[k];
    wu.x -= s0;
    wu.y -= s1;
    a.w.uv[k] = wu;
    a.w.h[k] -= s2;
    if (scaled) {
      const double2 d = a.scp[k];
      a.ws[k] = make_double2(d.x * wu.x, d.y * wu.y);
    }
  };
  const int G = ns <= 4 ? 4 : ns <= 8 ? 2 : 1;
  if (G == 1) {
    for (int i = lo + warp; i < hi; i += kCycWarps) {
      const int k = n0 + 32 * i + lane;
      if (32 * i + lane < nn) {
        double c0[3], c1[3], c2[3], c3[3];
        gm_class_sum(a, h, 0, j, k, c0);
        gm_class_sum(a, h, 2, j, k, c2);
        gm_class_sum(a, h, 1, j, k, c1);
        gm_class_sum(a, h, 3, j, k, c3);
        write(k, (c0[0] + c2[0]) + (c1[0] + c3[0]), (c0[1] + c2[1]) + (c1[1] + c3[1]),
              (c0[2] + c2[2]) + (c1[2] + c3[2]));
      }
    }
    return;
  }
  const int per = kCycWarps / G, i = lo + warp % per, r = warp / per, nl = 32 * per;  // slots per class
  if (i < hi && 32 * i + lane < nn) {
    double c[3];
    gm_class_sum(a, h, r, j, n0 + 32 * i + lane, c);
    if (G == 2) {
      double d[3];
      gm_class_sum(a, h, r + 2, j, n0 + 32 * i + lane, d);
      for (int q = 0; q < 3; ++q) c[q] += d[q];
    }
    const int at = r * nl + 32 * (i - lo) + lane;
    for (int q = 0; q < 3; ++q) sh.upd[q * kGmUpd + at] = c[q];
  }
  __syncthreads();
  for (int e = threadIdx.x; e < 32 * ns; e += kCycThreads)
    if (32 * lo + e < nn) {
      double s[3];
      for (int q = 0; q < 3; ++q) {
        const double* u = sh.upd + q * kGmUpd + e;
        s[q] = G == 2 ? u[0] + u[nl] : (u[0] + u[2 * nl]) + (u[nl] + u[3 * nl]);
      }
      write(n0 + 32 * lo + e, s[0], s[1], s[2]);
    }
}

#define UA_TEAM_SYNC(t) UA_TEAM_SYNC_WITH(t, []() {})
#define UA_TEAM_SYNC_WITH(t, ...)                                     \
  do {                                                                \
    if (!team_sync(t, __VA_ARGS__)) {                                            \
      if (threadIdx.x == 0) *a.cyc.err = 1;                           \
      return;                                                         \
    }                                                                 \
  } while (0)

// Right-preconditioned GMRES(mr) of the systems in the team's queue.  Preconditioner: the velocity
// block's V-cycle, then z_h = K_hh^-1 (r_h - K_hu z_u) with hsw l1-Jacobi sweeps from zero.  Passes of
// an Arnoldi step: the finest restriction (which also writes V_j = w / |w|), the other levels, the
// finest up pass, the thickness rows, hsw - 1 sweeps, the product with the dot products of the first
// Gram-Schmidt pass, its subtraction with those of the second, the second's with the norm.
__global__ void __launch_bounds__(kCycThreads, 1) k_gmres_team(const GmArgs a) {
  extern __shared__ __align__(16) char arena_mem[];
  __shared__ CycSys S;
  __shared__ LevS lev[kCycMaxLev];
  __shared__ FineS fine;
  __shared__ DenseSh dsh;
  __shared__ double2 zcs[kAmgMaxDense / 2], sbuf[kSoloBuf];
  __shared__ GmShared sh;
  __shared__ int ok;
  const int4 c = a.cyc.cta[blockIdx.x];
  TeamCtx t{c.z, c.w, a.cyc.bar + 32 * a.cyc.team[blockIdx.x], 0u, &ok, a.cyc.dbg};
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int qi = c.x; qi < c.y; ++qi) {
    const int s = a.cyc.queue[qi];
    __syncthreads();
    if (threadIdx.x < (int)(sizeof(CycSys) / sizeof(int)))
      reinterpret_cast<int*>(&S)[threadIdx.x] = reinterpret_cast<const int*>(a.cyc.sys + s)[threadIdx.x];
    __syncthreads();
    Arena ar{arena_mem, a.arena, 0};
    const double* dense;
    const int n0 = S.n0[0], nn = S.nn[0], dep = S.depth, U = gm_unit(S.nsl), units = (S.nsl + U - 1) / U;
    const int solo = t.size > 1 ? S.solo : dep;
    const ColRange range = UA_COL_RANGE(t.dbg, n0, nn);
    const double2* bL = (const double2*)a.cyc.lev[dep].b;
    int u0, u1;
    team_share(t, units, u0, u1);
    const int lo = u0 * U, hi = min(u1 * U, S.nsl);
    cyc_stage<double, double, double, double>(a.cyc, a.lv, a.lv, S, t, lo, hi, ar, lev, &fine, 32, dense, a.room);
    // vectors into slice order
    for (int i = lo + warp; i < hi; i += kCycWarps)
      if (32 * i + lane < nn) {
        const int k = n0 + 32 * i + lane, g = a.cyc.fine.perm[k], j = a.dof_off[s] + (g - n0);
        a.fs.uv[k] = make_double2(a.cmask[j] ? 0.0 : a.f[j], a.cmask[j + nn] ? 0.0 : a.f[j + nn]);
        a.fs.h[k] = a.cmask[j + 2 * nn] ? 0.0 : a.f[j + 2 * nn];
        a.x.uv[k] = make_double2(a.dX[j], a.dX[j + nn]);
        a.x.h[k] = a.dX[j + 2 * nn];
        a.scp[k] = a.sc[g];
      }
    UA_TEAM_SYNC(t);
    double *part1 = a.part1 + s * a.part_sys, *part2 = a.part2 + s * a.part_sys, *part3 = a.part3 + s * a.part_sys;
    int its = 0, cycles = 0;
    double beta0 = 0;
    const double tol = a.tol[s];
    while (true) {
      // residual
      for_slices(lo, hi, n0, nn, false, [&](int i, int k, bool in, int) {
        if (!in) return;
        double kx[3];
        gm_product(a.cyc.fine, a.v3, S.sl0 + i, lane, a.x, range, kx);
        const double2 f = a.fs.uv[k], d = a.scp[k];
        const double2 r = make_double2(f.x - kx[0], f.y - kx[1]);
        // constrained rows: f and the product are zero
        a.w.uv[k] = r;
        a.w.h[k] = a.fs.h[k] - kx[2];
        a.ws[k] = make_double2(d.x * r.x, d.y * r.y);
      });
      gm_dots(a, sh, S, U, u0, u1, 0, part3);
      UA_TEAM_SYNC(t);
      gm_totals(a, part3, units, 1, sh.scal);
      const double beta = sqrt(fmax(sh.scal[0], 0.0));
      if (cycles == 0) beta0 = beta;
      if (!(beta == beta) || beta <= tol * beta0 || beta == 0.0 || its >= a.maxit || cycles >= a.max_cycles) break;
      if (threadIdx.x == 0) {
        for (int i = 0; i <= a.mr; ++i) sh.g[i] = 0;
        sh.g[0] = beta;
      }
      double inv = 1.0 / beta;
      int j = 0;
      bool combine = false;  // the preconditioner pass of the cycle's update x += M^-1 (V y)
      while (true) {
        GmVec vj = combine ? a.w : gm_basis(a, j);
        // finest restriction; V_j = w inv
        if (!combine)
          for (int i = lo + warp; i < hi; i += kCycWarps) {
            const int k = n0 + 32 * i + lane;
            if (32 * i + lane < nn) {
              const double2 wu = a.w.uv[k];
              vj.uv[k] = make_double2(wu.x * inv, wu.y * inv);
              vj.h[k] = a.w.h[k] * inv;
            }
          }
        cyc_down<double, double>(lev[0], S, 0, t, a.ws, (double2*)a.cyc.lev[1].b, nullptr, 0.0, inv);
        UA_TEAM_SYNC(t);
        for (int l = 1; l < solo; ++l) {
          cyc_down<double, double>(lev[l], S, l, t, (const double2*)a.cyc.lev[l].b, (double2*)a.cyc.lev[l + 1].b);
          UA_TEAM_SYNC(t);
        }
        const double2* zc = zcs - S.n0[dep];
        if (solo < dep) zc = cyc_solo<double, double, double>(lev, S, a.cyc, dense, dsh, zcs, sbuf);
        else cyc_dense<double>(S, dense, bL, dsh, zcs);
        for (int l = solo - 1; l > 0; --l) {
          cyc_up<double, double, double>(lev[l], S, l, t, (const double2*)a.cyc.lev[l].b, (double2*)a.cyc.lev[l].z, zc);
          UA_TEAM_SYNC(t);
          zc = (const double2*)a.cyc.lev[l].z;
        }
        for_slices(lo, hi, n0, nn, false, [&](int i, int k, bool in, int) {
          if (!in) return;
          double z0, z1;
          cyc_up0_node<double, double, double>(fine, lev[0], S, t, S.sl0 + i, lane, a.ws, zc, inv, z0, z1);
          const double2 d = a.scp[k], b = a.ws[k];
          a.z.uv[k] = make_double2(d.x * (2.0 * inv * b.x + z0), d.y * (2.0 * inv * b.y + z1));
        });
        UA_TEAM_SYNC(t);
        // thickness rows; the sweeps ping-pong so that the last one writes z.h
        double* bufs[2] = {a.z.h, a.ht};
        int cur = (a.hsw - 1) % 2 == 0 ? 0 : 1;
        for_slices(lo, hi, n0, nn, false, [&](int i, int k, bool in, int) {
          if (!in) return;
          const double b = vj.h[k] - gm_hrow<0>(a.cyc.fine, a.v3, S.sl0 + i, lane, a.z.uv, nullptr, range);
          const double hi1 = a.hinv[k];
          a.bh[k] = hi1 > 0 ? b : 0.0;
          bufs[cur][k] = b * hi1;
        });
        UA_TEAM_SYNC(t);
        for (int q = 1; q < a.hsw; ++q) {
          const double* zi = bufs[cur];
          double* zo = bufs[1 - cur];
          for_slices(lo, hi, n0, nn, false, [&](int i, int k, bool in, int) {
            if (in)
              zo[k] = zi[k] + (a.bh[k] - gm_hrow<1>(a.cyc.fine, a.v3, S.sl0 + i, lane, nullptr, zi, range)) * a.hinv[k];
          });
          UA_TEAM_SYNC(t);
          cur = 1 - cur;
        }
        if (combine) break;
        // w = K z and its dot products
        for_slices(lo, hi, n0, nn, false, [&](int i, int k, bool in, int) {
          if (!in) return;
          double kx[3];
          gm_product(a.cyc.fine, a.v3, S.sl0 + i, lane, a.z, range, kx);
          a.w.uv[k] = make_double2(kx[0], kx[1]);
          a.w.h[k] = kx[2];
        });
        gm_dots(a, sh, S, U, u0, u1, j + 1, part1);
        UA_TEAM_SYNC(t);
        for (int pass = 0; pass < 2; ++pass) {
          double* h = pass ? sh.h2 : sh.h1;
          gm_totals(a, pass ? part2 : part1, units, j + 1, h);
          gm_update(a, sh, h, j, lo, hi, n0, nn, pass != 0);
          gm_dots(a, sh, S, U, u0, u1, pass ? 0 : j + 1, pass ? part3 : part2);
          // the previous rotations of the new column, while the team gathers
          UA_TEAM_SYNC_WITH(t, [&]() {
            if (!pass) return;
            double* R = sh.R + j * (j + 1) / 2;
            double up = sh.h1[0] + sh.h2[0];
            for (int i = 0; i < j; ++i) {
              const double nx = sh.h1[i + 1] + sh.h2[i + 1];
              R[i] = sh.cs[i] * up + sh.sn[i] * nx;
              up = -sh.sn[i] * up + sh.cs[i] * nx;
            }
            sh.scal[2] = up;
          });
        }
        gm_totals(a, part3, units, 1, sh.scal);
        if (threadIdx.x == 0) {
          double* R = sh.R + j * (j + 1) / 2;
          const double hn = sqrt(fmax(sh.scal[0], 0.0));
          const double up = sh.scal[2];
          const double den = hypot(up, hn);
          sh.cs[j] = den > 0 ? up / den : 1.0;
          sh.sn[j] = den > 0 ? hn / den : 0.0;
          R[j] = den;
          sh.g[j + 1] = -sh.sn[j] * sh.g[j];
          sh.g[j] = sh.cs[j] * sh.g[j];
          const double res = fabs(sh.g[j + 1]);
          sh.scal[1] = hn;
          sh.flag = res <= tol * beta0 || hn == 0.0 || !(res == res) || its + 1 >= a.maxit || j + 1 == a.mr;
          if (sh.flag)  // y from the triangular system
            for (int i = j; i >= 0; --i) {
              double acc = sh.g[i];
              for (int q = i + 1; q <= j; ++q) acc -= sh.R[q * (q + 1) / 2 + i] * sh.y[q];
              const double d = sh.R[i * (i + 1) / 2 + i];
              sh.y[i] = d != 0.0 ? acc / d : 0.0;
            }
        }
        __syncthreads();
        ++its;
        ++j;
        if (sh.flag) {  // w = V y: the next pass applies the preconditioner to it
          for (int i = lo + warp; i < hi; i += kCycWarps) {
            const int k = n0 + 32 * i + lane;
            if (32 * i + lane < nn) {
              double2 wu = make_double2(0, 0);
              double wh = 0;
              for (int q = 0; q < j; ++q) {
                const GmVec b = gm_basis(a, q);
                const double2 bu = b.uv[k], d = bu;
                wu.x = fma(sh.y[q], d.x, wu.x);
                wu.y = fma(sh.y[q], d.y, wu.y);
                wh = fma(sh.y[q], b.h[k], wh);
              }
              const double2 d = a.scp[k];
              a.w.uv[k] = wu;
              a.w.h[k] = wh;
              a.ws[k] = make_double2(d.x * wu.x, d.y * wu.y);
            }
          }
          UA_TEAM_SYNC(t);
          combine = true;
          inv = 1.0;
        } else {
          inv = sh.scal[1] > 0 ? 1.0 / sh.scal[1] : 0.0;
        }
      }
      // x += z (the own rows; the next residual reads the neighbours')
      for (int i = lo + warp; i < hi; i += kCycWarps) {
        const int k = n0 + 32 * i + lane;
        if (32 * i + lane < nn) {
          const double2 zu = a.z.uv[k];
          double2 xu = a.x.uv[k];
          xu.x += zu.x;
          xu.y += zu.y;
          a.x.uv[k] = xu;
          a.x.h[k] += a.z.h[k];
        }
      }
      UA_TEAM_SYNC(t);
      ++cycles;
    }
    for (int i = lo + warp; i < hi; i += kCycWarps)
      if (32 * i + lane < nn) {
        const int k = n0 + 32 * i + lane, j = a.dof_off[s] + (a.cyc.fine.perm[k] - n0);
        const double2 xu = a.x.uv[k];
        a.dX[j] = xu.x;
        a.dX[j + nn] = xu.y;
        a.dX[j + 2 * nn] = a.x.h[k];
      }
    if (t.rank == 0 && threadIdx.x == 0) {
      a.its[s] = its;
      a.done[s] = 1;
    }
  }
}

int gmres_resident_max_restart() { return kGmMaxRestart; }

int gmres_resident(ua_mesh* m, const GmSolve& v, const std::vector<int>& sel, const std::vector<int>& steps, int nsm,
                   long long* launches) {
  Amg* a = m->amg;
  Cycle& C = a->cyc;
  const Sell& S = a->sell;
  const long long npad = (a->lev[0].nn + 1) & ~1LL;
  long long ld = 1;
  for (const CycSys& y : C.sys) {
    const int U = gm_unit(y.nsl);
    ld = std::max(ld, (long long)(y.nsl + U - 1) / U);
  }
  // partials of system s start at its own offset: one block of [vector][ld] per system
  const size_t np = (size_t)(2 * (v.mr + 1) + 1) * ld;
  if (!alloc_for(C.gm_mr, v.mr,
                 {{(void**)&C.gm_buf, sizeof(double) * (size_t)(3 * (v.mr + 1) + 18) * npad},
                  {(void**)&C.gm_part, sizeof(double) * np * a->nsys},
                  {(void**)&C.gm_v3, sizeof(double) * 9 * (size_t)std::max(S.slots, 1LL)},
                  {(void**)&C.gm_hinv, sizeof(double) * (size_t)npad}},
                 [&](size_t n) { return dev_alloc(m, n); }, [&](void* p) { dev_free(m, p); }))
    return set_error(UA_ERR_OOM, "device allocation of the GMRES basis failed");
  k_gm_fill<<<std::max(S.nsb, 1), 256, 0, m->stream>>>(CycFine{S.perm, S.sl_off, C.d_pcol}, S.sb_n0, S.sb_cnt,
                                                       S.sb_sys, m->dm.sys_node_off, m->dm.sys_dof_off, v.rowptr,
                                                       v.K, v.cmask, C.gm_v3, C.gm_hinv, v.sel), ++*launches;
  UA_CUDA_TRY(cudaGetLastError());
  CycSchedule sch;
  cycle_schedule(C.sys, sel, steps, std::min(nsm, 1024), sch);
  if (sch.cta.empty()) return UA_OK;
  if (int rc = upload_schedule(m, sch)) return rc;
  GmArgs A{};
  A.cyc = cycle_args(m, CF_FP64, false);
  A.lv = S.v64;
  A.v3 = C.gm_v3;
  A.hinv = C.gm_hinv;
  A.f = v.f;
  A.dX = v.dX;
  A.cmask = v.cmask;
  A.dof_off = m->dm.sys_dof_off;
  A.sc = C.lev[0].sc;
  double* b = C.gm_buf;
  auto take = [&](long long n) {
    double* p = b;
    b += n;
    return p;
  };
  auto vec = [&]() {
    double* p = take(3 * npad);
    return GmVec{(double2*)p, p + 2 * npad};
  };
  A.V = take(3 * (v.mr + 1) * npad);
  A.w = vec();
  A.z = vec();
  A.x = vec();
  A.fs = vec();
  A.ws = (double2*)take(2 * npad);
  A.scp = (double2*)take(2 * npad);
  A.bh = take(npad);
  A.ht = take(npad);
  A.part1 = C.gm_part;
  A.part2 = A.part1 + (size_t)(v.mr + 1) * ld;
  A.part3 = A.part2 + (size_t)(v.mr + 1) * ld;
  A.part_sys = (long long)np;
  A.npad = npad;
  A.part_ld = ld;
  A.mr = v.mr;
  A.hsw = v.hsw;
  A.maxit = v.maxit;
  A.max_cycles = v.max_cycles;
  A.tol = v.tol;
  A.done = v.done;
  A.its = v.its;
  arena_size(C, sch, CF_FP64, kGmArena, kGmArenaSmall, A.arena, A.room);
  UA_CUDA_TRY(cudaFuncSetAttribute(k_gmres_team, cudaFuncAttributeMaxDynamicSharedMemorySize, kGmArena));
  const int rc = launch_team(m, k_gmres_team, A, (int)sch.cta.size(), A.arena);
  ++*launches;
  return rc;
}

}  // namespace ua
