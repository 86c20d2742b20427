// Aggregation AMG preconditioner for the constrained uv tangent.
//
// Preconditions the inner PCG that replaces the reference's direct solve of
// the Newton system (ABfgPreEliminate.m:110).  Every level keeps Úa's dof
// layout [u; v] per system.  Default: smoothed aggregation, P = (I - w D^-1 A) P0
// with P0 piecewise constant over the aggregates of fine nodes, on the first
// transfer of a quadratic mesh the linear interpolation from the corner nodes;
// the Galerkin operators P' A P are formed from every tangent.  Plain aggregation
// (P0 itself, a pure summation) on request.  Smoother: one l1-Jacobi sweep
// (x += kSmoothOmega (b - A x) / sum_j |a_ij|) before and after the coarse
// correction, a symmetric V(1,1) cycle and so an SPD preconditioner for CG.
// Coarsest level: a dense inverse per system (at most 2*kAmgCoarseNodes dofs)
// applied as a matrix-vector product.  The cycle itself runs in collapsed form
// inside the resident solves (ua_cycle.cuh), or pass by pass (vcycle_t) where a
// solve is launched.
//
// The hierarchy of a system depends only on that system's mesh and every
// kernel works on per-system ranges in a fixed summation order, so a
// system's result is the same alone and in a batch.  Constrained dofs (the
// masked rows and columns of the projected system) have no coarse image:
// they are left out of the Galerkin sums, the restriction and the
// prolongation.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>
#include <type_traits>
#include "ua_amg_int.h"

namespace ua {

// Calls f(std::integral_constant<int, LPR>) for the lanes-per-row value lpr (1, 2, 4, 8, 16 or 32).
template <class F>
static void dispatch_lpr(int lpr, F&& f) {
  switch (lpr) {
    case 1: f(std::integral_constant<int, 1>()); break;
    case 2: f(std::integral_constant<int, 2>()); break;
    case 4: f(std::integral_constant<int, 4>()); break;
    case 16: f(std::integral_constant<int, 16>()); break;
    case 32: f(std::integral_constant<int, 32>()); break;
    default: f(std::integral_constant<int, 8>());
  }
}

// ---------------------------------------------------------------------------
// host: aggregation and hierarchy
// ---------------------------------------------------------------------------

// Greedy aggregation of a node graph (system-local ids, self included):
// (1) a node whose neighbourhood is entirely unassigned becomes the root of
// an aggregate of that neighbourhood; (2) an unassigned node joins the
// aggregate of its first assigned neighbour; (3) what is left forms
// aggregates with its unassigned neighbours.
static int aggregate(int n, const std::vector<int>& ptr, const std::vector<int>& col, std::vector<int>& agg) {
  agg.assign(n, -1);
  int na = 0;
  for (int i = 0; i < n; ++i) {
    if (agg[i] >= 0) continue;
    bool free_nb = true;
    for (int k = ptr[i]; k < ptr[i + 1] && free_nb; ++k) free_nb = agg[col[k]] < 0;
    if (!free_nb) continue;
    for (int k = ptr[i]; k < ptr[i + 1]; ++k) agg[col[k]] = na;
    ++na;
  }
  for (int i = 0; i < n; ++i) {
    if (agg[i] >= 0) continue;
    for (int k = ptr[i]; k < ptr[i + 1]; ++k)
      if (agg[col[k]] >= 0) { agg[i] = agg[col[k]]; break; }
  }
  for (int i = 0; i < n; ++i) {
    if (agg[i] >= 0) continue;
    for (int k = ptr[i]; k < ptr[i + 1]; ++k)
      if (agg[col[k]] < 0) agg[col[k]] = na;
    agg[i] = na++;
  }
  return na;
}

// Linear interpolation of a six-node system from its corner nodes: per node its corners (ascending
// corner ids, and their nodes) and weights, 1 at a corner and 1/2 at the two ends of a mid node's edge.  Corner
// ids follow the node order.  Returns the number of corners, or 0 where the mesh does not allow it (a
// node that is a corner of one element and a mid node of another, or in no element).
//
// A quadratic mesh is coarsened this way once, before the aggregation: the velocity tangent's
// smooth errors are linear over an element, so the interpolation needs no smoothing, the next
// operator keeps the sparsity of a linear mesh (about 7 nodes per row, where aggregating the
// quadratic graph gave 22) and the coarsening ratio is 4 instead of 16.  PCG iterations of one
// Newton system (relative 1e-6): 101 x 51 vertices 108 -> 39, with the damped smoother below 80 -> 30.
static int linear_corners(const HostSystem& hs, std::vector<int>& ptr, std::vector<int>& col,
                          std::vector<int>& node, std::vector<double>& wgt) {
  const int n = hs.nn, ne = hs.ne;
  std::vector<int> c0(n, -1), c1(n, -1);  // a mid node's edge ends; c0 = the node itself at a corner
  for (int e = 0; e < ne; ++e)
    for (int k = 0; k < 6; k += 2) {
      const int a = hs.conn[(size_t)k * ne + e], m = hs.conn[(size_t)(k + 1) * ne + e];
      const int b = hs.conn[(size_t)((k + 2) % 6) * ne + e];
      if ((c0[a] >= 0 && c0[a] != a) || a == b || a == m || m == b) return 0;
      c0[a] = a;
      const int lo = std::min(a, b), hi = std::max(a, b);
      if (c0[m] >= 0 && (c0[m] != lo || c1[m] != hi)) return 0;
      c0[m] = lo;
      c1[m] = hi;
    }
  std::vector<int> id(n, -1);
  int nc = 0;
  for (int i = 0; i < n; ++i) {
    if (c0[i] < 0) return 0;
    if (c1[i] < 0) id[i] = nc++;
  }
  ptr.assign(1, 0);
  ptr.reserve(n + 1);
  col.clear();
  node.clear();
  wgt.clear();
  for (int i = 0; i < n; ++i) {
    if (c1[i] < 0) {
      col.push_back(id[i]);
      node.push_back(i);
      wgt.push_back(1.0);
    } else {
      if (id[c0[i]] < 0 || id[c1[i]] < 0) return 0;  // an edge end that is a mid node elsewhere
      col.push_back(id[c0[i]]);
      col.push_back(id[c1[i]]);
      node.push_back(c0[i]);
      node.push_back(c1[i]);
      wgt.push_back(0.5);
      wgt.push_back(0.5);
    }
    ptr.push_back((int)col.size());
  }
  return nc;
}

// Dof-level CSR of a level from its node graph (global ids of the level):
// row (c, I) holds 2 blocks of deg(I) columns (block b, k-th neighbour).
static void level_csr(AmgLevel& L, const std::vector<int>& gptr, const std::vector<int>& gcol, int nsys,
                      std::vector<int>& rowptr, std::vector<int>& colind, std::vector<int>& dof_sys) {
  const std::vector<int>& no = L.node_off;
  L.dof_off.assign(nsys + 1, 0);
  L.knz_off.assign(nsys + 1, 0);
  L.nnzn.assign(nsys, 0);
  for (int s = 0; s < nsys; ++s) {
    const int n = no[s + 1] - no[s];
    L.dof_off[s + 1] = L.dof_off[s] + 2 * n;
    L.nnzn[s] = gptr[no[s + 1]] - gptr[no[s]];
    L.knz_off[s + 1] = L.knz_off[s] + 4 * L.nnzn[s];
  }
  const int N = L.dof_off[nsys];
  rowptr.assign(N + 1, 0);
  colind.assign(L.knz_off[nsys], 0);
  dof_sys.assign(N, 0);
  for (int s = 0; s < nsys; ++s) {
    const int n0 = no[s], n = no[s + 1] - n0, base = gptr[n0];
    for (int I = n0; I < n0 + n; ++I) {
      const int p0 = gptr[I], deg = gptr[I + 1] - p0;
      for (int c = 0; c < 2; ++c) {
        const int dof = L.dof_off[s] + c * n + (I - n0);
        const int start = L.knz_off[s] + c * 2 * L.nnzn[s] + 2 * (p0 - base);
        rowptr[dof] = start;
        dof_sys[dof] = s;
        for (int b = 0; b < 2; ++b)
          for (int k = 0; k < deg; ++k) colind[start + b * deg + k] = L.dof_off[s] + b * n + (gcol[p0 + k] - n0);
      }
    }
  }
  rowptr[N] = L.knz_off[nsys];
  L.nn = no[nsys];
  L.ndof = N;
  L.nnz = L.knz_off[nsys];
}

static int amg_build(ua_mesh* m, bool smoothed) {
  const int nsys = m->dm.nsys;
  Amg* a = new Amg();
  a->nsys = nsys;
  a->depth.assign(nsys, 0);
  // node graphs per level (global ids of the level)
  std::vector<std::vector<int>> g_off{m->h_node_off}, g_ptr{m->h_nodeptr}, g_col{m->h_nodecol}, g_agg;
  // smoothed aggregation lists per transfer (index = fine level)
  std::vector<std::vector<int>> g_pnp, g_pnc, g_apnp, g_apnc, g_ptnp, g_ptnf, g_ptnk;
  std::vector<double> pn_w;  // weights of the finest level's linear interpolation (else empty),
  std::vector<int> pn_f;     // and the corner nodes they are for
  a->sa = smoothed;
  // quadratic meshes: the first transfer interpolates linearly from the corner nodes, for every
  // system of the handle or for none
  std::vector<std::vector<int>> lin_ptr(nsys), lin_col(nsys), lin_f(nsys);
  std::vector<std::vector<double>> lin_w(nsys);
  std::vector<int> lin_n(nsys, 0);
  bool linear0 = smoothed && m->nod == 6;
  for (int s = 0; s < nsys && linear0; ++s)
    linear0 = (lin_n[s] = linear_corners(m->sys[s], lin_ptr[s], lin_col[s], lin_f[s], lin_w[s])) > 0;
  std::vector<char> live(nsys, 1);
  auto fail = [&](const char* why) {
    delete a;
    return set_error(UA_ERR_INVALID, "AMG setup: %s", why);
  };
  while (std::find(live.begin(), live.end(), 1) != live.end()) {
    const std::vector<int>& no = g_off.back();
    const std::vector<int>& fp = g_ptr.back();
    const std::vector<int>& fc = g_col.back();
    std::vector<int> agg(no[nsys], -1), cno(nsys + 1, 0), cptr(1, 0), ccol;
    std::vector<int> pnp(1, 0), pnc, apnp(1, 0), apnc, ptnp(1, 0), ptnf, ptnk;
    for (int s = 0; s < nsys; ++s) {
      const int n = no[s + 1] - no[s];
      if (!live[s] || n == 0) {
        cno[s + 1] = cno[s];
        for (int i = 0; i < n; ++i) { pnp.push_back((int)pnc.size()); apnp.push_back((int)apnc.size()); }
        continue;
      }
      std::vector<int> lp(n + 1, 0), lc, la;
      for (int i = 0; i < n; ++i) {
        for (int k = fp[no[s] + i]; k < fp[no[s] + i + 1]; ++k) lc.push_back(fc[k] - no[s]);
        lp[i + 1] = (int)lc.size();
      }
      const bool lin = linear0 && g_agg.empty();
      int na;
      if (lin) {
        na = lin_n[s];
        la.resize(n);
        for (int i = 0; i < n; ++i) la[i] = lin_col[s][lin_ptr[s][i]];
      } else {
        na = aggregate(n, lp, lc, la);
      }
      for (int i = 0; i < n; ++i) agg[no[s] + i] = cno[s] + la[i];
      cno[s + 1] = cno[s] + na;
      std::vector<std::vector<int>> adj(na);
      if (!smoothed) {
        for (int i = 0; i < n; ++i)
          for (int k = lp[i]; k < lp[i + 1]; ++k) adj[la[i]].push_back(la[lc[k]]);
      } else {
        // prolongator pattern: node i reaches the aggregates of its neighbours (P = (I - w D^-1 A) P0)
        std::vector<int> lpn(n + 1, 0), lpc, stamp(na, -1);
        if (lin) {
          lpn = lin_ptr[s];
          lpc = lin_col[s];
          pn_w.insert(pn_w.end(), lin_w[s].begin(), lin_w[s].end());
          for (int f : lin_f[s]) pn_f.push_back(no[s] + f);
        }
        for (int i = 0; i < n && !lin; ++i) {
          const size_t b0 = lpc.size();
          for (int k = lp[i]; k < lp[i + 1]; ++k) {
            const int J = la[lc[k]];
            if (stamp[J] != i) { stamp[J] = i; lpc.push_back(J); }
          }
          std::sort(lpc.begin() + b0, lpc.end());
          lpn[i + 1] = (int)lpc.size();
        }
        // A P pattern: node i reaches the union of its neighbours' prolongator rows
        std::vector<int> lapn(n + 1, 0), lapc;
        std::fill(stamp.begin(), stamp.end(), -1);
        for (int i = 0; i < n; ++i) {
          const size_t b0 = lapc.size();
          for (int k = lp[i]; k < lp[i + 1]; ++k) {
            const int h = lc[k];
            for (int t = lpn[h]; t < lpn[h + 1]; ++t)
              if (stamp[lpc[t]] != i) { stamp[lpc[t]] = i; lapc.push_back(lpc[t]); }
          }
          std::sort(lapc.begin() + b0, lapc.end());
          lapn[i + 1] = (int)lapc.size();
        }
        // transpose of the prolongator pattern, with each entry's position in its fine row
        std::vector<int> ltp(na + 1, 0), ltf(lpc.size()), ltk(lpc.size());
        for (int t = 0; t < (int)lpc.size(); ++t) ltp[lpc[t] + 1]++;
        for (int J = 0; J < na; ++J) ltp[J + 1] += ltp[J];
        {
          std::vector<int> nx(ltp.begin(), ltp.end() - 1);
          for (int i = 0; i < n; ++i)
            for (int t = lpn[i]; t < lpn[i + 1]; ++t) { ltf[nx[lpc[t]]] = i; ltk[nx[lpc[t]]++] = t - lpn[i]; }
        }
        // coarse node graph of P' A P
        std::fill(stamp.begin(), stamp.end(), -1);
        for (int I = 0; I < na; ++I)
          for (int u = ltp[I]; u < ltp[I + 1]; ++u) {
            const int i = ltf[u];
            for (int t = lapn[i]; t < lapn[i + 1]; ++t)
              if (stamp[lapc[t]] != I) { stamp[lapc[t]] = I; adj[I].push_back(lapc[t]); }
          }
        for (int i = 0; i < n; ++i) {
          for (int t = lpn[i]; t < lpn[i + 1]; ++t) pnc.push_back(cno[s] + lpc[t]);
          pnp.push_back((int)pnc.size());
          for (int t = lapn[i]; t < lapn[i + 1]; ++t) apnc.push_back(cno[s] + lapc[t]);
          apnp.push_back((int)apnc.size());
        }
        for (int J = 0; J < na; ++J) {
          for (int u = ltp[J]; u < ltp[J + 1]; ++u) { ptnf.push_back(no[s] + ltf[u]); ptnk.push_back(ltk[u]); }
          ptnp.push_back((int)ptnf.size());
        }
      }
      for (int I = 0; I < na; ++I) {
        std::sort(adj[I].begin(), adj[I].end());
        adj[I].erase(std::unique(adj[I].begin(), adj[I].end()), adj[I].end());
        if (!smoothed && 2 * (int)adj[I].size() > kAmgMaxRow) return fail("coarse node degree above the row limit");
        if (smoothed && (int)adj[I].size() > kSaMaxDeg) return fail("smoothed coarse node degree above the limit");
        for (int J : adj[I]) ccol.push_back(cno[s] + J);
        cptr.push_back((int)ccol.size());
      }
      a->depth[s]++;
      if (na <= kAmgCoarseNodes) live[s] = 0;
      else if (na >= n) return fail("aggregation made no progress");
    }
    g_agg.push_back(agg);
    g_off.push_back(cno);
    g_ptr.push_back(cptr);
    g_col.push_back(ccol);
    g_pnp.push_back(pnp); g_pnc.push_back(pnc); g_apnp.push_back(apnp); g_apnc.push_back(apnc);
    g_ptnp.push_back(ptnp); g_ptnf.push_back(ptnf); g_ptnk.push_back(ptnk);
  }
  a->nlev = (int)g_off.size();
  a->lev.resize(a->nlev);
  bool ok = true;
  for (int l = 0; l < a->nlev; ++l) {
    AmgLevel& L = a->lev[l];
    L.node_off = g_off[l];
    std::vector<int> rowptr, colind, dof_sys;
    level_csr(L, g_ptr[l], g_col[l], nsys, rowptr, colind, dof_sys);
    if (l == 0 && m->ndof == 2 && (L.ndof != m->ndof_total || L.nnz != m->nnz_total))
      return fail("fine level does not match the handle");
    std::vector<int> rb_start, rb_sys;
    L.h_sys_rb_off.assign(nsys + 1, 0);
    for (int s = 0; s < nsys; ++s) {
      for (int r = L.dof_off[s]; r < L.dof_off[s + 1]; r += smoothed ? kSaRB : kAmgRB) {
        rb_start.push_back(r);
        rb_sys.push_back(s);
      }
      L.h_sys_rb_off[s + 1] = (int)rb_sys.size();
    }
    rb_start.push_back(L.ndof);
    L.nrb = (int)rb_sys.size();
    L.invd = dalloc(m, a, sizeof(double) * (size_t)L.ndof, ok);
    if (l == 0 && m->ndof == 3) {
      // uvh handle: the finest level is the velocity block, held apart from the 3-dof
      // tangent (values extracted per Newton step), with its own rows and vectors
      L.rb_start = upload(m, a, rb_start, ok);
      L.rb_sys = upload(m, a, rb_sys, ok);
      L.dof_sys = upload(m, a, dof_sys, ok);
      L.rowptr = upload(m, a, rowptr, ok);
      L.colind = upload(m, a, colind, ok);
      L.d_knz_off = upload(m, a, L.knz_off, ok);
      L.A = dalloc(m, a, sizeof(double) * (size_t)L.nnz, ok);
      a->uvh_mask = (unsigned char*)dalloc(m, a, (size_t)L.ndof, ok);
      for (double** v : {&a->uvh_r, &a->uvh_x0, &a->uvh_z, &a->uvh_t})
        *v = (double*)dalloc(m, a, sizeof(double) * (size_t)L.ndof, ok);
    }
    if (l > 0) {  // the fine level of a uv handle uses the handle's tangent structure and PCG vectors
      L.rb_start = upload(m, a, rb_start, ok);
      L.rb_sys = upload(m, a, rb_sys, ok);
      L.dof_sys = upload(m, a, dof_sys, ok);
      L.rowptr = upload(m, a, rowptr, ok);
      L.colind = upload(m, a, colind, ok);
      L.A = dalloc(m, a, sizeof(double) * (size_t)L.nnz, ok);
      L.b = dalloc(m, a, sizeof(double) * (size_t)L.ndof, ok);
      L.x = dalloc(m, a, sizeof(double) * (size_t)L.ndof, ok);
      L.x2 = dalloc(m, a, sizeof(double) * (size_t)L.ndof, ok);
      // coarse dof (c, I) gathers fine dofs (c, i) with agg[i] = I, in ascending order
      AmgLevel& F = a->lev[l - 1];
      const std::vector<int>& agg = g_agg[l - 1];
      std::vector<int> cmap(F.ndof, -1), cnt(L.ndof + 1, 0), mlist(F.ndof);
      for (int s = 0; s < nsys; ++s) {
        const int fno = F.node_off[s], fn = F.node_off[s + 1] - fno;
        const int cno = L.node_off[s], cn = L.node_off[s + 1] - cno;
        if (cn == 0) continue;
        for (int c = 0; c < 2; ++c)
          for (int i = 0; i < fn; ++i)
            cmap[F.dof_off[s] + c * fn + i] = L.dof_off[s] + c * cn + (agg[fno + i] - cno);
      }
      for (int d = 0; d < F.ndof; ++d)
        if (cmap[d] >= 0) cnt[cmap[d] + 1]++;
      for (int d = 0; d < L.ndof; ++d) cnt[d + 1] += cnt[d];
      std::vector<int> mptr = cnt;
      for (int d = 0; d < F.ndof; ++d)
        if (cmap[d] >= 0) mlist[cnt[cmap[d]]++] = d;
      mlist.resize(mptr[L.ndof]);
      F.cmap = upload(m, a, cmap, ok);
      L.mptr = upload(m, a, mptr, ok);
      L.mlist = upload(m, a, mlist, ok);
    }
  }
  a->h_dn.assign(nsys, 0);
  a->h_doff.assign(nsys + 1, 0);
  for (int s = 0; s < nsys; ++s) {
    const AmgLevel& L = a->lev[a->depth[s]];
    a->h_dn[s] = L.dof_off[s + 1] - L.dof_off[s];
    if (a->h_dn[s] > kAmgMaxDense) return fail("coarsest system above the dense limit");
    a->maxdn = std::max(a->maxdn, a->h_dn[s]);
    a->h_doff[s + 1] = a->h_doff[s] + a->h_dn[s] * a->h_dn[s];
  }
  a->dense = (double*)dalloc(m, a, sizeof(double) * (size_t)a->h_doff[nsys], ok);
  a->d_depth = upload(m, a, a->depth, ok);
  a->d_dn = upload(m, a, a->h_dn, ok);
  a->d_doff = upload(m, a, a->h_doff, ok);
  std::vector<void*> pb(a->nlev), px2(a->nlev), pA(a->nlev);
  std::vector<int*> prp(a->nlev), pci(a->nlev), pdo(a->nlev);
  for (int l = 0; l < a->nlev; ++l) {
    a->lev[l].d_node_off = upload(m, a, a->lev[l].node_off, ok);
    if (a->sa) {
      std::vector<int> ns(std::max(a->lev[l].node_off[nsys], 1), 0);
      for (int s = 0; s < nsys; ++s)
        for (int g = a->lev[l].node_off[s]; g < a->lev[l].node_off[s + 1]; ++g) ns[g] = s;
      a->lev[l].node_sys = upload(m, a, ns, ok);
      std::vector<int> nbs, nbsys;
      AmgLevel& L = a->lev[l];
      L.h_sys_nb_off.assign(nsys + 1, 0);
      for (int s = 0; s < nsys; ++s) {
        for (int g = L.node_off[s]; g < L.node_off[s + 1]; g += kAmgNB) {
          nbs.push_back(g);
          nbsys.push_back(s);
        }
        L.h_sys_nb_off[s + 1] = (int)nbsys.size();
      }
      nbs.push_back(L.node_off[nsys]);
      L.nnb = (int)nbsys.size();
      L.nb_start = upload(m, a, nbs, ok);
      L.nb_sys = upload(m, a, nbsys, ok);
    }
    if (!a->lev[l].dof_sys) {  // a uv handle's finest level: rows -> system, for the smoothed transfer
      std::vector<int> ds(a->lev[l].ndof);
      for (int s = 0; s < nsys; ++s)
        for (int d = a->lev[l].dof_off[s]; d < a->lev[l].dof_off[s + 1]; ++d) ds[d] = s;
      a->lev[l].dof_sys = upload(m, a, ds, ok);
    }
    if (a->sa && l + 1 < a->nlev) {
      AmgLevel& F = a->lev[l];
      const AmgLevel& C = a->lev[l + 1];
      F.sa_agg = upload(m, a, g_agg[l], ok);
      if (l == 0 && linear0) {
        F.pn_w = upload(m, a, pn_w, ok);
        F.pn_f = upload(m, a, pn_f, ok);
      }
      F.pn_ptr = upload(m, a, g_pnp[l], ok);
      F.pn_col = upload(m, a, g_pnc[l], ok);
      F.apn_ptr = upload(m, a, g_apnp[l], ok);
      F.apn_col = upload(m, a, g_apnc[l], ok);
      F.ptn_ptr = upload(m, a, g_ptnp[l], ok);
      F.ptn_fine = upload(m, a, g_ptnf[l], ok);
      F.ptn_k = upload(m, a, g_ptnk[l], ok);
      F.np = g_pnp[l].back();
      F.nap = g_apnp[l].back();
      F.sa_ap = dalloc(m, a, 4 * sizeof(double) * (size_t)std::max(F.nap, 1LL), ok);
      a->lev[l + 1].gptr = upload(m, a, g_ptr[l + 1], ok);
      a->lev[l + 1].ng = g_ptr[l + 1].back();
    }
    pb[l] = a->lev[l].b;
    px2[l] = a->lev[l].x2;
    pA[l] = a->lev[l].A;
    prp[l] = a->lev[l].rowptr;
    pci[l] = a->lev[l].colind;
    pdo[l] = upload(m, a, a->lev[l].dof_off, ok);
    a->lev[l].d_dof_off = pdo[l];
  }
  a->d_lev_b = upload(m, a, pb, ok);
  a->d_lev_x2 = upload(m, a, px2, ok);
  a->d_lev_A = upload(m, a, pA, ok);
  a->d_lev_rowptr = upload(m, a, prp, ok);
  a->d_lev_colind = upload(m, a, pci, ok);
  a->d_lev_dofoff = upload(m, a, pdo, ok);
  if (!ok) {
    delete a;
    return set_error(UA_ERR_OOM, "AMG setup: device allocation failed");
  }
  if (a->sa) {  // for the structure of the collapsed cycle (cycle_init)
    a->h_gptr = std::move(g_ptr);
    a->h_gcol = std::move(g_col);
    a->h_apnp = std::move(g_apnp);
    a->h_apnc = std::move(g_apnc);
  }
  m->amg = a;
  return UA_OK;
}

// smoothed aggregation first (when asked), plain aggregation if the smoothed hierarchy
// exceeds its limits; a shape neither can take keeps point Jacobi for the handle's life
int amg_setup(ua_mesh* m, bool smoothed) {
  if (m->amg) return UA_OK;
  if (m->amg_failed) return UA_ERR_INVALID;
  if (m->ndof != 2 && m->ndof != 3) return set_error(UA_ERR_INVALID, "the AMG preconditioner needs uv or uvh dofs");
  int rc = amg_build(m, smoothed);
  if (rc == UA_ERR_INVALID && smoothed) rc = amg_build(m, false);
  if (rc == UA_ERR_INVALID) m->amg_failed = true;
  return rc;
}

void amg_free(Amg* a) { delete a; }

int amg_levels(const ua_mesh* m) { return m->amg ? m->amg->nlev : 0; }

const void* amg_invd0(const ua_mesh* m) { return m->amg ? m->amg->lev[0].invd : nullptr; }

// ---------------------------------------------------------------------------
// device: numeric phase
// ---------------------------------------------------------------------------

// Galerkin product: coarse row R sums the unmasked entries of its member
// rows into the coarse columns cmap[j] (binary search in the sorted coarse row).
template <typename KT>
__global__ void k_amg_galerkin(int ncd, const int* mptr, const int* mlist, const int* frowptr, const int* fcolind,
                               const KT* fA, const int* cmap, const unsigned char* cmask, const int* crowptr,
                               const int* ccolind, KT* cA) {
  const int R = blockIdx.x * blockDim.x + threadIdx.x;
  if (R >= ncd) return;
  const int c0 = crowptr[R], len = crowptr[R + 1] - c0;
  double acc[kAmgMaxRow];
#pragma unroll
  for (int k = 0; k < kAmgMaxRow; ++k) acc[k] = 0;
  for (int t = mptr[R]; t < mptr[R + 1]; ++t) {
    const int i = mlist[t];
    if (cmask && cmask[i]) continue;
    for (int q = frowptr[i]; q < frowptr[i + 1]; ++q) {
      const int j = fcolind[q];
      if (cmask && cmask[j]) continue;
      const int C = cmap[j];
      int lo = 0, hi = len - 1;
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (ccolind[c0 + mid] < C) lo = mid + 1; else hi = mid;
      }
      acc[lo] += (double)fA[q];
    }
  }
  for (int k = 0; k < len; ++k) cA[c0 + k] = (KT)acc[k];
}

// Damped l1-Jacobi: invd_i = kSmoothOmega / sum_j |a_ij| over unmasked columns (0 on masked or empty rows)
template <typename KT, typename VT>
__global__ void k_amg_l1(int n, const int* rowptr, const int* colind, const KT* A, const unsigned char* cmask,
                         VT* invd, const int* dof_sys, const int* sel) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (sel && !sel[dof_sys[i]]) return;  // systems not in this Newton step keep their values
  double s = 0;
  if (!(cmask && cmask[i]))
    for (int q = rowptr[i]; q < rowptr[i + 1]; ++q)
      if (!(cmask && cmask[colind[q]])) s += fabs((double)A[q]);
  invd[i] = (VT)(s > 0 ? kSmoothOmega / s : 0.0);
}

// Inverse of each system's coarsest matrix: Gauss-Jordan in place, one CTA per system, row-major
// result.  A is the Galerkin product of the SPD tangent (symmetric positive definite on the free
// dofs), so no pivoting is needed; a zero row (an aggregate of constrained dofs only; its column is
// zero too) is replaced by the identity row.
//
// The matrix is scaled to a unit diagonal (pivots in (0, 1]) and lives in registers, kDiT x kDiT
// entries a thread; the pivot row and column go through shared memory, in two copies so that a step
// has one barrier.  Step k is one update e_ij -= f_i w_j for every entry, with w_j = row_j / p and
// f_i = column_i except w_k = 1 + 1/p and f_k = p - 1, which give the pivot row, the pivot column
// and the pivot their own values without a test in the tile (the additions there are of terms of
// equal sign as p <= 1).  The steps are unrolled over a tile's pivots, so that a pivot's place in the
// tile is a compile-time index, and the pivot's owner takes the reciprocal: n = 94 in 44 us (every
// thread selecting and dividing, 265 instructions a step: 102 us).
constexpr int kDiT = 6, kDiG = kAmgMaxDense / kDiT, kDiThreads = kDiG * kDiG;
static_assert(kAmgMaxDense % kDiT == 0 && kDiThreads <= 1024, "the threads' tiles cover the largest coarsest matrix");
template <typename KT>
__global__ void __launch_bounds__(kDiThreads) k_amg_dense_inverse(const int* depth, const int* dn_arr,
                                                                  const int* doff, int* const* lev_rowptr,
                                                                  int* const* lev_colind, void* const* lev_A,
                                                                  int* const* lev_dofoff, double* dense,
                                                                  const int* sel) {
  constexpr int ND = kAmgMaxDense;
  extern __shared__ double M[];  // n x n staging of the matrix
  __shared__ double prow[2][ND], pcol[2][ND], dg[ND];
  __shared__ double2 piv[2];  // the pivot and its reciprocal
  const int s = blockIdx.x;
  const int n = dn_arr[s];
  if (n == 0 || (sel && !sel[s])) return;
  const int l = depth[s];
  const int* rp = lev_rowptr[l];
  const int* ci = lev_colind[l];
  const KT* A = (const KT*)lev_A[l];
  const int d0 = lev_dofoff[l][s];
  for (int t = threadIdx.x; t < n * n; t += kDiThreads) M[t] = 0;
  __syncthreads();
  for (int r = threadIdx.x >> 3; r < n; r += kDiThreads / 8)  // 8 lanes per row
    for (int q = rp[d0 + r] + (threadIdx.x & 7); q < rp[d0 + r + 1]; q += 8) M[r * n + (ci[q] - d0)] = (double)A[q];
  __syncthreads();
  for (int r = threadIdx.x; r < n; r += kDiThreads) {
    double d = M[r * n + r];
    if (!(d > 0)) {
      bool zero = true;
      for (int c = 0; c < n; ++c) zero = zero && M[r * n + c] == 0.0;
      if (zero) M[r * n + r] = 1.0;
      d = 1.0;
    }
    dg[r] = 1.0 / sqrt(d);
  }
  __syncthreads();
  const int r0 = (threadIdx.x / kDiG) * kDiT, c0 = (threadIdx.x % kDiG) * kDiT;
  const bool mine = r0 < n && c0 < n;
  double e[kDiT][kDiT];
#pragma unroll
  for (int i = 0; i < kDiT; ++i)
#pragma unroll
    for (int j = 0; j < kDiT; ++j)
      e[i][j] = (r0 + i < n && c0 + j < n) ? M[(r0 + i) * n + c0 + j] * dg[r0 + i] * dg[c0 + j] : 0.0;
  const int ty = threadIdx.x / kDiG, tx = threadIdx.x % kDiG;
  for (int kb = 0; kb * kDiT < n; ++kb) {
#pragma unroll
    for (int kk = 0; kk < kDiT; ++kk) {  // pivot kb kDiT + kk: entry kk of tile row and column kb
      const int k = kb * kDiT + kk;
      if (k >= n) break;
      double *pr = prow[kk & 1], *pc = pcol[kk & 1];
      if (ty == kb) {
        if (tx == kb) piv[kk & 1] = make_double2(e[kk][kk], 1.0 / e[kk][kk]);
#pragma unroll
        for (int j = 0; j < kDiT; ++j) pr[c0 + j] = e[kk][j];
      }
      if (tx == kb) {
#pragma unroll
        for (int i = 0; i < kDiT; ++i) pc[r0 + i] = e[i][kk];
      }
      __syncthreads();
      if (!mine) continue;  // padding only (it still meets the barriers)
      const double p = piv[kk & 1].x, inv = piv[kk & 1].y;
      double w[kDiT], f[kDiT];
#pragma unroll
      for (int j = 0; j < kDiT; ++j) w[j] = pr[c0 + j] * inv;
      if (tx == kb) w[kk] = 1.0 + inv;
#pragma unroll
      for (int i = 0; i < kDiT; ++i) f[i] = pc[r0 + i];
      if (ty == kb) f[kk] = p - 1.0;
#pragma unroll
      for (int i = 0; i < kDiT; ++i)
#pragma unroll
        for (int j = 0; j < kDiT; ++j) e[i][j] = fma(-f[i], w[j], e[i][j]);
    }
  }
  if (!mine) return;
#pragma unroll
  for (int i = 0; i < kDiT; ++i)
#pragma unroll
    for (int j = 0; j < kDiT; ++j)
      if (r0 + i < n && c0 + j < n)
        dense[doff[s] + (r0 + i) * n + c0 + j] = e[i][j] * dg[r0 + i] * dg[c0 + j];
}

// ---------------------------------------------------------------------------
// device: V-cycle
// ---------------------------------------------------------------------------

// x2 = inv(A_L) b on each system's coarsest level L: grid (system, 32-row
// slab), one warp per row with the lanes over the columns (row-major inverse,
// coalesced), b staged in shared memory.
template <typename VT>
__global__ void __launch_bounds__(256) k_amg_dense_apply(const int* sel, const int* done, const int* depth,
                                                         const int* dn_arr, const int* doff, int* const* lev_dofoff,
                                                         void* const* lev_b, void* const* lev_x2,
                                                         const double* dense) {
  pdl_enter();
  __shared__ double sb[kAmgMaxDense];
  const int s = blockIdx.x;
  if (!sel[s] || done[s]) return;
  const int n = dn_arr[s], r0 = blockIdx.y * 32;
  if (r0 >= n) return;
  const int l = depth[s];
  const int d0 = lev_dofoff[l][s];
  const VT* b = (const VT*)lev_b[l] + d0;
  VT* x = (VT*)lev_x2[l] + d0;
  for (int c = threadIdx.x; c < n; c += blockDim.x) sb[c] = (double)b[c];
  __syncthreads();
  const double* Mi = dense + doff[s];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int r1 = min(r0 + 32, n);
  for (int r = r0 + warp; r < r1; r += nw) {  // warp-uniform
    double acc = 0;
    for (int c = lane; c < n; c += 32) acc += Mi[r * n + c] * sb[c];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if (lane == 0) x[r] = (VT)acc;
  }
}

// Split V-cycle kernels (every level; coalesced row blocks with LPR lanes per
// row instead of one thread per aggregate).  Residual of the pre-smoothed
// vector of level l: res = mask(b - A x), for systems deeper than l.
// Row product in the uv block layout of every level: row (c, I) holds the u
// block then the v block of deg(I) entries on the same node columns, v column
// = u column + nhalf, so only the u block's indices are read (used for FP64
// values, where it is faster).
template <typename KT, typename XT, int LPR>
__device__ __forceinline__ double row_dot_uv(const int* rowptr, const int* colind, const KT* A, const XT* x, int row,
                                             bool valid, int lane, int nhalf) {
  double acc = 0;
  if (valid) {
    const int r0 = rowptr[row], deg = (rowptr[row + 1] - r0) >> 1;
    for (int k = lane; k < deg; k += LPR) {
      const int j = colind[r0 + k];
      acc += (double)A[r0 + k] * (double)x[j] + (double)A[r0 + deg + k] * (double)x[j + nhalf];
    }
  }
#pragma unroll
  for (int o = LPR / 2; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o, LPR);
  return acc;
}

// Plain CSR row product (every index read); the form that is faster for FP32 and BF16 values.
template <typename KT, typename XT, int LPR>
__device__ __forceinline__ double row_dot_csr(const int* rowptr, const int* colind, const KT* A, const XT* x, int row,
                                              bool valid, int lane) {
  double acc = 0;
  if (valid)
    for (int q = rowptr[row] + lane; q < rowptr[row + 1]; q += LPR) acc += to_d(A[q]) * (double)x[colind[q]];
#pragma unroll
  for (int o = LPR / 2; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o, LPR);
  return acc;
}

// BF16 copy of an FP32 tangent (the finest-level matrix of the mixed-precision
// V-cycle's residual and smoothing passes)
__global__ void k_to_bf16(long long n, const float* in, __nv_bfloat16* out) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    out[i] = __float2bfloat16_rn(in[i]);
}

template <typename KT, typename VT, int LPR>
__global__ void __launch_bounds__(256) k_amg_residual(const int* rb_start, const int* rb_sys, ActList act,
                                                      const int* sel, const int* done, const int* depth, int l,
                                                      const int* rowptr, const int* colind, const KT* A,
                                                      const VT* b, const VT* x, const unsigned char* cmask, VT* res,
                                                      const int* dof_off) {
  pdl_enter();
  const int nv = act.cnt ? *act.cnt : gridDim.x;  // list entries, else one block per CTA
  for (int vb = blockIdx.x; vb < nv; vb += gridDim.x) {
    const int blk = act.map ? act.map[vb] : vb;
    const int s = rb_sys[blk];
    if (!sel[s] || done[s] || depth[s] <= l) continue;  // uniform over the block
    const int rs = rb_start[blk], re = rb_start[blk + 1];
    const int nhalf = (dof_off[s + 1] - dof_off[s]) >> 1;
    const int lane = threadIdx.x % LPR, grp = threadIdx.x / LPR, ngrp = blockDim.x / LPR;
    for (int row0 = rs; row0 < re; row0 += ngrp) {  // same trip count for every thread of the block
      const int row = row0 + grp;
      const bool valid = row < re;
      const double ax = sizeof(KT) == 8 ? row_dot_uv<KT, VT, LPR>(rowptr, colind, A, x, row, valid, lane, nhalf)
                                        : row_dot_csr<KT, VT, LPR>(rowptr, colind, A, x, row, valid, lane);
      if (valid && lane == 0) res[row] = (VT)((cmask && cmask[row]) ? 0.0 : (double)b[row] - ax);
    }
  }
}

// Aggregation of a fine vector: b(R) = sum over members (ascending) of res;
// coarse pre-smoothing x = invd b unless lc is the system's coarsest level.
template <typename VT>
__global__ void k_amg_gather(int ncd, const int* dof_sys_c, const int* depth, int lc, const int* sel,
                             const int* done, const int* mptr, const int* mlist, const VT* res, const VT* cinvd,
                             VT* cb, VT* cx) {
  const int R = blockIdx.x * blockDim.x + threadIdx.x;
  if (R >= ncd) return;
  const int s = dof_sys_c[R];
  if (!sel[s] || done[s]) return;
  double acc = 0;
  for (int t = mptr[R]; t < mptr[R + 1]; ++t) acc += (double)res[mlist[t]];
  cb[R] = (VT)acc;
  if (depth[s] > lc) cx[R] = (VT)((double)cinvd[R] * acc);
}

// Coarse correction of level l, in place: x = mask(x + xc[cmap]) for systems deeper than l.
template <typename VT>
__global__ void __launch_bounds__(256) k_amg_correct(const int* rb_start, const int* rb_sys, const int* sel,
                                                     const int* done, const int* depth, int l, VT* x,
                                                     const VT* xc, const int* cmap, const unsigned char* cmask) {
  const int blk = blockIdx.x;
  const int s = rb_sys[blk];
  if (!sel[s] || done[s] || depth[s] <= l) return;
  for (int i = rb_start[blk] + threadIdx.x; i < rb_start[blk + 1]; i += blockDim.x)
    x[i] = (cmask && cmask[i]) ? (VT)0 : (VT)((double)x[i] + (double)xc[cmap[i]]);
}

// Post-smoothing of level l: out = xp + invd (b - A xp) (0 on masked rows)
// for systems deeper than l; on the finest level pcopy (if set) receives a
// copy and part the block partials of b.out.
template <typename KT, typename VT, int LPR>
__global__ void __launch_bounds__(256) k_amg_smooth(const int* rb_start, const int* rb_sys, ActList act,
                                                    const int* sel, const int* done, const int* depth, int l,
                                                    const int* rowptr, const int* colind, const KT* A, const VT* b,
                                                    const VT* xp, const VT* invd, const unsigned char* cmask, VT* out,
                                                    VT* pcopy, double* part, const int* dof_off) {
  pdl_enter();
  __shared__ double red[8];
  const int nv = act.cnt ? *act.cnt : gridDim.x;  // list entries, else one block per CTA
  for (int vb = blockIdx.x; vb < nv; vb += gridDim.x) {
    const int blk = act.map ? act.map[vb] : vb;
    const int s = rb_sys[blk];
    double rz = 0;
    if (sel[s] && !done[s] && depth[s] > l) {
      const int rs = rb_start[blk], re = rb_start[blk + 1];
      const int nhalf = (dof_off[s + 1] - dof_off[s]) >> 1;
      const int lane = threadIdx.x % LPR, grp = threadIdx.x / LPR, ngrp = blockDim.x / LPR;
      for (int row0 = rs; row0 < re; row0 += ngrp) {  // same trip count for every thread of the block
        const int row = row0 + grp;
        const bool valid = row < re;
        const double ax = sizeof(KT) == 8 ? row_dot_uv<KT, VT, LPR>(rowptr, colind, A, xp, row, valid, lane, nhalf)
                                          : row_dot_csr<KT, VT, LPR>(rowptr, colind, A, xp, row, valid, lane);
        if (valid && lane == 0) {
          const double v =
              (cmask && cmask[row]) ? 0.0 : (double)xp[row] + (double)invd[row] * ((double)b[row] - ax);
          out[row] = (VT)v;
          if (pcopy) pcopy[row] = (VT)v;
          rz += (double)b[row] * v;
        }
      }
    }
    if (!part) continue;  // uniform per launch
    double t = rz;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = t;
    __syncthreads();
    if (threadIdx.x == 0) {
      double sum = 0;
      for (int i = 0; i < (int)(blockDim.x >> 5); ++i) sum += red[i];
      part[blk] = sum;
    }
    __syncthreads();  // red is rewritten by the next entry
  }
}

// ---------------------------------------------------------------------------
// device: finest-level node slices (both rows of a node per thread)
// ---------------------------------------------------------------------------

struct SellDev {
  const int *sb_sys, *sb_n0, *sb_cnt, *perm;
  const long long* sl_off;
  const int* cols;
  const int *dof_off, *node_off;  // per system, of the slices' level
  unsigned long long* dbg;        // first bounds violation (debug build)
  int lev;                        // the level (residual and smoothing: systems deeper than it)
};

// Slice values (and, once per handle, the columns) from the tangent's CSR layout: row (c, g)
// starts at knz_off[s] + 2 c nnzn[s] + 2 lp(g) and holds the u block then the v block of deg(g)
// entries.  One CTA per slice block, one warp per slice, one lane per node; writes are contiguous.
template <typename KT>
__global__ void __launch_bounds__(256) k_sell_fill(SellDev S, const DevMesh dm, const KT* K, KT* vk,
                                                   __nv_bfloat16* vlo, int* cols, const int* sel) {
  const int sb = blockIdx.x;
  const int w = threadIdx.x >> 5, t = threadIdx.x & 31, pos = w * 32 + t;
  const int sl = sb * kSellSlices + w;
  const long long o0 = S.sl_off[sl];
  const int W = (int)((S.sl_off[sl + 1] - o0) >> 5);
  if (W == 0) return;  // empty slice (warp-uniform)
  const int s = S.sb_sys[sb];
  if (sel && K && !sel[s]) return;  // values of the systems of this Newton step only
  const int no = dm.sys_node_off[s], d0 = dm.sys_dof_off[s];
  const bool has = pos < S.sb_cnt[sb];
  int g = no, np0 = 0, deg = 0;
  if (has) {
    g = S.perm[S.sb_n0[sb] + pos];
    np0 = dm.nodeptr[g];
    deg = dm.nodeptr[g + 1] - np0;
  }
  const long long lp = (long long)np0 - dm.nodeptr[no];
  const long long bu = (long long)dm.sys_knz_off[s] + 2 * lp, bv = bu + 2LL * dm.sys_nnzn[s];
  for (int k = 0; k < W; ++k) {
    const bool in = has && k < deg;
    const long long d = o0 + 32LL * k + t;
    if (cols) cols[d] = d0 + (in ? dm.nodecol[np0 + k] : g) - no;
    if (!K) continue;
    KT e0 = 0, e1 = 0, e2 = 0, e3 = 0;
    if (in) { e0 = K[bu + k]; e1 = K[bu + deg + k]; e2 = K[bv + k]; e3 = K[bv + deg + k]; }
    if (vk) { vk[4 * d] = e0; vk[4 * d + 1] = e1; vk[4 * d + 2] = e2; vk[4 * d + 3] = e3; }
    if (vlo) {
      vlo[4 * d] = __float2bfloat16_rn((float)e0); vlo[4 * d + 1] = __float2bfloat16_rn((float)e1);
      vlo[4 * d + 2] = __float2bfloat16_rn((float)e2); vlo[4 * d + 3] = __float2bfloat16_rn((float)e3);
    }
  }
}

// Coarse-level slice values (and, once, the columns) from the level's CSR: row (c, I) holds the
// u block then the v block of deg(I) entries.  Same slice layout as the finest level.
template <typename KT>
__global__ void __launch_bounds__(256) k_csell_fill(SellDev S, const int* rowptr, const int* colind, const KT* A,
                                                    __nv_bfloat16* vlo, int* cols, const int* sel) {
  const int sb = blockIdx.x;
  const int w = threadIdx.x >> 5, t = threadIdx.x & 31, pos = w * 32 + t;
  const int sl = sb * kSellSlices + w;
  const long long o0 = S.sl_off[sl];
  const int W = (int)((S.sl_off[sl + 1] - o0) >> 5);
  if (W == 0) return;  // empty slice (warp-uniform)
  const int s = S.sb_sys[sb];
  if (sel && A && !sel[s]) return;  // values of the systems of this Newton step only
  const int no = S.node_off[s], nn = S.node_off[s + 1] - no, d0 = S.dof_off[s];
  const bool has = pos < S.sb_cnt[sb];
  int R0 = d0, q0 = 0, q1 = 0, deg = 0;
  if (has) {
    R0 = d0 + (S.perm[S.sb_n0[sb] + pos] - no);
    q0 = rowptr[R0];
    q1 = rowptr[R0 + nn];
    deg = (rowptr[R0 + 1] - q0) >> 1;
  }
  for (int k = 0; k < W; ++k) {
    const bool in = has && k < deg;
    const long long d = o0 + 32LL * k + t;
    if (cols) cols[d] = in ? colind[q0 + k] : R0;
    if (!A) continue;
    float e0 = 0, e1 = 0, e2 = 0, e3 = 0;
    if (in) {
      e0 = (float)A[q0 + k];
      e1 = (float)A[q0 + deg + k];
      e2 = (float)A[q1 + k];
      e3 = (float)A[q1 + deg + k];
    }
    vlo[4 * d] = __float2bfloat16_rn(e0); vlo[4 * d + 1] = __float2bfloat16_rn(e1);
    vlo[4 * d + 2] = __float2bfloat16_rn(e2); vlo[4 * d + 3] = __float2bfloat16_rn(e3);
  }
}

// Finest-level row products over the node slices, both rows (u, v) of a node per thread.
//   MODE 0 (PCG SpMV):    out = mask(K x); partial x.out
//   MODE 1 (AMG residual): out = mask(b - K x)                 (systems deeper than level 0)
//   MODE 2 (AMG smoothing): out = mask(x + invd (b - K x)), pcopy = out; partial b.out
// The partials go per slice: part[slice block * kSellSlices + warp].  List-driven when act.cnt is
// set (the CTAs loop over the active slice blocks), else one slice block per CTA.
// The slot loop is unrolled eight deep (a P1 slice's width in one pass), so a thread has eight
// column loads and their gathers in flight.  FP32 vectors: the SpMV (FP32 values) at most 64
// registers, four CTAs per SM; the BF16 passes at most 48, five CTAs per SM; FP64 vectors: the
// compiler's choice.  Measured on B200 (256-mesh batch, algorithmic bytes): three deep at 40
// registers, SpMV 3.41 and smoothing 2.88 TB/s; eight deep, SpMV 4.10 at four CTAs per SM and
// the BF16 passes 3.56 at five.
template <typename KT, typename VT, int MODE>
__global__ void __launch_bounds__(256, sizeof(VT) == 4 ? (MODE == 0 ? 4 : 5) : 0) k_sell(SellDev S, int nsb, ActList act, const int* sel, const int* done,
                                              const int* depth, const KT* vals, const VT* x, const VT* b,
                                              const VT* invd, const unsigned char* cmask, VT* out, VT* pcopy,
                                              double* part) {
  pdl_enter();
  const int nv = act.cnt ? *act.cnt : nsb;
  const int w = threadIdx.x >> 5, t = threadIdx.x & 31, pos = w * 32 + t;
  for (int vb = blockIdx.x; vb < nv; vb += gridDim.x) {
    const int sb = act.map ? act.map[vb] : vb;
    const int s = S.sb_sys[sb];
    const bool live = sel[s] && !done[s] && (MODE == 0 || depth[s] > S.lev);
    if (MODE == 1 && !live) continue;  // uniform over the block
    double pv = 0;
    if (live && pos < S.sb_cnt[sb]) {
      const int sl = sb * kSellSlices + w;
      const long long o0 = S.sl_off[sl];
      const int W = (int)((S.sl_off[sl + 1] - o0) >> 5);
      const int no = S.node_off[s], nn = S.node_off[s + 1] - no;
      const int g = S.perm[S.sb_n0[sb] + pos];
      const int ru = S.dof_off[s] + (g - no), rv = ru + nn;
      // the node's own rows, loaded ahead of the row products
      const bool mu = cmask && cmask[ru], mv = cmask && cmask[rv];
      double xu0 = 0, xv0 = 0, bu0 = 0, bv0 = 0, du = 0, dv = 0;
      if (MODE != 1) { xu0 = to_d(x[ru]); xv0 = to_d(x[rv]); }
      if (MODE != 0) { bu0 = to_d(b[ru]); bv0 = to_d(b[rv]); }
      if (MODE == 2) { du = to_d(invd[ru]); dv = to_d(invd[rv]); }
      const int* cp = S.cols + o0 + t;
      const KT* vp = vals + 4 * (o0 + t);
      double au = 0, av = 0;
#pragma unroll 8
      for (int k = 0; k < W; ++k) {
        int j = __ldg(cp + 32 * k);
        bool okj = true;
        UA_CHECK_INDEX(S.dbg, j, S.dof_off[s], S.dof_off[s] + nn, BS_SELL_COL, okj);
        (void)okj;
        double e[4];
        Quad<KT>::get(vp + 128 * k, e);
        const double xu = to_d(x[j]), xv = to_d(x[j + nn]);
        au = fma(e[0], xu, au);
        au = fma(e[1], xv, au);
        av = fma(e[2], xu, av);
        av = fma(e[3], xv, av);
      }
      if (MODE == 0) {
        const double qu = mu ? 0.0 : au, qv = mv ? 0.0 : av;
        out[ru] = (VT)qu;
        out[rv] = (VT)qv;
        pv = xu0 * qu + xv0 * qv;
      } else if (MODE == 1) {
        out[ru] = (VT)(mu ? 0.0 : bu0 - au);
        out[rv] = (VT)(mv ? 0.0 : bv0 - av);
      } else {
        const double zu = mu ? 0.0 : xu0 + du * (bu0 - au);
        const double zv = mv ? 0.0 : xv0 + dv * (bv0 - av);
        out[ru] = (VT)zu;
        out[rv] = (VT)zv;
        if (pcopy) { pcopy[ru] = (VT)zu; pcopy[rv] = (VT)zv; }
        pv = bu0 * zu + bv0 * zv;
      }
    }
    if (MODE == 1 || !part) continue;  // uniform per launch
    // one partial per slice (a fixed-order warp sum): no CTA barrier, so the warps of the short
    // slices do not wait for the long ones
    double tw = pv;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) tw += __shfl_down_sync(0xffffffffu, tw, o);
    if (t == 0) part[sb * kSellSlices + w] = tw;
  }
}

// ---------------------------------------------------------------------------
// device: smoothed aggregation (P = (I - w D^-1 A) P0, coarse operator P' A P)
// ---------------------------------------------------------------------------
//
// Values are quads (the four entries of a node pair) on node-level lists.  The products that make an
// entry of A P or of the coarse operator are listed once per handle (sa_lists), so a set-up has no
// searches: a lane owns an entry, reads its products and writes it, in a fixed order and without
// atomics.  (Scattering the products of a row into shared memory, with a search per product, issued
// 456 warp instructions per node of P2 401x201; the lists issue about 30.)

__device__ __forceinline__ int sa_find(const int* list, int n, int key) {  // list sorted ascending
  int lo = 0, hi = n;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (list[mid] < key) lo = mid + 1; else hi = mid;
  }
  return lo < n && list[lo] == key ? lo : -1;
}

// ---- lists (once per handle) ----

__global__ void k_sa_nrow(int nn, const int* node_sys, const int* node_off, const int* dof_off, const int* rowptr,
                          int4* nrow) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= nn) return;
  const int s = node_sys[g], no = node_off[s], n = node_off[s + 1] - no, i = dof_off[s] + (g - no);
  nrow[g] = make_int4(rowptr[i], rowptr[i + n], (rowptr[i + 1] - rowptr[i]) >> 1, s);
}
__global__ void k_sa_ids(int nn, const int* ptr, int* node) {
  const int g = (blockIdx.x * blockDim.x + threadIdx.x) >> 2, lane = threadIdx.x & 3;
  if (g >= nn) return;
  for (int e = ptr[g] + lane; e < ptr[g + 1]; e += 4) node[e] = g;
}
// products of A P entry e = (g, J): neighbours h of g with J in P(h); lst = null: counts only
__global__ void k_sa_ap_list(long long n, const int* node, const int* col, const int4* nrow, const int* node_off,
                             const int* dof_off, const int* colind, const int* pn_ptr, const int* pn_col,
                             unsigned* ptr, int2* lst, int* own) {
  const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (e >= n) return;
  const int g = node[e], J = col[e];
  const int4 r = nrow[g];
  const int sh = node_off[r.w] - dof_off[r.w];
  unsigned at = lst ? ptr[e] : 0;
  int p = -1;
  for (int k = 0; k < r.z; ++k) {
    const int h = colind[r.x + k] + sh;
    for (int t = pn_ptr[h]; t < pn_ptr[h + 1]; ++t)
      if (pn_col[t] == J) {
        if (h == g) p = t;
        if (lst) lst[at] = make_int2(k, t);
        ++at;
      }
  }
  if (!lst) ptr[e] = at;
  else own[e] = p;
}
// products of coarse entry o = (J, K): fine nodes g of P'(J) with K in A P(g)
__global__ void k_sa_ac_list(long long n, const int* node, const int* gptr, const int4* nrow_c, const int* node_off,
                             const int* dof_off, const int* colind, const int* ptn_ptr, const int* ptn_fine,
                             const int* ptn_k, const int* pn_ptr, const int* apn_ptr, const int* apn_col,
                             unsigned* ptr, int2* lst) {
  const long long o = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (o >= n) return;
  const int J = node[o];
  const int4 r = nrow_c[J];
  const int K = colind[r.x + (int)(o - gptr[J])] + node_off[r.w] - dof_off[r.w];
  unsigned at = lst ? ptr[o] : 0;
  for (int u = ptn_ptr[J]; u < ptn_ptr[J + 1]; ++u) {
    const int g = ptn_fine[u], a0 = apn_ptr[g];
    const int t = sa_find(apn_col + a0, apn_ptr[g + 1] - a0, K);
    if (t < 0) continue;
    if (lst) lst[at] = make_int2(pn_ptr[g] + ptn_k[u], a0 + t);
    ++at;
  }
  if (!lst) ptr[o] = at;
}
// exclusive scan of v[0..n) in place, the sum in v[n] and total (one CTA of 1024 threads)
__device__ int block_excl_scan(int v, int* sh, int& total);
__global__ void __launch_bounds__(1024) k_sa_scan(long long n, unsigned* v, unsigned long long* total) {
  __shared__ int sh[32];
  constexpr int IT = 8;
  unsigned long long base = 0;
  for (long long b = 0; b < n; b += 1024 * IT) {
    const long long i0 = b + (long long)threadIdx.x * IT;
    int c[IT], sum = 0;
#pragma unroll
    for (int t = 0; t < IT; ++t) {
      c[t] = i0 + t < n ? (int)v[i0 + t] : 0;
      sum += c[t];
    }
    int tot;
    const int ex = block_excl_scan(sum, sh, tot);
    unsigned at = (unsigned)(base + (unsigned)ex);
#pragma unroll
    for (int t = 0; t < IT; ++t)
      if (i0 + t < n) {
        v[i0 + t] = at;
        at += c[t];
      }
    base += (unsigned)tot;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    v[n] = (unsigned)base;
    *total = base;
  }
}

// ---- values ----

// Smoother diagonal and prolongator rows of fine node g, kSaGL lanes per node: the damped l1 diagonal
// invd = kSmoothOmega / sum |a| over unmasked columns (0 on masked or empty rows) with its square root
// sc and, in slice order, its inverse dw for the collapsed cycle; and P(g,:) = P0 - w/l1 A P0 on
// unmasked rows and columns, or the linear interpolation pn_w from the unmasked ones of the corners pn_f: a
// masked corner's error is zero, and where a mid node lies between two of them their columns alone would make
// the coarse operator singular (a 2x2 mesh with its sides held: 40206 iterations instead of 29).  The row's entries are staged in shared
// memory with their neighbours' aggregates; a lane owns an entry of P and takes the neighbours of its
// aggregate in row order.  ST: the type of the sums (FP32 in the mixed-precision form, else FP64).
// One pass over the row instead of an l1 kernel, a scattered P, a repacking and the scaling: latency on
// the coarse levels (P1 141x71, three levels: 113 -> 23 us cold), the row's bytes on large ones (P2
// 401x201, four levels: 276 -> 133 us).
constexpr int kSaGL = 8;
constexpr int kSaStage = 32;  // neighbours staged at a time
template <typename KT, typename VT, typename QT>
__global__ void __launch_bounds__(128) k_sa_P(int nf, const int4* nrow, const int* dof_off, const int* node_off,
                                              const int* colind, const KT* A, const unsigned char* mask,
                                              const int* agg, const int* pn_ptr, const int* pn_col,
                                              const double* pn_w, const int* pn_f, QT* Q, VT* invd, double2* sc, VT* dw,
                                              const int* ipos, const int* sel, const int* psel) {
  using ST = KT;
  __shared__ ST sv[128 / kSaGL][4][kSaStage];
  __shared__ int sj[128 / kSaGL][kSaStage];
  const int gi = threadIdx.x / kSaGL, lane = threadIdx.x % kSaGL;
  const int g = blockIdx.x * (128 / kSaGL) + gi;
  if (g >= nf) return;  // whole groups leave together
  const unsigned gmask = ((1u << kSaGL) - 1u) << ((threadIdx.x & 31) & ~(kSaGL - 1));
  const int4 r = nrow[g];
  const int s = r.w, deg = r.z;
  if (sel && !sel[s]) return;
  const int no = node_off[s], nn = node_off[s + 1] - no, d0 = dof_off[s];
  const int i0 = d0 + (g - no), i1 = i0 + nn;
  const bool m0 = mask && mask[i0], m1 = mask && mask[i1];
  const int pr = pn_ptr[g], dP = pn_ptr[g + 1] - pr, ag = agg[g];
  double l0 = 0, l1 = 0;
  const bool smooth = !pn_w;
  auto stage = [&](int k0) {  // two neighbours a lane at a time, all their loads ahead of the uses
    for (int b = 0; b < kSaStage && k0 + b < deg; b += 2 * kSaGL) {
      int ju[2];
      KT a[2][4];
      bool in[2], cu[2], cv[2];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int k = k0 + b + q * kSaGL + lane;
        in[q] = k < deg;
        const int kc = min(k, deg - 1);
        ju[q] = colind[r.x + kc];
        a[q][0] = A[r.x + kc];
        a[q][1] = A[r.x + deg + kc];
        a[q][2] = A[r.y + kc];
        a[q][3] = A[r.y + deg + kc];
      }
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        cu[q] = mask && mask[ju[q]];
        cv[q] = mask && mask[ju[q] + nn];
        const int c = b + q * kSaGL + lane;
        if (smooth && in[q]) sj[gi][c] = agg[no + (ju[q] - d0)];
      }
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        if (!in[q]) continue;
        const int c = b + q * kSaGL + lane;
        const ST a00 = (m0 || cu[q]) ? ST(0) : a[q][0], a01 = (m0 || cv[q]) ? ST(0) : a[q][1];
        const ST a10 = (m1 || cu[q]) ? ST(0) : a[q][2], a11 = (m1 || cv[q]) ? ST(0) : a[q][3];
        if (smooth) {
          sv[gi][0][c] = a00; sv[gi][1][c] = a01; sv[gi][2][c] = a10; sv[gi][3][c] = a11;
        }
        l0 += fabs((double)a00) + fabs((double)a01);
        l1 += fabs((double)a10) + fabs((double)a11);
      }
    }
  };
  for (int k0 = 0; k0 < deg; k0 += kSaStage) {
    __syncwarp(gmask);
    stage(k0);
  }
#pragma unroll
  for (int o = kSaGL / 2; o > 0; o >>= 1) {
    l0 += __shfl_xor_sync(gmask, l0, o, kSaGL);
    l1 += __shfl_xor_sync(gmask, l1, o, kSaGL);
  }
  const VT v0 = (VT)(l0 > 0 ? kSmoothOmega / l0 : 0.0), v1 = (VT)(l1 > 0 ? kSmoothOmega / l1 : 0.0);
  if (lane == 0) {
    invd[i0] = v0;
    invd[i1] = v1;
    if (sc) sc[g] = make_double2(sqrt((double)v0), sqrt((double)v1));
    if (dw) {
      const size_t k = 2 * (size_t)ipos[g];
      dw[k] = (VT)(v0 > 0 ? 1.0 / (double)v0 : 0.0);
      dw[k + 1] = (VT)(v1 > 0 ? 1.0 / (double)v1 : 0.0);
    }
  }
  if (psel && !psel[s]) return;
  const ST f0 = (ST)(kSaOmega / kSmoothOmega * (double)v0), f1 = (ST)(kSaOmega / kSmoothOmega * (double)v1);
  __syncwarp(gmask);
  for (int t0 = 0; t0 < dP; t0 += kSaGL) {
    const int t = t0 + lane;
    if (pn_w) {  // the same weights for both components, no smoothing
      if (t < dP) {
        const int j0 = d0 + (pn_f[pr + t] - no), j1 = j0 + nn;
        pq_set(Q + pr + t, m0 || (mask && mask[j0]) ? 0.0 : pn_w[pr + t], 0.0, 0.0,
               m1 || (mask && mask[j1]) ? 0.0 : pn_w[pr + t]);
      }
      continue;
    }
    const int J = t < dP ? pn_col[pr + t] : -1;
    ST p00 = (J == ag && !m0) ? ST(1) : ST(0), p11 = (J == ag && !m1) ? ST(1) : ST(0), p01 = 0, p10 = 0;
    for (int k0 = 0; k0 < deg; k0 += kSaStage) {
      if (deg > kSaStage) {
        __syncwarp(gmask);
        stage(k0);
        __syncwarp(gmask);
      }
      const int nk = min(kSaStage, deg - k0);
      for (int c = 0; c < nk; ++c)
        if (sj[gi][c] == J) {
          p00 -= f0 * sv[gi][0][c];
          p01 -= f0 * sv[gi][1][c];
          p10 -= f1 * sv[gi][2][c];
          p11 -= f1 * sv[gi][3][c];
        }
    }
    if (t < dP) pq_set(Q + pr + t, (double)p00, (double)p01, (double)p10, (double)p11);
  }
}

// A P, one lane per entry (g, J).  Masked columns are zero rows of P.  Bound by the gathers of A and
// the product list (8 bytes a product) on large levels: P2 401x201, four levels, 330 -> 137 us; P1
// 141x71, three levels, 37 -> 29 us.
template <typename KT>
__global__ void __launch_bounds__(256) k_sa_AP(long long n, const int* node, const int4* nrow, const int* dof_off,
                                               const int* node_off, const KT* A, const unsigned char* mask,
                                               const typename PQuadOf<KT>::T* Q, const unsigned* lptr,
                                               const int2* lst, KT* AP, const int* sel) {
  using ST = KT;
  const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (e >= n) return;
  const int g = node[e];
  const unsigned u0 = lptr[e], u1 = lptr[e + 1];
  const int4 r = nrow[g];
  if (sel && !sel[r.w]) return;
  bool m0 = false, m1 = false;
  if (mask) {
    const int no = node_off[r.w], i0 = dof_off[r.w] + (g - no);
    m0 = mask[i0];
    m1 = mask[i0 + node_off[r.w + 1] - no];
  }
  ST b00 = 0, b01 = 0, b10 = 0, b11 = 0;
#pragma unroll 4
  for (unsigned u = u0; u < u1; ++u) {
    const int2 c = lst[u];
    double pq[4];
    pq_get(Q + c.y, pq);
    const ST p00 = (ST)pq[0], p01 = (ST)pq[1], p10 = (ST)pq[2], p11 = (ST)pq[3];
    const ST a00 = (ST)A[r.x + c.x], a01 = (ST)A[r.x + r.z + c.x], a10 = (ST)A[r.y + c.x],
             a11 = (ST)A[r.y + r.z + c.x];
    b00 += a00 * p00 + a01 * p10;
    b01 += a00 * p01 + a01 * p11;
    b10 += a10 * p00 + a11 * p10;
    b11 += a10 * p01 + a11 * p11;
  }
  quad_put(AP, e, m0 ? ST(0) : b00, m0 ? ST(0) : b01, m1 ? ST(0) : b10, m1 ? ST(0) : b11);
}

// the same quads in ptn order (coarse node J, its fine nodes u): thread per ptn entry (its
// system is its fine node's); every P entry is the image of exactly one ptn entry
template <typename QT>
__global__ void k_sa_qt(long long np, const int* fnode_sys, const int* ptn_fine, const int* ptn_k,
                        const int* pn_ptr, const QT* Q, QT* QTr, const int* sel) {
  const long long u = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (u >= np) return;
  const int g = ptn_fine[u];
  if (sel && !sel[fnode_sys[g]]) return;
  QTr[u] = Q[pn_ptr[g] + ptn_k[u]];
}

// Coarse operator, kSaAcL lanes per entry (J, K): Ac = sum of P(g, J)' A P(g, K) in FP64, a lane sum in
// a fixed order; the diagonal entries have several times the products of the others.  P2 401x201, four
// levels: 205 -> 121 us; P1 141x71, three levels: 57 -> 31 us.
constexpr int kSaAcL = 4;
template <typename KT>
__global__ void __launch_bounds__(256) k_sa_Ac(long long n, const int* node, const int* gptr, const int4* nrow_c,
                                               const typename PQuadOf<KT>::T* Q, const KT* AP,
                                               const unsigned* lptr, const int2* lst, KT* Ac, const int* sel) {
  const long long o = (blockIdx.x * (long long)blockDim.x + threadIdx.x) / kSaAcL;
  const int lane = threadIdx.x % kSaAcL;
  if (o >= n) return;  // whole groups leave together
  const int J = node[o];
  const unsigned u0 = lptr[o], u1 = lptr[o + 1];
  const int4 r = nrow_c[J];
  if (sel && !sel[r.w]) return;
  const int k = (int)(o - gptr[J]);
  double b00 = 0, b01 = 0, b10 = 0, b11 = 0;
#pragma unroll 4
  for (unsigned u = u0 + lane; u < u1; u += kSaAcL) {
    const int2 c = lst[u];
    double p[4], x[4];
    pq_get(Q + c.x, p);  // P((c,g),(c2,J)) at 2 c + c2
    quad_at(AP, c.y, x);
    b00 += p[0] * x[0] + p[2] * x[2];
    b01 += p[0] * x[1] + p[2] * x[3];
    b10 += p[1] * x[0] + p[3] * x[2];
    b11 += p[1] * x[1] + p[3] * x[3];
  }
  const unsigned gmask = ((1u << kSaAcL) - 1u) << ((threadIdx.x & 31) & ~(kSaAcL - 1));
#pragma unroll
  for (int d = kSaAcL / 2; d > 0; d >>= 1) {
    b00 += __shfl_xor_sync(gmask, b00, d, kSaAcL);
    b01 += __shfl_xor_sync(gmask, b01, d, kSaAcL);
    b10 += __shfl_xor_sync(gmask, b10, d, kSaAcL);
    b11 += __shfl_xor_sync(gmask, b11, d, kSaAcL);
  }
  static_assert(kSaAcL == 4, "a lane writes one of the four values");
  const double v = lane == 0 ? b00 : lane == 1 ? b01 : lane == 2 ? b10 : b11;
  Ac[(lane < 2 ? r.x : r.y) + (lane & 1 ? r.z : 0) + k] = (KT)v;
}

// The transfers are gather chains (list entry -> node block -> P list -> vector entries).  They
// load what a node block needs (its system, its nodes' P lists) ahead of the system's flags, and
// take the entries of a P list in chunks of kSaChunk (half that in FP64): the chunk's columns and
// P quads load together, then its vector entries, then the sums in list order.
constexpr int kSaChunk = 4;

// restriction b_c = P' res (coarse pre-smoothing x_c = invd b_c unless lc is the system's coarsest),
// kSaRL lanes per coarse node: both rows (c2 = 0, 1) of the node share the fine-node list and
// the gathered residuals; a lane sum in a fixed order.  A CTA of 32 kSaRL threads takes one node
// block (kAmgNB = 32 coarse nodes) per pass.
constexpr int kSaRL = 8;
template <typename VT>
__global__ void __launch_bounds__(32 * kSaRL, 4) k_sa_restrict(const int* nb_start, const int* nb_sys, ActList act,
                                                            const int* cdof_off, const int* cnode_off,
                                                            const int* depth, int lc, const int* sel,
                                                            const int* done, const int* ptn_ptr,
                                                            const int* ptn_fine,
                                                            const typename PQuadOf<VT>::T* QTr,
                                                            const int* fdof_off, const int* fnode_off,
                                                            const VT* res, const VT* cinvd, VT* cb, VT* cx) {
  pdl_enter();
  static_assert(kAmgNB == 32, "one coarse node per kSaRL-lane group of a 32 kSaRL-thread CTA");
  constexpr int CH = sizeof(VT) == 4 ? kSaChunk : kSaChunk / 2;  // FP64 chunks held to the register budget
  const int sub = threadIdx.x / kSaRL, lane = threadIdx.x % kSaRL;
  const int nv = act.cnt ? *act.cnt : gridDim.x;  // list entries, else one node block per CTA
  for (int vb = blockIdx.x; vb < nv; vb += gridDim.x) {
    const int b = act.map ? act.map[vb] : vb;
    const int s = nb_sys[b];
    const int J = nb_start[b] + sub;
    const bool valid = J < nb_start[b + 1];
    int tr = 0, t1 = 0;
    if (valid) {  // ahead of the flags
      tr = ptn_ptr[J];
      t1 = ptn_ptr[J + 1];
    }
    if (!sel[s] || done[s]) continue;  // uniform over the block
    const int cno = cnode_off[s], cnn = cnode_off[s + 1] - cno, cd = cdof_off[s];
    const int fno = fnode_off[s], fnn = fnode_off[s + 1] - fno, fd = fdof_off[s];
    const bool presmooth = depth[s] > lc;
    double a0 = 0, a1 = 0;
    for (int u0 = tr + lane; u0 < t1; u0 += kSaRL * CH) {
      int f[CH];
      VT q[CH][4];  // P((c,g),(c2,J)) at 2 c + c2 (BF16 quads widen exactly to FP32)
#pragma unroll
      for (int k = 0; k < CH; ++k) {
        const int u = u0 + k * kSaRL;
        f[k] = -1;
        if (u < t1) {
          f[k] = fd + (ptn_fine[u] - fno);
          pq_get(QTr + u, q[k]);
        }
      }
      VT r0[CH], r1[CH];
#pragma unroll
      for (int k = 0; k < CH; ++k)
        if (f[k] >= 0) {
          r0[k] = res[f[k]];
          r1[k] = res[f[k] + fnn];
        }
#pragma unroll
      for (int k = 0; k < CH; ++k)
        if (f[k] >= 0) {
          a0 += (double)q[k][0] * (double)r0[k] + (double)q[k][2] * (double)r1[k];
          a1 += (double)q[k][1] * (double)r0[k] + (double)q[k][3] * (double)r1[k];
        }
    }
#pragma unroll
    for (int o = kSaRL / 2; o > 0; o >>= 1) {
      a0 += __shfl_down_sync(0xffffffffu, a0, o, kSaRL);
      a1 += __shfl_down_sync(0xffffffffu, a1, o, kSaRL);
    }
    if (valid && lane == 0) {
      const int R0 = cd + (J - cno), R1 = R0 + cnn;
      cb[R0] = (VT)a0;
      cb[R1] = (VT)a1;
      if (presmooth) {
        cx[R0] = (VT)((double)cinvd[R0] * a0);
        cx[R1] = (VT)((double)cinvd[R1] * a1);
      }
    }
  }
}

// prolongation x += P x_c on level l (systems deeper than l; masked rows have zero P rows),
// one thread per fine node of a node block: both rows share the coarse-node list and the gathered x_c
// (one warp per node block of kAmgNB = 32 nodes, kSaPW warps per CTA)
constexpr int kSaPW = 8;
template <typename VT>
__global__ void __launch_bounds__(32 * kSaPW, 4) k_sa_prolong(int nnb, const int* nb_start, const int* nb_sys,
                                                           ActList act, const int* dof_off, const int* node_off,
                                                           const int* depth, int l, const int* sel, const int* done,
                                                           const int* pn_ptr, const int* pn_col,
                                                           const typename PQuadOf<VT>::T* Q, const int* cdof_off,
                                                           const int* cnode_off, const VT* xc,
                                                           VT* x) {
  pdl_enter();
  static_assert(kAmgNB == 32, "one fine node per lane");
  constexpr int CH = sizeof(VT) == 4 ? kSaChunk : kSaChunk / 2;  // FP64 chunks held to the register budget
  const int nv = act.cnt ? *act.cnt : nnb;  // list entries, else every node block
  const int lane = threadIdx.x & 31;
  for (int vb = blockIdx.x * kSaPW + (threadIdx.x >> 5); vb < nv; vb += gridDim.x * kSaPW) {
    const int b = act.map ? act.map[vb] : vb;
    const int s = nb_sys[b];
    const int g = nb_start[b] + lane;
    const bool valid = g < nb_start[b + 1];
    int pr = 0, pe = 0;
    if (valid) {  // ahead of the flags
      pr = pn_ptr[g];
      pe = pn_ptr[g + 1];
    }
    if (!sel[s] || done[s] || depth[s] <= l) continue;  // uniform over the warp
    if (!valid) continue;
    const int cno = cnode_off[s], cnn = cnode_off[s + 1] - cno, cd = cdof_off[s];
    const int no = node_off[s], nn = node_off[s + 1] - no, d0 = dof_off[s];
    const int i0 = d0 + (g - no), i1 = i0 + nn;
    double a0 = (double)x[i0], a1 = (double)x[i1];
    for (int k0 = pr; k0 < pe; k0 += CH) {
      int K[CH];
      VT q[CH][4];  // P((c,g),(c2,K)) at 2 c + c2 (BF16 quads widen exactly to FP32)
#pragma unroll
      for (int k = 0; k < CH; ++k) {
        K[k] = -1;
        if (k0 + k < pe) {
          K[k] = cd + (pn_col[k0 + k] - cno);
          pq_get(Q + k0 + k, q[k]);
        }
      }
      VT xu[CH], xv[CH];
#pragma unroll
      for (int k = 0; k < CH; ++k)
        if (K[k] >= 0) {
          xu[k] = xc[K[k]];
          xv[k] = xc[K[k] + cnn];
        }
#pragma unroll
      for (int k = 0; k < CH; ++k)
        if (K[k] >= 0) {
          a0 += (double)q[k][0] * (double)xu[k] + (double)q[k][1] * (double)xv[k];
          a1 += (double)q[k][2] * (double)xu[k] + (double)q[k][3] * (double)xv[k];
        }
    }
    x[i0] = (VT)a0;
    x[i1] = (VT)a1;
  }
}

// ---------------------------------------------------------------------------
// host drivers
// ---------------------------------------------------------------------------

// The lists of a smoothed hierarchy's set-up, once per handle.
static int sa_lists(ua_mesh* m, const int* rowptr0, const int* colind0) {
  Amg* a = m->amg;
  cudaStream_t st = m->stream;
  const size_t mark = m->owned.size(), bytes = a->bytes;
  bool ok = true;
  auto grid = [](long long n, int t) { return (unsigned)std::max<long long>(1, (n + t - 1) / t); };
  unsigned long long* d_tot = (unsigned long long*)dalloc(m, a, sizeof(unsigned long long), ok);
  for (int l = 0; ok && l < a->nlev; ++l) {
    AmgLevel& L = a->lev[l];
    L.nrow = (int4*)dalloc(m, a, sizeof(int4) * (size_t)std::max(L.nn, 1), ok);
    if (ok && L.nn)
      k_sa_nrow<<<grid(L.nn, 256), 256, 0, st>>>(L.nn, L.node_sys, L.d_node_off, L.d_dof_off,
                                                 l == 0 ? rowptr0 : L.rowptr, L.nrow);
  }
  // counts, offsets, products: fill(lst) launches the list kernel
  auto build = [&](long long n, unsigned*& ptr, int2*& lst, auto fill) -> int {
    ptr = (unsigned*)dalloc(m, a, sizeof(unsigned) * (size_t)(n + 1), ok);
    if (!ok) return UA_ERR_OOM;
    fill((int2*)nullptr);
    k_sa_scan<<<1, 1024, 0, st>>>(n, ptr, d_tot);
    unsigned long long tot = 0;
    UA_CUDA_TRY(cudaMemcpyAsync(&tot, d_tot, sizeof(tot), cudaMemcpyDeviceToHost, st));
    UA_CUDA_TRY(cudaStreamSynchronize(st));
    if (tot > 0xffffffffull) return UA_ERR_OOM;  // 34 GB of products
    lst = (int2*)dalloc(m, a, sizeof(int2) * (size_t)std::max<unsigned long long>(tot, 1), ok);
    if (!ok) return UA_ERR_OOM;
    fill(lst);
    return UA_OK;
  };
  for (int l = 0; ok && l + 1 < a->nlev; ++l) {
    AmgLevel& F = a->lev[l];
    const AmgLevel& C = a->lev[l + 1];
    F.ap_node = (int*)dalloc(m, a, sizeof(int) * (size_t)std::max(F.nap, 1LL), ok);
    F.ap_p = (int*)dalloc(m, a, sizeof(int) * (size_t)std::max(F.nap, 1LL), ok);
    F.ac_node = (int*)dalloc(m, a, sizeof(int) * (size_t)std::max(C.ng, 1LL), ok);
    if (!ok) break;
    k_sa_ids<<<grid(4LL * F.nn, 256), 256, 0, st>>>(F.nn, F.apn_ptr, F.ap_node);
    k_sa_ids<<<grid(4LL * C.nn, 256), 256, 0, st>>>(C.nn, C.gptr, F.ac_node);
    int rc = build(F.nap, F.ap_lptr, F.ap_l, [&](int2* lst) {
      k_sa_ap_list<<<grid(F.nap, 256), 256, 0, st>>>(F.nap, F.ap_node, F.apn_col, F.nrow, F.d_node_off, F.d_dof_off,
                                                     l == 0 ? colind0 : F.colind, F.pn_ptr, F.pn_col, F.ap_lptr,
                                                     lst, F.ap_p);
    });
    if (!rc)
      rc = build(C.ng, F.ac_lptr, F.ac_l, [&](int2* lst) {
        k_sa_ac_list<<<grid(C.ng, 256), 256, 0, st>>>(C.ng, F.ac_node, C.gptr, C.nrow, C.d_node_off, C.d_dof_off,
                                                      C.colind, F.ptn_ptr, F.ptn_fine, F.ptn_k, F.pn_ptr, F.apn_ptr,
                                                      F.apn_col, F.ac_lptr, lst);
      });
    if (rc == UA_ERR_OOM) ok = false;
    else if (rc) return rc;
  }
  if (!ok) {  // the next set-up starts over
    dev_free_since(m, mark);
    a->bytes = bytes;
    return set_error(UA_ERR_OOM, "AMG: device allocation of the set-up lists failed");
  }
  UA_CUDA_TRY(cudaGetLastError());
  a->lists = true;
  return UA_OK;
}

// cyc: also the values of the collapsed cycle; branch: run them beside the coarse levels (a capture)
template <typename KT, typename VT>
static int numeric_t(ua_mesh* m, const int* rowptr0, const int* colind0, const KT* K0, const unsigned char* cmask,
                     const int* sel, const int* psel, const CycFillReq* cyc, bool branch, long long* launches) {
  Amg* a = m->amg;
  cudaStream_t st = m->stream, sd = branch ? a->side : st;
  auto l1 = [&](int l) {
    const AmgLevel& L = a->lev[l];
    k_amg_l1<KT, VT><<<(L.ndof + 255) / 256, 256, 0, st>>>(
        L.ndof, l == 0 ? rowptr0 : L.rowptr, l == 0 ? colind0 : L.colind, l == 0 ? K0 : (const KT*)L.A,
        l == 0 ? cmask : nullptr, (VT*)L.invd, L.dof_sys, sel), ++*launches;
  };
  if (a->sa) {
    auto grid = [](long long n, int t) { return (unsigned)std::max<long long>(1, (n + t - 1) / t); };
    // the mixed form sums in FP32, the FP64 form in FP64 (the coarse operators in FP64 in both)
    using QT = typename PQuadOf<KT>::T;
    // per level: smoother diagonal and smoothed prolongator, A P, coarse operator
    for (int l = 0; l + 1 < a->nlev; ++l) {
      AmgLevel& F = a->lev[l];
      AmgLevel& C = a->lev[l + 1];
      const int* ci = l == 0 ? colind0 : F.colind;
      const KT* A = l == 0 ? K0 : (const KT*)F.A;
      const unsigned char* mk = l == 0 ? cmask : nullptr;
      KT* APv = (KT*)F.sa_ap;
      QT* Qv = (QT*)(sizeof(KT) == 4 ? F.sa_qh : F.sa_qd);
      k_sa_P<KT, VT, QT><<<grid((long long)F.nn * kSaGL, 128), 128, 0, st>>>(
          F.nn, F.nrow, F.d_dof_off, F.d_node_off, ci, A, mk, F.sa_agg, F.pn_ptr, F.pn_col, F.pn_w, F.pn_f, Qv, (VT*)F.invd,
          cyc ? a->cyc.lev[l].sc : nullptr, cyc && l == 0 ? (VT*)cyc->dw : nullptr, a->cyc.d_ipos, sel, psel),
          ++*launches;
      if (cyc && l == 0) {  // the finest level's slice values need its diagonal only
        if (branch) {
          UA_CUDA_TRY(cudaEventRecord(a->fork, st));
          UA_CUDA_TRY(cudaStreamWaitEvent(sd, a->fork, 0));
        }
        cycle_fill_fine(m, colind0, K0, sizeof(KT) == 4, cyc->lo, sel, sd, launches);
      }
      if (!cyc)
        k_sa_qt<QT><<<grid(F.np, 256), 256, 0, st>>>(F.np, F.node_sys, F.ptn_fine, F.ptn_k, F.pn_ptr, Qv,
                                                     (QT*)(sizeof(KT) == 4 ? F.sa_qth : F.sa_qtd), sel), ++*launches;
      k_sa_AP<KT><<<grid(F.nap, 256), 256, 0, st>>>(F.nap, F.ap_node, F.nrow, F.d_dof_off, F.d_node_off, A, mk, Qv,
                                                    F.ap_lptr, F.ap_l, APv, sel), ++*launches;
      if (cyc && l + 2 == a->nlev) {  // every diagonal and A P is there
        if (branch) {
          UA_CUDA_TRY(cudaEventRecord(a->fork, st));
          UA_CUDA_TRY(cudaStreamWaitEvent(sd, a->fork, 0));
        }
        cycle_fill_levels(m, sizeof(KT) == 4, cyc->lo, sel, sd, launches);
      }
      k_sa_Ac<KT><<<grid(C.ng * kSaAcL, 256), 256, 0, st>>>(C.ng, F.ac_node, C.gptr, C.nrow, Qv, APv, F.ac_lptr,
                                                            F.ac_l, (KT*)C.A, sel), ++*launches;
    }
  } else {
    for (int l = 0; l + 1 < a->nlev; ++l) {
      const AmgLevel& F = a->lev[l];
      const AmgLevel& C = a->lev[l + 1];
      k_amg_galerkin<KT><<<(C.ndof + 127) / 128, 128, 0, st>>>(
          C.ndof, C.mptr, C.mlist, l == 0 ? rowptr0 : F.rowptr, l == 0 ? colind0 : F.colind,
          l == 0 ? K0 : (const KT*)F.A, F.cmap, l == 0 ? cmask : nullptr, C.rowptr, C.colind, (KT*)C.A), ++*launches;
    }
    for (int l = 0; l < a->nlev; ++l) l1(l);
  }
  const int sm = (int)(sizeof(double) * (size_t)a->maxdn * a->maxdn);  // attribute set by the caller
  k_amg_dense_inverse<KT><<<a->nsys, kDiThreads, sm, st>>>(a->d_depth, a->d_dn, a->d_doff, a->d_lev_rowptr,
                                                     a->d_lev_colind, a->d_lev_A, a->d_lev_dofoff, a->dense, sel),
      ++*launches;
  if (cyc && branch) {
    UA_CUDA_TRY(cudaEventRecord(a->join, sd));
    UA_CUDA_TRY(cudaStreamWaitEvent(st, a->join, 0));
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return set_error(UA_ERR_CUDA, "AMG numeric phase: %s", cudaGetErrorString(e));
  return UA_OK;
}

static SellDev sell_dev(const ua_mesh* m, const Sell& S) {
  return SellDev{S.sb_sys, S.sb_n0, S.sb_cnt, S.perm, S.sl_off, S.cols,
                 m->dm.sys_dof_off, m->dm.sys_node_off, m->dm.dbg, 0};
}
static SellDev csell_dev(const ua_mesh* m, const Sell& S, const AmgLevel& L, int l) {
  return SellDev{S.sb_sys, S.sb_n0, S.sb_cnt, S.perm, S.sl_off, S.cols,
                 L.d_dof_off, L.d_node_off, m->dm.dbg, l};
}

// Node slices of the coarse levels that run a residual and a smoothing pass (1 .. nlev-2) and
// hold at least kCsellMinNodes nodes (below that the CSR row blocks, finer-grained than the slice
// blocks of 256 nodes, spread better over the SMs): per system, blocks of kSellNodes nodes
// ordered by decreasing degree, slices of 32 (the finest level's layout; node degrees from the
// level's CSR).
constexpr int kCsellMinNodes = 131072;
static void csell_init(ua_mesh* m) {
  Amg* a = m->amg;
  const int nsys = a->nsys;
  a->csell.assign(std::max(a->nlev, 1), Sell());
  for (int l = 1; l + 1 < a->nlev; ++l) {
    AmgLevel& L = a->lev[l];
    Sell& S = a->csell[l];
    if (L.nn < kCsellMinNodes) continue;
    std::vector<int> rowptr(L.ndof + 1);
    if (dev_read(m, rowptr.data(), L.rowptr, sizeof(int) * rowptr.size()) != cudaSuccess) {
      S.failed = true;
      return;
    }
    std::vector<int> sb_sys, sb_n0, sb_cnt, perm(std::max(L.nn, 1)), idx;
    std::vector<long long> sl_off(1, 0);
    S.h_sys_sb_off.assign(nsys + 1, 0);
    for (int s = 0; s < nsys; ++s) {
      const int no = L.node_off[s], nn = L.node_off[s + 1] - no, d0 = L.dof_off[s];
      auto deg = [&](int g) { return (rowptr[d0 + (g - no) + 1] - rowptr[d0 + (g - no)]) >> 1; };
      for (int n0 = no; n0 < no + nn; n0 += kSellNodes) {
        const int cnt = std::min(kSellNodes, no + nn - n0);
        idx.resize(cnt);
        for (int k = 0; k < cnt; ++k) idx[k] = n0 + k;
        std::stable_sort(idx.begin(), idx.end(), [&](int p, int q) { return deg(p) > deg(q); });
        for (int k = 0; k < cnt; ++k) perm[n0 + k] = idx[k];
        for (int j = 0; j < kSellSlices; ++j) {
          int W = 0;
          for (int k = j * 32; k < std::min(cnt, j * 32 + 32); ++k) W = std::max(W, deg(idx[k]));
          sl_off.push_back(sl_off.back() + 32LL * W);
        }
        sb_sys.push_back(s);
        sb_n0.push_back(n0);
        sb_cnt.push_back(cnt);
      }
      S.h_sys_sb_off[s + 1] = (int)sb_sys.size();
    }
    bool ok = true;
    S.nsb = (int)sb_sys.size();
    S.slots = sl_off.back();
    S.sb_sys = upload(m, a, sb_sys, ok);
    S.sb_n0 = upload(m, a, sb_n0, ok);
    S.sb_cnt = upload(m, a, sb_cnt, ok);
    S.perm = upload(m, a, perm, ok);
    S.sl_off = upload(m, a, sl_off, ok);
    S.cols = (int*)dalloc(m, a, sizeof(int) * (size_t)S.slots, ok);
    S.vlo = (__nv_bfloat16*)dalloc(m, a, sizeof(__nv_bfloat16) * 4 * (size_t)S.slots, ok);
    if (!ok) { S.failed = true; return; }
    if (S.nsb)
      k_csell_fill<float><<<S.nsb, 256, 0, m->stream>>>(csell_dev(m, S, L, l), L.rowptr, L.colind, nullptr,
                                                       nullptr, S.cols, nullptr);
    if (cudaGetLastError() != cudaSuccess) { S.failed = true; return; }
    S.ready = true;
  }
}

int amg_sell_init(ua_mesh* m, const std::vector<int>& sys_rb_off0) {
  Amg* a = m->amg;
  if (!a || m->h_nodeptr.empty()) return UA_ERR_INVALID;
  Sell& S = a->sell;
  if (S.ready) return UA_OK;
  if (S.failed) return UA_ERR_INVALID;
  const int nsys = a->nsys;
  if ((int)sys_rb_off0.size() != nsys + 1) { S.failed = true; return UA_ERR_INVALID; }
  std::vector<int> sb_sys, sb_n0, sb_cnt, perm(m->nn_total), idx;
  std::vector<long long> sl_off(1, 0);
  S.h_sys_sb_off.assign(nsys + 1, 0);
  auto deg = [&](int g) { return m->h_nodeptr[g + 1] - m->h_nodeptr[g]; };
  for (int s = 0; s < nsys; ++s) {
    const int no = m->h_node_off[s], nn = m->h_node_off[s + 1] - no;
    const int nbc = (nn + kSellNodes - 1) / kSellNodes;
    // the handle's row blocks must be the u blocks then the v blocks of kSellNodes rows each
    if (m->ndof == 2 && (sys_rb_off0[s + 1] - sys_rb_off0[s] != 2 * nbc || 2 * nn != m->h_dof_off[s + 1] - m->h_dof_off[s])) {
      S.failed = true;
      return set_error(UA_ERR_INVALID, "node slices: row blocks of system %d do not split at the u/v boundary", s);
    }
    for (int i = 0; i < nbc; ++i) {
      const int n0 = no + i * kSellNodes, cnt = std::min(kSellNodes, nn - i * kSellNodes);
      idx.resize(cnt);
      for (int k = 0; k < cnt; ++k) idx[k] = n0 + k;
      std::stable_sort(idx.begin(), idx.end(), [&](int p, int q) { return deg(p) > deg(q); });
      for (int k = 0; k < cnt; ++k) perm[n0 + k] = idx[k];
      for (int j = 0; j < kSellSlices; ++j) {
        int W = 0;
        for (int k = j * 32; k < std::min(cnt, j * 32 + 32); ++k) W = std::max(W, deg(idx[k]));
        sl_off.push_back(sl_off.back() + 32LL * W);
      }
      sb_sys.push_back(s);
      sb_n0.push_back(n0);
      sb_cnt.push_back(cnt);
    }
    S.h_sys_sb_off[s + 1] = (int)sb_sys.size();
  }
  bool ok = true;
  S.nsb = (int)sb_sys.size();
  S.slots = sl_off.back();
  S.sb_sys = upload(m, a, sb_sys, ok);
  S.sb_n0 = upload(m, a, sb_n0, ok);
  S.sb_cnt = upload(m, a, sb_cnt, ok);
  S.perm = upload(m, a, perm, ok);
  S.h_perm = perm;
  S.h_sl_off = sl_off;
  S.sl_off = upload(m, a, sl_off, ok);
  if (m->ndof == 2) S.cols = (int*)dalloc(m, a, sizeof(int) * (size_t)S.slots, ok);
  S.spart = (double*)dalloc(m, a, sizeof(double) * kSellSlices * (size_t)std::max(S.nsb, 1), ok);
  std::vector<int> sl_pre(nsys + 1);
  for (int s = 0; s <= nsys; ++s) sl_pre[s] = kSellSlices * S.h_sys_sb_off[s];
  S.sys_sl_off = upload(m, a, sl_pre, ok);
  if (!ok) { S.failed = true; return set_error(UA_ERR_OOM, "node slices: device allocation failed"); }
  if (S.nsb && m->ndof == 2)
    k_sell_fill<double><<<S.nsb, 256, 0, m->stream>>>(sell_dev(m, S), m->dm, nullptr, nullptr, nullptr, S.cols,
                                                       nullptr);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { S.failed = true; return set_error(UA_ERR_CUDA, "node slices: %s", cudaGetErrorString(e)); }
  S.ready = true;
  return UA_OK;
}

int amg_sell_fill(ua_mesh* m, const void* K0, bool fp32, bool lo, long long* launches, const int* sel) {
  Amg* a = m->amg;
  if (!a || !a->sell.ready) return UA_ERR_INVALID;
  Sell& S = a->sell;
  if (a->sa && lo && !a->csell_tried) {  // the coarse levels keep their CSR passes if this fails
    a->csell_tried = true;
    csell_init(m);
  }
  bool ok = true;
  const size_t nv = 4 * (size_t)S.slots;
  if (fp32 && !S.v32) S.v32 = (float*)dalloc(m, a, sizeof(float) * nv, ok);
  if (!fp32 && !S.v64) S.v64 = (double*)dalloc(m, a, sizeof(double) * nv, ok);
  if (lo && !S.vlo) S.vlo = (__nv_bfloat16*)dalloc(m, a, sizeof(__nv_bfloat16) * nv, ok);
  if (!ok) return set_error(UA_ERR_OOM, "node slices: device allocation of the values failed");
  if (!S.nsb) return UA_OK;
  if (fp32)
    k_sell_fill<float><<<S.nsb, 256, 0, m->stream>>>(sell_dev(m, S), m->dm, (const float*)K0, S.v32,
                                                      lo ? S.vlo : nullptr, nullptr, sel);
  else
    k_sell_fill<double><<<S.nsb, 256, 0, m->stream>>>(sell_dev(m, S), m->dm, (const double*)K0, S.v64,
                                                       lo ? S.vlo : nullptr, nullptr, sel);
  ++*launches;
  if (lo && fp32)  // the coarse operators of this Newton step's set-up (FP32) into their BF16 slices
    for (int l = 1; l < (int)a->csell.size(); ++l) {
      const Sell& C = a->csell[l];
      if (!C.ready || !C.nsb) continue;
      const AmgLevel& L = a->lev[l];
      k_csell_fill<float><<<C.nsb, 256, 0, m->stream>>>(csell_dev(m, C, L, l), L.rowptr, L.colind,
                                                       (const float*)L.A, C.vlo, nullptr, sel), ++*launches;
    }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return set_error(UA_ERR_CUDA, "node slices: %s", cudaGetErrorString(e));
  return UA_OK;
}

// Grid of a slice kernel: one slice block per CTA, or, list-driven, the CTAs resident at once
// (per-instantiation occupancy, so that no partial second wave trails the list loop).
template <typename KT, typename VT, int MODE>
static int sell_grid(const Amg* a, bool listed, int nsb = -1) {
  if (nsb < 0) nsb = a->sell.nsb;
  if (!listed) return nsb;
  static int occ = 0;
  if (!occ && (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_sell<KT, VT, MODE>, 256, 0) != cudaSuccess ||
               occ < 1))
    occ = 1;
  return std::max(1, std::min(nsb, occ * a->nsm));
}

void amg_sell_partials(const ua_mesh* m, const double** spart, const int** sys_sl_off) {
  *spart = m->amg->sell.spart;
  *sys_sl_off = m->amg->sell.sys_sl_off;
}

int amg_sell_spmv(ua_mesh* m, bool fp32, bool act, const int* sel, const int* done, const void* p,
                  const unsigned char* cmask, void* q, long long* launches) {
  Amg* a = m->amg;
  const Sell& S = a->sell;
  const bool useact = act && S.act.map;
  const ActList L = useact ? S.act : ActList{};
  if (!S.nsb) return UA_OK;
  if (fp32)
    launch_pdl(k_sell<float, float, 0>, sell_grid<float, float, 0>(a, useact), 256, 0, m->stream, sell_dev(m, S), S.nsb, L, sel, done, a->d_depth, S.v32,
                                                         (const float*)p, nullptr, nullptr, cmask, (float*)q,
                                                         nullptr, S.spart);
  else
    launch_pdl(k_sell<double, double, 0>, sell_grid<double, double, 0>(a, useact), 256, 0, m->stream, sell_dev(m, S), S.nsb, L, sel, done, a->d_depth, S.v64,
                                                           (const double*)p, nullptr, nullptr, cmask, (double*)q,
                                                           nullptr, S.spart);
  ++*launches;
  return UA_OK;
}

const void* amg_bf16_copy(ua_mesh* m, const float* K0, long long nnz, long long* launches) {
  Amg* a = m->amg;
  if (!a) return nullptr;
  if (!a->k0lo) {
    a->k0lo = (__nv_bfloat16*)dev_alloc(m, sizeof(__nv_bfloat16) * (size_t)std::max(nnz, 1LL));
    if (!a->k0lo) return nullptr;
    a->bytes += sizeof(__nv_bfloat16) * (size_t)nnz;
  }
  k_to_bf16<<<1184, 256, 0, m->stream>>>(nnz, K0, a->k0lo), ++*launches;
  return a->k0lo;
}

int amg_numeric(ua_mesh* m, const int* rowptr0, const int* colind0, const void* K0, bool fp32,
                const unsigned char* cmask, long long* launches, const int* sel, const std::vector<int>* h_sel,
                int p_refresh, bool graph, const CycFillReq* cyc) {
  // prolongators: recomputed for the selected systems on the first set-up of their solve and then
  // every p_refresh-th one (all of them when no host selection is given)
  Amg* a = m->amg;
  const int* psel = sel;
  if (a && a->sa && h_sel && p_refresh > 1) {
    const int ns = a->nsys;
    if ((int)a->p_age.size() != ns) a->p_age.assign(ns, 0);
    a->h_prefresh.assign(ns, 0);
    for (int s = 0; s < ns; ++s) {
      if (!(*h_sel)[s]) continue;
      a->h_prefresh[s] = a->p_age[s] % p_refresh == 0 ? 1 : 0;
      a->p_age[s] += 1;
    }
    bool ok = true;
    if (!a->d_prefresh) a->d_prefresh = (int*)dalloc(m, a, sizeof(int) * ns, ok);
    if (!ok) return set_error(UA_ERR_OOM, "AMG: device allocation failed");
    // the pinned copies alternate, so that one is rewritten two set-ups later (a Newton step drains
    // the stream in between)
    if (!a->h_pin && cudaMallocHost(&a->h_pin, 2 * sizeof(int) * ns) != cudaSuccess)
      return set_error(UA_ERR_OOM, "AMG: pinned host allocation failed");
    int* hp = a->h_pin + (a->pin_at ^= 1) * ns;
    std::copy(a->h_prefresh.begin(), a->h_prefresh.end(), hp);
    UA_CUDA_TRY(cudaMemcpyAsync(a->d_prefresh, hp, sizeof(int) * ns, cudaMemcpyHostToDevice, m->stream));
    psel = a->d_prefresh;
  }
  constexpr int sm = sizeof(double) * kAmgMaxDense * kAmgMaxDense;  // a constant: the attribute is the process's
  if (fp32)
    UA_CUDA_TRY(cudaFuncSetAttribute(k_amg_dense_inverse<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm));
  else
    UA_CUDA_TRY(cudaFuncSetAttribute(k_amg_dense_inverse<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm));
  if (a->sa && !a->lists)
    if (int rc = sa_lists(m, rowptr0, colind0)) return rc;
  if (a->sa) {  // the transfer quads of this precision, allocated before any capture
    bool ok = true;
    for (int l = 0; l + 1 < a->nlev; ++l) {
      AmgLevel& F = a->lev[l];
      void*& q = fp32 ? F.sa_qh : F.sa_qd;
      void*& qt = fp32 ? F.sa_qth : F.sa_qtd;
      const size_t qb = fp32 ? sizeof(PQuadH) : sizeof(PQuadD);
      if (!q) q = dalloc(m, a, qb * (size_t)std::max(F.np, 1LL), ok);
      if (!qt && !cyc) qt = dalloc(m, a, qb * (size_t)std::max(F.np, 1LL), ok);
    }
    if (!ok) return set_error(UA_ERR_OOM, "AMG: device allocation of the transfer values failed");
  }
  if (a->sa && cyc && graph && !a->side) {
    UA_CUDA_TRY(cudaStreamCreateWithFlags(&a->side, cudaStreamNonBlocking));
    UA_CUDA_TRY(cudaEventCreateWithFlags(&a->fork, cudaEventDisableTiming));
    UA_CUDA_TRY(cudaEventCreateWithFlags(&a->join, cudaEventDisableTiming));
  }
  auto run = [&](long long* l) {
    return fp32 ? numeric_t<float, float>(m, rowptr0, colind0, (const float*)K0, cmask, sel, psel, cyc, graph, l)
                : numeric_t<double, double>(m, rowptr0, colind0, (const double*)K0, cmask, sel, psel, cyc, graph, l);
  };
  if (!graph) return run(launches);
  // one captured graph per kind of call (FP32/FP64 values, prolongator selection, handle's
  // selection), replayed at every later Newton step
  const int key = (fp32 ? 1 : 0) + (psel == a->d_prefresh && psel ? 2 : 0) + (sel ? 4 : 0) + (cyc ? 8 : 0) +
                  (cyc && cyc->lo ? 16 : 0);
  if (!a->setup_exec[key]) {
    long long n = 0;
    cudaGraph_t gr = nullptr;
    UA_CUDA_TRY(cudaStreamBeginCapture(m->stream, cudaStreamCaptureModeThreadLocal));
    int rc = run(&n);
    cudaError_t ce = cudaStreamEndCapture(m->stream, &gr);
    if (rc) { if (gr) cudaGraphDestroy(gr); return rc; }
    if (ce != cudaSuccess) return set_error(UA_ERR_CUDA, "AMG set-up graph capture: %s", cudaGetErrorString(ce));
    ce = cudaGraphInstantiate(&a->setup_exec[key], gr, 0);
    cudaGraphDestroy(gr);
    if (ce != cudaSuccess) return set_error(UA_ERR_CUDA, "AMG set-up graph: %s", cudaGetErrorString(ce));
    a->setup_nodes[key] = n;
  }
  UA_CUDA_TRY(cudaGraphLaunch(a->setup_exec[key], m->stream));
  *launches += a->setup_nodes[key];
  return UA_OK;
}

void amg_restart_P(ua_mesh* m, const std::vector<int>& run) {
  Amg* a = m->amg;
  if (!a) return;
  if ((int)a->p_age.size() != a->nsys) a->p_age.assign(a->nsys, 0);
  for (int s = 0; s < a->nsys && s < (int)run.size(); ++s)
    if (run[s]) a->p_age[s] = 0;
}

// the transfer quads of the vector precision
template <typename VT>
static const typename PQuadOf<VT>::T* sa_quads(void* qd, void* qh) {
  return (const typename PQuadOf<VT>::T*)(std::is_same<VT, float>::value ? qh : qd);
}

// Finest-level residual (MODE 1: W = mask(r - K x0)) or smoothing (MODE 2: z = mask(x + invd (r - K x)),
// pcopy, partials r.z) over the node slices, with BF16 values when v.sell_lo.
template <typename KT, typename VT, int MODE>
static void sell_pass(ua_mesh* m, const AmgPcgView& v, bool useact, const VT* invd, VT* out) {
  Amg* a = m->amg;
  const Sell& S = a->sell;
  if (!S.nsb) return;
  const bool la = useact && S.act.map;
  const ActList L = la ? S.act : ActList{};
  const VT* x = (const VT*)v.x0;
  VT* pcopy = MODE == 2 ? (VT*)v.pcopy : nullptr;
  double* part = MODE == 2 ? S.spart : nullptr;
  const VT* b = (const VT*)v.r;
  const KT* vk = nullptr;
  if constexpr (std::is_same<KT, float>::value) vk = S.v32;
  else vk = S.v64;
  if (v.sell_lo)
    launch_pdl(k_sell<__nv_bfloat16, VT, MODE>, sell_grid<__nv_bfloat16, VT, MODE>(a, la), 256, 0, m->stream, sell_dev(m, S), S.nsb, L, v.sel, v.done, a->d_depth,
                                                                 S.vlo, x, b, invd, v.cmask, out, pcopy, part);
  else
    launch_pdl(k_sell<KT, VT, MODE>, sell_grid<KT, VT, MODE>(a, la), 256, 0, m->stream, sell_dev(m, S), S.nsb, L, v.sel, v.done, a->d_depth, vk, x, b,
                                                      invd, v.cmask, out, pcopy, part);
}

// Coarse-level residual (MODE 1) or smoothing (MODE 2, no partials) over level l's BF16 node slices.
template <typename VT, int MODE>
static void csell_pass(ua_mesh* m, const AmgPcgView& v, int l, bool useact, const VT* x, const VT* b,
                       const VT* invd, VT* out) {
  Amg* a = m->amg;
  const Sell& S = a->csell[l];
  if (!S.nsb) return;
  const bool la = useact && S.act.map;
  const ActList L = la ? S.act : ActList{};
  launch_pdl(k_sell<__nv_bfloat16, VT, MODE>, sell_grid<__nv_bfloat16, VT, MODE>(a, la, S.nsb), 256, 0, m->stream, csell_dev(m, S, a->lev[l], l), S.nsb, L, v.sel, v.done, a->d_depth, S.vlo, x, b, invd, nullptr, out, nullptr,
      nullptr);
}

template <typename KT, typename VT>
static int vcycle_t(ua_mesh* m, const AmgPcgView& v, long long* launches) {
  Amg* a = m->amg;
  cudaStream_t st = m->stream;
  const int nl = a->nlev;
  // per level l: row blocks, matrix, rhs b, pre-smoothed x, residual / post-smoothed buffer
  auto rbs = [&](int l) { return l == 0 ? v.rb_start0 : a->lev[l].rb_start; };
  auto rbsys = [&](int l) { return l == 0 ? v.rb_sys0 : a->lev[l].rb_sys; };
  auto nrb = [&](int l) { return l == 0 ? v.nrb0 : a->lev[l].nrb; };
  auto rp = [&](int l) { return l == 0 ? v.rowptr0 : a->lev[l].rowptr; };
  auto ci = [&](int l) { return l == 0 ? v.colind0 : a->lev[l].colind; };
  auto A = [&](int l) { return l == 0 ? (const KT*)v.K0 : (const KT*)a->lev[l].A; };
  auto B = [&](int l) { return l == 0 ? (const VT*)v.r : (const VT*)a->lev[l].b; };
  auto X = [&](int l) { return l == 0 ? (VT*)v.x0 : (VT*)a->lev[l].x; };
  auto W = [&](int l) { return l == 0 ? (VT*)v.tmp : (VT*)a->lev[l].x2; };
  auto mask = [&](int l) { return l == 0 ? v.cmask : nullptr; };
  auto doff = [&](int l) { return (const int*)a->lev[l].d_dof_off; };
  const int lpr0 = v.lpr, lprc = a->sa ? kSaLPR : 1;  // lanes per row: finest level, coarse levels
  // list-driven launches (the PCG of a uv handle): a grid of about one wave over the active blocks
  const bool useact = v.act && a->act_ready;
  auto rows_act = [&](int l) { return useact ? a->rows[l] : ActList{}; };
  auto rows_grid = [&](int l) { return useact ? act_grid(nrb(l), a->nsm) : nrb(l); };
  // coarse levels on BF16 node slices: the mixed-precision cycle with node slices at the finest level
  auto cslices = [&](int l) { return v.sell && v.sell_lo && l < (int)a->csell.size() && a->csell[l].ready; };
  for (int l = 0; l + 1 < nl; ++l) {  // down: residual of level l, aggregated into level l+1
    const AmgLevel& C = a->lev[l + 1];
    if (l == 0 && v.mark) v.mark(v.mark_ctx, 0, 0);
    if (l == 0 && v.sell)
      sell_pass<KT, VT, 1>(m, v, useact, (const VT*)nullptr, W(0));
    else if (l > 0 && cslices(l))
      csell_pass<VT, 1>(m, v, l, useact, X(l), B(l), nullptr, W(l));
    else
    dispatch_lpr(l == 0 ? lpr0 : lprc, [&](auto L) {
      if (l == 0 && v.K0lo)
        launch_pdl(k_amg_residual<__nv_bfloat16, VT, decltype(L)::value>, rows_grid(l), 256, 0, st, rbs(l), rbsys(l), rows_act(l), v.sel, v.done, a->d_depth, l, rp(l), ci(l), (const __nv_bfloat16*)v.K0lo, B(l), X(l),
            mask(l), W(l), doff(l));
      else
        launch_pdl(k_amg_residual<KT, VT, decltype(L)::value>, rows_grid(l), 256, 0, st, rbs(l), rbsys(l), rows_act(l), v.sel, v.done, a->d_depth, l, rp(l), ci(l), A(l), B(l), X(l), mask(l), W(l), doff(l));
    });
    ++*launches;
    if (l == 0 && v.mark) v.mark(v.mark_ctx, 0, 1);
    const AmgLevel& F = a->lev[l];
    if (a->sa)
      launch_pdl(k_sa_restrict<VT>, useact ? act_grid(C.nnb, a->nsm) : C.nnb, 256, 0, st, C.nb_start, C.nb_sys, useact ? a->cnodes[l] : ActList{}, C.d_dof_off, C.d_node_off, a->d_depth, l + 1,
          v.sel, v.done, F.ptn_ptr, F.ptn_fine, sa_quads<VT>(F.sa_qtd, F.sa_qth), F.d_dof_off, F.d_node_off, W(l), (const VT*)C.invd, (VT*)C.b, (VT*)C.x), ++*launches;
    else
      k_amg_gather<VT><<<(C.ndof + 127) / 128, 128, 0, st>>>(C.ndof, C.dof_sys, a->d_depth, l + 1, v.sel, v.done,
                                                             C.mptr, C.mlist, W(l), (const VT*)C.invd, (VT*)C.b,
                                                             (VT*)C.x), ++*launches;
  }
  launch_pdl(k_amg_dense_apply<VT>, dim3(a->nsys, (a->maxdn + 31) / 32), 256, 0, st, v.sel, v.done, a->d_depth, a->d_dn, a->d_doff, a->d_lev_dofoff, a->d_lev_b, a->d_lev_x2, a->dense), ++*launches;
  for (int l = nl - 2; l >= 0; --l) {  // up: correction from level l+1's post-smoothed x2, then smoothing
    const AmgLevel& F = a->lev[l];
    const AmgLevel& C = a->lev[l + 1];
    if (a->sa)
      launch_pdl(k_sa_prolong<VT>, useact ? act_grid((F.nnb + kSaPW - 1) / kSaPW, a->nsm) : (F.nnb + kSaPW - 1) / kSaPW, 32 * kSaPW, 0, st, F.nnb, F.nb_start, F.nb_sys, useact ? a->fnodes[l] : ActList{}, F.d_dof_off, F.d_node_off, a->d_depth, l,
          v.sel, v.done, F.pn_ptr, F.pn_col, sa_quads<VT>(F.sa_qd, F.sa_qh), C.d_dof_off,
          C.d_node_off, (const VT*)C.x2, X(l)), ++*launches;
    else
      k_amg_correct<VT><<<nrb(l), 256, 0, st>>>(rbs(l), rbsys(l), v.sel, v.done, a->d_depth, l, X(l),
                                                (const VT*)C.x2, F.cmap, mask(l)), ++*launches;
    VT* out = l == 0 ? (VT*)v.z : (VT*)F.x2;
    VT* pcopy = l == 0 ? (VT*)v.pcopy : nullptr;
    double* part = l == 0 ? v.part_rz : nullptr;
    if (l == 0 && v.mark) v.mark(v.mark_ctx, 1, 0);
    if (l == 0 && v.sell)
      sell_pass<KT, VT, 2>(m, v, useact, (const VT*)F.invd, out);
    else if (l > 0 && cslices(l))
      csell_pass<VT, 2>(m, v, l, useact, X(l), B(l), (const VT*)F.invd, out);
    else
    dispatch_lpr(l == 0 ? lpr0 : lprc, [&](auto L) {
      if (l == 0 && v.K0lo)
        launch_pdl(k_amg_smooth<__nv_bfloat16, VT, decltype(L)::value>, rows_grid(l), 256, 0, st, rbs(l), rbsys(l), rows_act(l), v.sel, v.done, a->d_depth, l, rp(l), ci(l), (const __nv_bfloat16*)v.K0lo, B(l), X(l),
            (const VT*)F.invd, mask(l), out, pcopy, part, doff(l));
      else
        launch_pdl(k_amg_smooth<KT, VT, decltype(L)::value>, rows_grid(l), 256, 0, st, rbs(l), rbsys(l), rows_act(l), v.sel, v.done, a->d_depth, l, rp(l), ci(l), A(l), B(l), X(l), (const VT*)F.invd,
            mask(l), out, pcopy, part, doff(l));
    });
    ++*launches;
    if (l == 0 && v.mark) v.mark(v.mark_ctx, 1, 1);
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return set_error(UA_ERR_CUDA, "AMG V-cycle: %s", cudaGetErrorString(e));
  return UA_OK;
}

int amg_vcycle(ua_mesh* m, bool fp32, const AmgPcgView& v, long long* launches) {
  if (fp32) return vcycle_t<float, float>(m, v, launches);
  return vcycle_t<double, double>(m, v, launches);
}

// ---------------------------------------------------------------------------
// uvh: block preconditioner, AMG on the velocity block
// ---------------------------------------------------------------------------

// 3-dof row (c, g) of a uvh tangent holds blocks b = u, v, h of deg(g)
// entries; its u and v blocks are the velocity block's row (c, g), c < 2.
// One thread per velocity row copies them, and the row's constraint mask.
__global__ void k_uvh_extract(const DevMesh dm, int n2, const int* dof_sys2, const int* dof2_off, const int* knz2_off,
                              const double* K3, const unsigned char* cmask3, double* K2, unsigned char* cmask2) {
  const int i2 = blockIdx.x * blockDim.x + threadIdx.x;
  if (i2 >= n2) return;
  const int s = dof_sys2[i2];
  const int no = dm.sys_node_off[s], nn = dm.sys_node_off[s + 1] - no;
  const int local = i2 - dof2_off[s], c = local / nn, gl = local - c * nn;
  const int g = no + gl;
  const int np0 = dm.nodeptr[g], deg = dm.nodeptr[g + 1] - np0, lp = np0 - dm.nodeptr[no];
  const double* src = K3 + dm.sys_knz_off[s] + (size_t)c * 3 * dm.sys_nnzn[s] + 3 * (size_t)lp;
  double* dst = K2 + knz2_off[s] + (size_t)c * 2 * dm.sys_nnzn[s] + 2 * (size_t)lp;
  for (int k = 0; k < 2 * deg; ++k) dst[k] = src[k];
  cmask2[i2] = cmask3[dm.sys_dof_off[s] + local];
}

// r2 = mask(p3 on the velocity rows), x0 = l1-Jacobi of r2 (pre-smoothing).
__global__ void k_uvh_gather(const DevMesh dm, int n2, const int* dof_sys2, const int* dof2_off, const int* sel,
                             const int* done, const unsigned char* cmask2, const double* p3, const double* invd2,
                             double* r2, double* x0) {
  const int i2 = blockIdx.x * blockDim.x + threadIdx.x;
  if (i2 >= n2) return;
  const int s = dof_sys2[i2];
  if (!sel[s] || done[s]) return;
  const double v = cmask2[i2] ? 0.0 : p3[dm.sys_dof_off[s] + (i2 - dof2_off[s])];
  r2[i2] = v;
  x0[i2] = invd2[i2] * v;
}

__global__ void k_uvh_scatter(const DevMesh dm, int n2, const int* dof_sys2, const int* dof2_off, const int* sel,
                              const int* done, const double* z2, double* out3) {
  const int i2 = blockIdx.x * blockDim.x + threadIdx.x;
  if (i2 >= n2) return;
  const int s = dof_sys2[i2];
  if (!sel[s] || done[s]) return;
  out3[dm.sys_dof_off[s] + (i2 - dof2_off[s])] = z2[i2];
}

int amg_numeric_uvh(ua_mesh* m, const double* K3, const unsigned char* cmask3, long long* launches,
                    const CycFillReq* cyc, bool graph) {
  Amg* a = m->amg;
  if (!a || m->ndof != 3) return set_error(UA_ERR_INVALID, "no uvh AMG hierarchy");
  AmgLevel& F = a->lev[0];
  k_uvh_extract<<<(F.ndof + 255) / 256, 256, 0, m->stream>>>(m->dm, F.ndof, F.dof_sys, F.d_dof_off, F.d_knz_off,
                                                             K3, cmask3, (double*)F.A, a->uvh_mask), ++*launches;
  return amg_numeric(m, F.rowptr, F.colind, F.A, false, a->uvh_mask, launches, nullptr, nullptr, 1, graph, cyc);
}

int amg_apply_uvh(ua_mesh* m, const double* p3, double* out3, const int* sel, const int* done, int lpr,
                  long long* launches) {
  Amg* a = m->amg;
  AmgLevel& F = a->lev[0];
  const int nb = (F.ndof + 255) / 256;
  k_uvh_gather<<<nb, 256, 0, m->stream>>>(m->dm, F.ndof, F.dof_sys, F.d_dof_off, sel, done, a->uvh_mask, p3,
                                          (const double*)F.invd, a->uvh_r, a->uvh_x0), ++*launches;
  AmgPcgView v{F.rowptr, F.colind, F.A, a->uvh_r, a->uvh_x0, a->uvh_z, nullptr, nullptr, a->uvh_mask, sel, done,
               F.rb_start, F.rb_sys, F.nrb, lpr, a->uvh_t};
  int rc = vcycle_t<double, double>(m, v, launches);
  if (rc) return rc;
  k_uvh_scatter<<<nb, 256, 0, m->stream>>>(m->dm, F.ndof, F.dof_sys, F.d_dof_off, sel, done, a->uvh_z, out3),
      ++*launches;
  return UA_OK;
}

// ---------------------------------------------------------------------------
// active-block lists
// ---------------------------------------------------------------------------

int act_grid(int nblocks, int nsm) { return std::max(1, std::min(nblocks, 8 * nsm)); }

// exclusive block-wide scan of v (blockDim.x a multiple of 32, at most 1024); total = sum
__device__ int block_excl_scan(int v, int* sh, int& total) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) sh[wid] = x;
  __syncthreads();
  if (wid == 0) {
    int t = lane < nw ? sh[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, t, o);
      if (lane >= o) t += y;
    }
    sh[lane] = t;
  }
  __syncthreads();
  const int pre = wid ? sh[wid - 1] : 0;
  total = sh[nw - 1];
  __syncthreads();  // sh is reused by the next call
  return pre + x - v;
}

// one CTA per list: scan the systems in order (a chunk of blockDim.x systems at a time), then
// one warp per active system writes its block ids, the lanes striding over them
__global__ void __launch_bounds__(1024) k_act_compact(const ActSpec* specs, int nsys, const int* sel,
                                                      const int* done, const int* depth) {
  pdl_enter();
  __shared__ int sh[32];
  __shared__ int s_ex[1024], s_n[1024], s_b0[1024];
  const ActSpec sp = specs[blockIdx.x];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  int base = 0;
  for (int c0 = 0; c0 < nsys; c0 += blockDim.x) {  // same trip count for every thread
    const int s = c0 + threadIdx.x;
    int n = 0, b0 = 0;
    if (s < nsys && sel[s] && !done[s] && depth[s] > sp.lmin) {
      b0 = sp.blk_off[s];
      n = sp.blk_off[s + 1] - b0;
    }
    int tot;
    const int ex = block_excl_scan(n, sh, tot);
    s_ex[threadIdx.x] = ex;
    s_n[threadIdx.x] = n;
    s_b0[threadIdx.x] = b0;
    __syncthreads();
    const int cn = min((int)blockDim.x, nsys - c0);
    for (int t = wid; t < cn; t += nw) {
      const int nt = s_n[t], et = base + s_ex[t], bt = s_b0[t];
      for (int k = lane; k < nt; k += 32) sp.map[et + k] = bt + k;
    }
    __syncthreads();  // the shared arrays are rewritten by the next chunk
    base += tot;
  }
  if (threadIdx.x == 0) *sp.cnt = base;
}

int amg_act_init(ua_mesh* m, const std::vector<int>& sys_rb_off0) {
  Amg* a = m->amg;
  if (!a) return UA_ERR_INVALID;
  if (a->act_ready) return UA_OK;
  const int nsys = a->nsys;
  if ((int)sys_rb_off0.size() != nsys + 1) return set_error(UA_ERR_INVALID, "active lists: row-block prefix size");
  int dev = 0;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&a->nsm, cudaDevAttrMultiProcessorCount, dev);
  bool ok = true;
  std::vector<ActSpec> specs;
  auto make = [&](const std::vector<int>& off, int lmin) {
    ActList L;
    L.cap = off[nsys];
    int* map = (int*)dalloc(m, a, sizeof(int) * (size_t)std::max(L.cap, 1), ok);
    int* cnt = (int*)dalloc(m, a, sizeof(int), ok);
    int* doff = upload(m, a, off, ok);
    L.map = map;
    L.cnt = cnt;
    specs.push_back(ActSpec{doff, lmin, map, cnt});
    return L;
  };
  const int nl = a->nlev;
  a->rows.resize(std::max(nl - 1, 1));
  a->fnodes.resize(std::max(nl - 1, 0));
  a->cnodes.resize(std::max(nl - 1, 0));
  a->rows[0] = make(sys_rb_off0, -1);  // the handle's Krylov rows: every active system
  for (int l = 1; l + 1 < nl; ++l) a->rows[l] = make(a->lev[l].h_sys_rb_off, l);
  if (a->sa)
    for (int l = 0; l + 1 < nl; ++l) {
      a->fnodes[l] = make(a->lev[l].h_sys_nb_off, l);
      a->cnodes[l] = make(a->lev[l + 1].h_sys_nb_off, l);
    }
  if (a->sell.ready) a->sell.act = make(a->sell.h_sys_sb_off, -1);  // node slice blocks: every active system
  for (int l = 1; l < (int)a->csell.size(); ++l)
    if (a->csell[l].ready) a->csell[l].act = make(a->csell[l].h_sys_sb_off, l);  // depth > l
  a->d_specs = upload(m, a, specs, ok);
  a->nspecs = (int)specs.size();
  if (!ok) return set_error(UA_ERR_OOM, "active lists: device allocation failed");
  a->act_ready = true;
  return UA_OK;
}

void amg_act_compact(ua_mesh* m, const int* sel, const int* done, long long* launches) {
  Amg* a = m->amg;
  launch_pdl(k_act_compact, a->nspecs, 1024, 0, m->stream, a->d_specs, a->nsys, sel, done, a->d_depth), ++*launches;
}

ActList amg_act_rows0(const ua_mesh* m) { return m->amg && m->amg->act_ready ? m->amg->rows[0] : ActList{}; }

}  // namespace ua
