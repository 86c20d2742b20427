// uvh residual/tangent assembly of the fully implicit transient step:
// uvhMatrixAssembly.m:6-585 -> uvhAssemblyIntPointImplicitSUPG.m:10-531 ->
// uvhNodalLoopSSTREAM.m:1-229 on the device.
//
// One CTA per node patch.  Threads map to (element, local node I): each
// thread evaluates the integration-point quantities of its element (the
// nodal fields are staged in shared memory) and accumulates the three rows
// (x-momentum, y-momentum, mass conservation) of its node I against all nodes
// J in the nine blocks Kxu..Khh, directly in shared memory slots it alone
// owns.  The patch's node-level non-zeros are then summed over their element
// contributions in increasing global element order (deterministic segmented
// sum, no atomics), nine dof-level values each.
#include "ua_internal.h"
#include "ua_physics.cuh"
#include "ua_kernels.h"

#include <algorithm>

namespace ua {

// Nodal quantities staged per element (index into the field block).
enum { F_X = 0, F_Y, F_H1, F_U1, F_V1, F_S, F_B, F_RHO, F_A, F_N, F_C, F_M, F_H0, F_U0, F_V0, F_A0, F_A1, F_DADH,
       F_B1, F_COUNT };

// SUPGtau.m:7-111
__device__ __forceinline__ double supg_tau(const UvhPhys& P, double v, double l, double dt) {
  const double eps = 2.220446049250313e-16;
  const double taut = dt / 2 + eps;
  const double taus = l / (2 * v + P.SpeedZero);
  double tau;
  switch (P.tau_kind) {
    case 1: tau = taut; break;                                  // "taut"
    case 2: {                                                   // "tau1"
      const double ECN = taut / taus;
      tau = (ECN < 1e-6 ? ECN / 3 : 1.0 / tanh(ECN) - 1.0 / ECN) * taus;
      break;
    }
    case 3: tau = (dt / 2) / (1 + taut / taus); break;          // "tau2"
    default: tau = taus;                                        // "taus" (:61-62)
  }
  return P.tau_mult * tau;
}

// Fields of node gn at the current iterate, field k at f[k * ld].
__device__ __forceinline__ void stage_node(const DevMesh& M, const UvhPhys& P, const UvhIn& in, const SysScal& S,
                                           int gn, int uoff, int voff, int hoff, double gam, double* f, int ld) {
  double h1 = in.X[hoff + gn], u1 = in.X[uoff + gn], v1 = in.X[voff + gn];
  if (in.dX) { h1 += gam * in.dX[hoff + gn]; u1 += gam * in.dX[uoff + gn]; v1 += gam * in.dX[voff + gn]; }
  const double h0 = __ldg(in.h0 + gn);
  double u0 = __ldg(in.u0 + gn), v0 = __ldg(in.v0 + gn);
  double a0 = __ldg(in.as0 + gn) + __ldg(in.ab0 + gn), a1 = __ldg(in.as1 + gn) + __ldg(in.ab1 + gn);
  if (in.zero_fields) {  // uvhMatrixAssembly.m:9-15
    u1 = v1 = u0 = v0 = 0;
    h1 = h0;
    a0 = 2 * fabs(__ldg(in.ab0 + gn)) + 1;
    a1 = 2 * fabs(__ldg(in.ab1 + gn)) + 1;
  }
  const double Sg = __ldg(in.S + gn), Bg = __ldg(in.B + gn), rg = __ldg(in.rho + gn);
  // Calc_bs_From_hBS.m:71-79 at the current h (uvhMatrixAssembly.m:36)
  const double hf = S.rhow * (Sg - Bg) / rg;
  const double GF = heaviside_approx(P.kH, h1 - hf, P.Hh0);
  f[F_X * ld] = __ldg(M.x + gn); f[F_Y * ld] = __ldg(M.y + gn);
  f[F_H1 * ld] = h1; f[F_U1 * ld] = u1; f[F_V1 * ld] = v1;
  f[F_S * ld] = Sg; f[F_B * ld] = Bg; f[F_RHO * ld] = rg;
  f[F_A * ld] = __ldg(in.A + gn); f[F_N * ld] = __ldg(in.n + gn);
  f[F_C * ld] = __ldg(in.C + gn); f[F_M * ld] = __ldg(in.m + gn);
  f[F_H0 * ld] = h0; f[F_U0 * ld] = u0; f[F_V0 * ld] = v0;
  f[F_A0 * ld] = a0; f[F_A1 * ld] = a1;
  f[F_DADH * ld] = in.dadh ? __ldg(in.dadh + gn) : 0.0;
  f[F_B1 * ld] = GF * Bg + (1 - GF) * (Sg - rg * h1 / S.rhow);
}

// ---------------------------------------------------------------------------
// linear elements
// ---------------------------------------------------------------------------
constexpr int NOD = 3, kThreads = 512;

// The patch's non-zeros and residuals, summed over their element contributions in increasing global
// element order.
template <bool WITHK, typename KT>
__device__ __forceinline__ void uvh_scatter(const DevMesh& M, const UvOut& out, int p, int s, int uoff, int voff,
                                            int hoff, const KT* sK, const double* sR, int E, int ne) {
  const int pn0 = M.patch_node_ptr[p];
  const int nr = M.patch_node_ptr[p + 1] - pn0;
  if (WITHK && out.K) {
    const int q0 = M.patch_q_ptr[p], q1 = M.patch_q_ptr[p + 1];
    const int nbase = M.nodeptr[M.sys_node_off[s]];
    const int nnzn = M.sys_nnzn[s];
    const int kbase = M.sys_knz_off[s];
    KT* Ko = reinterpret_cast<KT*>(out.K);
    for (int q = q0 + threadIdx.x; q < q1; q += blockDim.x) {
      const uint32_t rk = __ldg(M.pq_rk + q);
      const int r = rk >> 16, k = rk & 0xffff;
      const int gnd = __ldg(M.patch_nodes + pn0 + r);
      const int np0 = __ldg(M.nodeptr + gnd);
      const int deg = __ldg(M.nodeptr + gnd + 1) - np0;
      const int lp = np0 - nbase;
      KT v[9];
#pragma unroll
      for (int i = 0; i < 9; ++i) v[i] = 0;
      const int cend = __ldg(M.pq_cptr + q + 1);
      for (int c = __ldg(M.pq_cptr + q); c < cend; ++c) {
        const uint16_t code = __ldg(M.contrib + c);
        int ce = code >> 6;
        const int a = (code >> 3) & 7, b = code & 7;
        bool ok = true;
        UA_CHECK_INDEX(M.dbg, ce, 0, ne, BS_CONTRIB_ELEM, ok);
        if (!ok) continue;
        const KT* src = sK + (size_t)(a * 9 * NOD + b) * E + ce;
#pragma unroll
        for (int i = 0; i < 9; ++i) v[i] += src[(size_t)i * NOD * E];
      }
      {
        size_t last = (size_t)kbase + 6 * (size_t)nnzn + 3 * (size_t)lp + 2 * (size_t)deg + k;  // largest index
        bool okk = true;
        UA_CHECK_INDEX(M.dbg, last, (size_t)kbase, (size_t)M.sys_knz_off[s + 1], BS_K_INDEX, okk);
        (void)last;
        if (!okk) continue;
      }
#pragma unroll
      for (int cr = 0; cr < 3; ++cr) {
        const size_t base = (size_t)kbase + (size_t)cr * 3 * nnzn + 3 * (size_t)lp;
#pragma unroll
        for (int cc = 0; cc < 3; ++cc) Ko[base + (size_t)cc * deg + k] = v[cr * 3 + cc];
      }
    }
  }
  for (int r = threadIdx.x; r < nr; r += blockDim.x) {
    int gnd = __ldg(M.patch_nodes + pn0 + r);
    bool okr = true;
    UA_CHECK_INDEX(M.dbg, gnd, M.sys_node_off[s], M.sys_node_off[s + 1], BS_R_INDEX, okr);
    if (!okr) continue;
    const int q = __ldg(M.prow_diag + pn0 + r);
    double acc[6] = {0, 0, 0, 0, 0, 0};
    const int cend = __ldg(M.pq_cptr + q + 1);
    for (int c = __ldg(M.pq_cptr + q); c < cend; ++c) {
      const uint16_t code = __ldg(M.contrib + c);
      int ce = code >> 6;
      const int a = (code >> 3) & 7;
      bool ok = true;
      UA_CHECK_INDEX(M.dbg, ce, 0, ne, BS_CONTRIB_ELEM, ok);
      if (!ok) continue;
#pragma unroll
      for (int i = 0; i < 6; ++i) acc[i] += sR[(i * NOD + a) * E + ce];
    }
    out.R[uoff + gnd] = acc[0] - acc[1];
    out.R[voff + gnd] = acc[2] - acc[3];
    out.R[hoff + gnd] = acc[4] - acc[5];
    if (out.Tint) { out.Tint[uoff + gnd] = acc[0]; out.Tint[voff + gnd] = acc[2]; out.Tint[hoff + gnd] = acc[4]; }
    if (out.Fext) { out.Fext[uoff + gnd] = acc[1]; out.Fext[voff + gnd] = acc[3]; out.Fext[hoff + gnd] = acc[5]; }
  }
}

// GEN: any sliding law and the melange terms (Weertman chosen at run time); else Weertman only
// (the general code stays out of that build)
template <bool WITHK, typename KT, bool GEN>
__global__ void __launch_bounds__(kThreads) uvh_patch_kernel(DevMesh M, QuadTable Q, UvhPhys P, UvhIn in,
                                                             UvOut out) {
  constexpr int NB = 9 * NOD * NOD;   // tangent entries per element
  extern __shared__ __align__(16) unsigned char smem[];
  const int p = blockIdx.x;
  const int s = M.patch_sys[p];
  if (in.active && !in.active[s]) return;
  const int E = M.max_patch_elems;
  KT* sK = reinterpret_cast<KT*>(smem);
  size_t off = WITHK ? (((size_t)NB * E * sizeof(KT) + 15) & ~(size_t)15) : 0;
  double* sR = reinterpret_cast<double*>(smem + off);                 // [6*NOD][E]
  double* sF = sR + (size_t)6 * NOD * E;                               // [F_COUNT][E*NOD]
  const int e0 = M.patch_elem_ptr[p], ne = M.patch_elem_ptr[p + 1] - e0;
  const int no = M.sys_node_off[s];
  const int nn_s = M.sys_node_off[s + 1] - no;
  const int uoff = M.sys_dof_off[s] - no, voff = uoff + nn_s, hoff = voff + nn_s;
  const double gam = in.gamma ? in.gamma[s] : 0.0;
  const SysScal S = in.scal[s];
  const double rhow = S.rhow, g = S.g, ca = S.ca, sa = S.sa, dt = S.dt;
  const double theta = P.theta;
  const int EN = E * NOD;
  // stage the nodal fields (one thread per element node)
  for (int t = threadIdx.x; t < ne * NOD; t += blockDim.x) {
    const int el = t / NOD, a = t % NOD;
    bool inb = true;
    int e = __ldg(M.patch_elems + e0 + el);
    UA_CHECK_INDEX(M.dbg, e, 0, M.ne, BS_PATCH_ELEM, inb);
    int gn = __ldg(M.conn + (size_t)a * M.ne + e);
    UA_CHECK_INDEX(M.dbg, gn, 0, M.nn, BS_ELEM_NODE, inb);
    (void)inb;
    stage_node(M, P, in, S, gn, uoff, voff, hoff, gam, sF + el * NOD + a, EN);
  }
  __syncthreads();
  const int t = threadIdx.x;
  const int el = t / NOD, I = t % NOD;
  if (el < ne) {
    const double* f = sF + el * NOD;
    auto fv = [&](int k, int a) { return f[k * EN + a]; };
    if (WITHK) {
      for (int k = 0; k < 9 * NOD; ++k) sK[(size_t)(I * 9 * NOD + k) * E + el] = 0;
    }
    double Tx = 0, Fx = 0, Ty = 0, Fy = 0, Th = 0, Fh = 0;
    // element area (TriAreaFE.m / TriArea.m) -> l = sqrt(2*area) (:156)
    const double area = 0.5 * fabs((fv(F_X, 0) - fv(F_X, 2)) * (fv(F_Y, 1) - fv(F_Y, 0)) -
                                   (fv(F_X, 0) - fv(F_X, 1)) * (fv(F_Y, 2) - fv(F_Y, 0)));
    const double lsupg = sqrt(2 * area);
    // derivVector.m:96-109, constant over the element
    double Dx[NOD], Dy[NOD], J11 = 0, J12 = 0, J21 = 0, J22 = 0;
#pragma unroll
    for (int a = 0; a < NOD; ++a) {
      J11 += fv(F_X, a) * Q.der[0][0][a];
      J12 += fv(F_Y, a) * Q.der[0][0][a];
      J21 += fv(F_X, a) * Q.der[0][1][a];
      J22 += fv(F_Y, a) * Q.der[0][1][a];
    }
    const double detJ = J11 * J22 - J12 * J21;
#pragma unroll
    for (int a = 0; a < NOD; ++a) {
      Dx[a] = (J22 * Q.der[0][0][a] - J12 * Q.der[0][1][a]) / detJ;
      Dy[a] = (-J21 * Q.der[0][0][a] + J11 * Q.der[0][1][a]) / detJ;
    }
#pragma unroll 1
    for (int ip = 0; ip < Q.nip; ++ip) {
      double N[NOD];
#pragma unroll
      for (int a = 0; a < NOD; ++a) N[a] = Q.fun[ip][a];
      auto itp = [&](int k) {
        double v = 0;
#pragma unroll
        for (int a = 0; a < NOD; ++a) v += fv(k, a) * N[a];
        return v;
      };
      auto ddx = [&](int k) {
        double v = 0;
#pragma unroll
        for (int a = 0; a < NOD; ++a) v += Dx[a] * fv(k, a);
        return v;
      };
      auto ddy = [&](int k) {
        double v = 0;
#pragma unroll
        for (int a = 0; a < NOD; ++a) v += Dy[a] * fv(k, a);
        return v;
      };
      // uvhAssemblyIntPointImplicitSUPG.m:62-121 (no level set, no thickness penalty/barrier)
      const double hint = itp(F_H1), uint = itp(F_U1), vint = itp(F_V1);
      const double Cint = itp(F_C), mint = itp(F_M), Aint = itp(F_A), nint = itp(F_N);
      const double h0int = itp(F_H0), u0int = itp(F_U0), v0int = itp(F_V0);
      const double a1int = itp(F_A1), a0int = itp(F_A0), dadhint = itp(F_DADH);
      const double Bint = itp(F_B), Sint = itp(F_S), rhoint = itp(F_RHO);
      const double Hint = Sint - Bint;
      const double hfint = rhow * Hint / rhoint;
      // flotation steps and pulses: one expm1 per argument (for Hh0 = 0 the mirrored step is
      // 1 - the step and the pulse is even)
      const StepPulse fl = step_pulse(P.kH, hint - hfint, P.Hh0);
      const double Heint = 0.5 + 0.5 * fl.t;
      const double deltaint = fl.delta;
      double HEint, Deltaint;
      if (P.Hh0 == 0.0) {
        HEint = 0.5 - 0.5 * fl.t;
        Deltaint = fl.delta;
      } else {
        const StepPulse fm = step_pulse(P.kH, hfint - hint, P.Hh0);
        HEint = 0.5 + 0.5 * fm.t;
        Deltaint = fm.delta;
      }
      const double Hposint = (0.5 + 0.5 * step_pulse(P.kH, Hint, P.Hh0).t) * Hint;
      const bool cube = S.cube != 0.0;  // n = m = 3 at every node of the system
      const double dint = HEint * rhoint * hint / rhow + Heint * Hposint;
      const double Dddhint = HEint * rhoint / rhow - Deltaint * hint * rhoint / rhow + deltaint * Hposint;
      // :132-148
      const double dhdx = ddx(F_H1), dhdy = ddy(F_H1), dh0dx = ddx(F_H0), dh0dy = ddy(F_H0);
      const double exx0 = ddx(F_U0), eyy0 = ddy(F_V0);
      const double dbdx = ddx(F_B1), dbdy = ddy(F_B1), drhodx = ddx(F_RHO), drhody = ddy(F_RHO);
      const double exx = ddx(F_U1), eyy = ddy(F_V1);
      const double exy = 0.5 * (ddx(F_V1) + ddy(F_U1));
      double eta, Ev;
      effective_viscosity(P.uv, Aint, nint, exx, eyy, exy, eta, Ev, cube);  // :149
      Drag d;  // :150
      if (!GEN || (P.uv.law == UA_SLIDING_WEERTMAN && !P.uv.melange)) {
        d = basal_drag_weertman(P.uv, Heint, deltaint, uint, vint, Cint, mint, cube);
      } else {
        int gn[NOD];
        const int e = __ldg(M.patch_elems + e0 + el);
#pragma unroll
        for (int a = 0; a < NOD; ++a) gn[a] = __ldg(M.conn + (size_t)a * M.ne + e);
        d = basal_drag_general(P.uv, Heint, deltaint, hint, Hint, rhoint, rhow, g, uint, vint, Cint, mint,
                               drag_interp<NOD>(in.drag, gn, N));
      }
      const double speed0 = sqrt(u0int * u0int + v0int * v0int + P.SpeedZero * P.SpeedZero);  // :157
      const double tau0 = P.beta0 * supg_tau(P, speed0, lsupg, dt);                         // :158-159
      const double detJw = detJ * Q.w[ip];
      // uvhNodalLoopSSTREAM.m
      const double qx1dx = rhoint * exx * hint + rhoint * uint * dhdx + drhodx * uint * hint;  // :39
      const double qy1dy = rhoint * eyy * hint + rhoint * vint * dhdy + drhody * vint * hint;
      const double qx0dx = rhoint * exx0 * h0int + rhoint * u0int * dh0dx + drhodx * u0int * h0int;
      const double qy0dy = rhoint * eyy0 * h0int + rhoint * v0int * dh0dy + drhody * v0int * h0int;
      const double DxI = Dx[I], DyI = Dy[I], funI = N[I];
      const double SUPG = funI + 0.5 * tau0 * (u0int * DxI + v0int * DyI);  // :55
      if (WITHK) {
        const double Pu_I = (4 * exx + 2 * eyy) * DxI + 2 * exy * DyI;   // h-derivative of t3+t4 / h eta
        const double Pv_I = (4 * eyy + 2 * exx) * DyI + 2 * exy * DxI;
        const double cxh_nn = d.dxh + ca * g * (rhoint - rhow * Dddhint) * dbdx - sa * g * rhoint;
        const double cyh_nn = d.dyh + ca * g * (rhoint - rhow * Dddhint) * dbdy;
        const double ch_d = -ca * g * (rhoint * hint - rhow * dint * Dddhint);
        const double khh_n = rhoint - dt * theta * rhoint * dadhint +
                             dt * theta * (rhoint * exx + drhodx * uint + rhoint * eyy + drhody * vint);
        KT* row = sK + (size_t)I * 9 * NOD * E + el;
#pragma unroll
        for (int J = 0; J < NOD; ++J) {
          const double DxJ = Dx[J], DyJ = Dy[J], fJ = N[J];
          const double Deu = Ev * ((2 * exx + eyy) * DxJ + exy * DyJ);
          const double Dev = Ev * ((2 * eyy + exx) * DyJ + exy * DxJ);
          const double E11 = hint * (4 * exx + 2 * eyy) * Deu * DxI + 2 * hint * exy * Deu * DyI;
          const double E12 = hint * (4 * exx + 2 * eyy) * Dev * DxI + 2 * hint * exy * Dev * DyI;
          const double E22 = hint * (4 * eyy + 2 * exx) * Dev * DyI + 2 * hint * exy * Dev * DxI;
          const double E21 = hint * (4 * eyy + 2 * exx) * Deu * DyI + 2 * hint * exy * Deu * DxI;
          const double he = hint * eta;
          // :84-110 (Kxu, Kyv, Kxv, Kyu), :141-157 post-2025 (Kxh, Kyh), :164-179 (Khu, Khv, Khh)
          row[(0 * NOD + J) * E] += (KT)((4 * he * DxI * DxJ + he * DyI * DyJ + E11 + d.dxu * fJ * funI) * detJw);
          row[(1 * NOD + J) * E] += (KT)((he * (2 * DxI * DyJ + DyI * DxJ) + E12 + d.dxv * fJ * funI) * detJw);
          row[(2 * NOD + J) * E] += (KT)((eta * Pu_I * fJ + cxh_nn * funI * fJ + ch_d * DxI * fJ) * detJw);
          row[(3 * NOD + J) * E] += (KT)((he * (2 * DyI * DxJ + DxI * DyJ) + E21 + d.dxv * fJ * funI) * detJw);
          row[(4 * NOD + J) * E] += (KT)((4 * he * DyI * DyJ + he * DxI * DxJ + E22 + d.dyv * fJ * funI) * detJw);
          row[(5 * NOD + J) * E] += (KT)((eta * Pv_I * fJ + cyh_nn * funI * fJ + ch_d * DyI * fJ) * detJw);
          row[(6 * NOD + J) * E] += (KT)(theta * (rhoint * dhdx * fJ + drhodx * hint * fJ + rhoint * hint * DxJ) *
                                         SUPG * detJw * dt);
          row[(7 * NOD + J) * E] += (KT)(theta * (rhoint * dhdy * fJ + drhody * hint * fJ + rhoint * hint * DyJ) *
                                         SUPG * detJw * dt);
          row[(8 * NOD + J) * E] += (KT)((khh_n * fJ + dt * theta * (rhoint * uint * DxJ + rhoint * vint * DyJ)) *
                                         SUPG * detJw);
        }
      }
      // :189-226 residual
      const double rr = rhoint * hint - rhow * dint;
      const double pp = 0.5 * ca * g * (rhoint * hint * hint - rhow * dint * dint);
      Tx += (hint * eta * (4 * exx + 2 * eyy) * DxI + hint * eta * 2 * exy * DyI + d.taux * funI) * detJw;
      Fx += (-ca * g * rr * dbdx * funI + rhoint * g * hint * sa * funI + pp * DxI) * detJw;
      Ty += (hint * eta * (4 * eyy + 2 * exx) * DyI + hint * eta * 2 * exy * DxI + d.tauy * funI) * detJw;
      Fy += (-ca * g * rr * dbdy * funI + pp * DyI) * detJw;
      const double qterm = dt * (theta * qx1dx + (1 - theta) * qx0dx + theta * qy1dy + (1 - theta) * qy0dy) * SUPG;
      const double dhdt = rhoint * (h0int - hint) * SUPG;  // h0barr = h1barr = 0
      const double accterm = dt * rhoint * ((1 - theta) * a0int + theta * a1int) * SUPG;
      Th += -dhdt * detJw;
      Fh += (accterm - qterm) * detJw;
    }
    sR[(0 * NOD + I) * E + el] = Tx;
    sR[(1 * NOD + I) * E + el] = Fx;
    sR[(2 * NOD + I) * E + el] = Ty;
    sR[(3 * NOD + I) * E + el] = Fy;
    sR[(4 * NOD + I) * E + el] = Th;
    sR[(5 * NOD + I) * E + el] = Fh;
  }
  __syncthreads();
  uvh_scatter<WITHK, KT>(M, out, p, s, uoff, voff, hoff, sK, sR, E, ne);
}

// ---------------------------------------------------------------------------
// quadratic elements: integration points on threads, then element rows
// ---------------------------------------------------------------------------
//
// A thread per (element, node) evaluates the physics of every point six times and keeps its 54 tangent
// entries in shared memory (P2 101x51: 506 us with the tangent, 279 us without).  Here a thread per
// point evaluates it once and leaves 22 pairs of coefficients, in reference coordinates (the inverse
// Jacobian multiplied in, so that the rows need only the rule's tables); then a thread per (element, row
// component, node) sums its 18 entries over the points in registers.  The element rows go to global
// memory, 2.9 kB an element, and a second kernel sums each patch's non-zeros over them: with the rows in
// shared memory a patch held 50 elements and every element was evaluated in three patches (285 us and
// 103 us; now 134 us and 62 us with the gather).  Bound by the latency of the two phases, few warps an SM.
namespace p2h {
constexpr int kIps = 16, kIpc = 8;
enum { PR_UU = 0, PR_UUC, PR_VV, PR_VVC, PR_UV1, PR_UV2, PR_XV, PR_XH, PR_YH, PR_CH, PR_TX, PR_TY, PR_PX, PR_PY,
       PR_TN, PR_FN, PR_S, PR_HC, PR_HU, PR_HV, PR_HH, PR_TF, kPairs };
constexpr size_t kPoint = (size_t)kIpc * kPairs * sizeof(double2);  // an element's points
}  // namespace p2h

// blk: {system, first element, elements} of each block, at most G elements.  Rows of element e: tangent
// kel[((6 e + a) 6 + b) 9 + 3 c + column component], residual parts rel[6 (6 e + a) + 2 c + {0, 1}].
template <bool GEN, bool KW>
__global__ void __launch_bounds__(KW ? 384 : 256, KW ? 1 : 2) uvh_p2_elements(DevMesh M, QuadTable Q, UvhPhys P, UvhIn in,
                                                                             const int4* blk, int G, int rows,
                                                                             double* kel, double* rel) {
  using namespace p2h;
  extern __shared__ __align__(16) unsigned char smem[];
  const int4 bk = blk[blockIdx.x];
  const int s = bk.x, eb = bk.y, gn_ = bk.z;
  if (in.active && !in.active[s]) return;
  constexpr bool kw = KW;
  const int MH = 6 * G;
  double2* pts = reinterpret_cast<double2*>(smem);        // [G][kIpc][kPairs]
  double2* sD = pts + (size_t)G * kIpc * kPairs;          // reference derivatives [ip][6]
  double* sN = reinterpret_cast<double*>(sD + kIps * 6);  // N [ip][6]
  double* nd = sN + kIps * 6;                             // [F_COUNT][MH], node k of element el at 6 el + k
  const int no = M.sys_node_off[s], nn_s = M.sys_node_off[s + 1] - no;
  const int uoff = M.sys_dof_off[s] - no, voff = uoff + nn_s, hoff = voff + nn_s;
  const double gam = in.gamma ? in.gamma[s] : 0.0;
  const SysScal S = in.scal[s];
  const double rhow = S.rhow, g = S.g, ca = S.ca, sa = S.sa, dt = S.dt, theta = P.theta;
  const bool cube = S.cube != 0.0;  // n = m = 3 at every node of the system
  for (int t = threadIdx.x; t < kIps * 6; t += blockDim.x) {
    sN[t] = Q.fun[t / 6][t % 6];
    sD[t] = make_double2(Q.der[t / 6][0][t % 6], Q.der[t / 6][1][t % 6]);
  }
  for (int t = threadIdx.x; t < 6 * gn_; t += blockDim.x) {
    int e = eb + t / 6;
    bool okn = true;
    UA_CHECK_INDEX(M.dbg, e, 0, M.ne, BS_PATCH_ELEM, okn);
    int gn = __ldg(M.conn + (size_t)(t % 6) * M.ne + e);
    UA_CHECK_INDEX(M.dbg, gn, no, no + nn_s, BS_ELEM_NODE, okn);
    (void)okn;
    stage_node(M, P, in, S, gn, uoff, voff, hoff, gam, nd + t, MH);
  }
  __syncthreads();
  // row component c (uniform over a warp where rows is a multiple of 32; else two meet in some warps)
  const int c = threadIdx.x / rows, ri = threadIdx.x - c * rows, a = ri % 6, el = c < 3 ? ri / 6 : G;
  {
    double ku[6] = {}, kv[6] = {}, kh[6] = {}, T = 0, F = 0;  // row c of node a against u, v, h
    for (int ip0 = 0; ip0 < kIps; ip0 += kIpc) {
      // (a) points
      for (int t = threadIdx.x; t < gn_ * kIpc; t += blockDim.x) {
        const int pe = t / kIpc, pi = t - pe * kIpc, ip = ip0 + pi;
        int l[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) l[k] = 6 * pe + k;
        const double* N = sN + ip * 6;
        const double2* dr = sD + ip * 6;
        auto itp = [&](int k) {
          double v = 0;
#pragma unroll
          for (int q = 0; q < 6; ++q) v += nd[k * MH + l[q]] * N[q];
          return v;
        };
        auto grad = [&](int k) {  // reference derivatives
          double2 v = make_double2(0, 0);
#pragma unroll
          for (int q = 0; q < 6; ++q) {
            const double f = nd[k * MH + l[q]];
            v.x += f * dr[q].x;
            v.y += f * dr[q].y;
          }
          return v;
        };
        // element area from the corner nodes (TriAreaFE.m / TriArea.m) -> l = sqrt(2*area) (:156)
        const double x0 = nd[F_X * MH + l[0]], x1 = nd[F_X * MH + l[2]], x2 = nd[F_X * MH + l[4]];
        const double y0 = nd[F_Y * MH + l[0]], y1 = nd[F_Y * MH + l[2]], y2 = nd[F_Y * MH + l[4]];
        const double lsupg = sqrt(fabs((x0 - x2) * (y1 - y0) - (x0 - x1) * (y2 - y0)));
        // derivVector.m:96-109, gradients by the chain rule
        const double2 gx = grad(F_X), gy = grad(F_Y);  // (J11, J21), (J12, J22)
        const double detJ = gx.x * gy.y - gy.x * gx.y, rd = 1.0 / detJ;
        // d/dx = ix d/dxi + jx d/deta, d/dy = iy d/dxi + jy d/deta
        const double ix = gy.y * rd, jx = -gy.x * rd, iy = -gx.y * rd, jy = gx.x * rd;
        const double w = detJ * Q.w[ip];
        // uvhAssemblyIntPointImplicitSUPG.m:62-121 (no level set, no thickness penalty/barrier)
        const double hint = itp(F_H1), uint = itp(F_U1), vint = itp(F_V1);
        const double rhoint = itp(F_RHO), Hint = itp(F_S) - itp(F_B);
        const double hfint = rhow * Hint / rhoint;
        // flotation steps and pulses: one expm1 per argument (for Hh0 = 0 the mirrored step is
        // 1 - the step and the pulse is even)
        const StepPulse fl = step_pulse(P.kH, hint - hfint, P.Hh0);
        const double Heint = 0.5 + 0.5 * fl.t, deltaint = fl.delta;
        double HEint, Deltaint;
        if (P.Hh0 == 0.0) {
          HEint = 0.5 - 0.5 * fl.t;
          Deltaint = fl.delta;
        } else {
          const StepPulse fm = step_pulse(P.kH, hfint - hint, P.Hh0);
          HEint = 0.5 + 0.5 * fm.t;
          Deltaint = fm.delta;
        }
        const double Hposint = (0.5 + 0.5 * step_pulse(P.kH, Hint, P.Hh0).t) * Hint;
        const double dint = HEint * rhoint * hint / rhow + Heint * Hposint;
        const double Dddhint = HEint * rhoint / rhow - Deltaint * hint * rhoint / rhow + deltaint * Hposint;
        double2* o = pts + ((size_t)pe * kIpc + pi) * kPairs;
        // :132-148
        const double2 gu = grad(F_U1), gv = grad(F_V1), gb1 = grad(F_B1);
        const double exx = ix * gu.x + jx * gu.y, eyy = iy * gv.x + jy * gv.y;
        const double exy = 0.5 * ((ix * gv.x + jx * gv.y) + (iy * gu.x + jy * gu.y));
        const double dbdx = ix * gb1.x + jx * gb1.y, dbdy = iy * gb1.x + jy * gb1.y;
        Drag d;  // :150
        {
          const double Cint = itp(F_C), mint = cube ? 3.0 : itp(F_M);
          if (!GEN || (P.uv.law == UA_SLIDING_WEERTMAN && !P.uv.melange)) {
            d = basal_drag_weertman(P.uv, Heint, deltaint, uint, vint, Cint, mint, cube);
          } else {
            int gn[6];
            double Nw[6];
#pragma unroll
            for (int k = 0; k < 6; ++k) { gn[k] = __ldg(M.conn + (size_t)k * M.ne + eb + pe); Nw[k] = N[k]; }
            d = basal_drag_general(P.uv, Heint, deltaint, hint, Hint, rhoint, rhow, g, uint, vint, Cint, mint,
                                   drag_interp<6>(in.drag, gn, Nw));
          }
        }
        double eta, Ev;
        effective_viscosity(P.uv, itp(F_A), cube ? 3.0 : itp(F_N), exx, eyy, exy, eta, Ev, cube);  // :149
        const double he = hint * eta * w;
        const double t1 = 4 * exx + 2 * eyy, t2 = 4 * eyy + 2 * exx, t3 = 2 * exy;
        if (kw) {
          const double hE = 2.0 * hint * Ev * w;
          const double p1 = 2 * exx + eyy, q1 = 2 * eyy + exx, q2 = exy;  // P_u = p1 Dx + q2 Dy, P_v = q1 Dy + q2 Dx
          // the rows of a 2x2 matrix between the inverse Jacobian's columns (ix, jx) and (iy, jy)
          auto ref = [&](double axx, double axy, double ayx, double ayy, double2& r1, double2& r2) {
            const double xa = axx * ix + axy * iy, xb = axx * jx + axy * jy;
            const double ya = ayx * ix + ayy * iy, yb = ayx * jx + ayy * jy;
            r1 = make_double2(ix * xa + iy * ya, ix * xb + iy * yb);
            r2 = make_double2(jx * xa + jy * ya, jx * xb + jy * yb);
          };
          double2 r1, r2;
          // :84-110 (Kxu, Kyv, Kxv, Kyu)
          ref(4 * he + hE * p1 * p1, hE * p1 * q2, hE * p1 * q2, he + hE * q2 * q2, r1, r2);
          o[PR_UU] = r1;
          o[PR_UUC] = make_double2(r2.y, d.dxu * w);
          ref(he + hE * q2 * q2, hE * q1 * q2, hE * q1 * q2, 4 * he + hE * q1 * q1, r1, r2);
          o[PR_VV] = r1;
          o[PR_VVC] = make_double2(r2.y, d.dyv * w);
          ref(hE * p1 * q2, 2 * he + hE * p1 * q1, he + hE * q2 * q2, hE * q2 * q1, r1, r2);
          o[PR_UV1] = r1;
          o[PR_UV2] = r2;
          // :141-157 post-2025 (Kxh, Kyh)
          const double chd = -ca * g * (rhoint * hint - rhow * dint * Dddhint) * w, ew = eta * w;
          o[PR_XH] = make_double2((ew * t1 + chd) * ix + ew * t3 * iy, (ew * t1 + chd) * jx + ew * t3 * jy);
          o[PR_YH] = make_double2((ew * t2 + chd) * iy + ew * t3 * ix, (ew * t2 + chd) * jy + ew * t3 * jx);
          o[PR_CH] = make_double2((d.dxh + ca * g * (rhoint - rhow * Dddhint) * dbdx - sa * g * rhoint) * w,
                                  (d.dyh + ca * g * (rhoint - rhow * Dddhint) * dbdy) * w);
        }
        // :189-226 residual
        const double rr = rhoint * hint - rhow * dint;
        const double pp = 0.5 * ca * g * (rhoint * hint * hint - rhow * dint * dint) * w;
        o[PR_TX] = make_double2(he * (t1 * ix + t3 * iy), he * (t1 * jx + t3 * jy));
        o[PR_TY] = make_double2(he * (t2 * iy + t3 * ix), he * (t2 * jy + t3 * jx));
        o[PR_PX] = make_double2(pp * ix, pp * jx);
        o[PR_PY] = make_double2(pp * iy, pp * jy);
        o[PR_TN] = make_double2(d.taux * w, d.tauy * w);
        o[PR_FN] = make_double2((-ca * g * rr * dbdx + rhoint * g * hint * sa) * w, -ca * g * rr * dbdy * w);
        // mass conservation (uvhNodalLoopSSTREAM.m:39-55, :164-179)
        const double u0int = itp(F_U0), v0int = itp(F_V0), h0int = itp(F_H0);
        const double speed0 = sqrt(u0int * u0int + v0int * v0int + P.SpeedZero * P.SpeedZero);  // :157
        const double tau0 = P.beta0 * supg_tau(P, speed0, lsupg, dt);                           // :158-159
        o[PR_S] = make_double2(0.5 * tau0 * (u0int * ix + v0int * iy), 0.5 * tau0 * (u0int * jx + v0int * jy));
        const double2 gh = grad(F_H1), gr = grad(F_RHO);
        const double dhdx = ix * gh.x + jx * gh.y, dhdy = iy * gh.x + jy * gh.y;
        const double drhodx = ix * gr.x + jx * gr.y, drhody = iy * gr.x + jy * gr.y;
        if (kw) {
          const double tw = theta * dt * w;
          o[PR_XV] = make_double2(d.dxv * w, (rhoint - dt * theta * rhoint * itp(F_DADH)) * w +
                                                 tw * (rhoint * exx + drhodx * uint + rhoint * eyy + drhody * vint));
          o[PR_HC] = make_double2(tw * (rhoint * dhdx + drhodx * hint), tw * (rhoint * dhdy + drhody * hint));
          const double rh = tw * rhoint * hint, ru = tw * rhoint * uint, rv = tw * rhoint * vint;
          o[PR_HU] = make_double2(rh * ix, rh * jx);
          o[PR_HV] = make_double2(rh * iy, rh * jy);
          o[PR_HH] = make_double2(ru * ix + rv * iy, ru * jx + rv * jy);
        }
        const double2 gu0 = grad(F_U0), gv0 = grad(F_V0), gh0 = grad(F_H0);
        const double exx0 = ix * gu0.x + jx * gu0.y, eyy0 = iy * gv0.x + jy * gv0.y;
        const double dh0dx = ix * gh0.x + jx * gh0.y, dh0dy = iy * gh0.x + jy * gh0.y;
        const double qx1dx = rhoint * exx * hint + rhoint * uint * dhdx + drhodx * uint * hint;  // :39
        const double qy1dy = rhoint * eyy * hint + rhoint * vint * dhdy + drhody * vint * hint;
        const double qx0dx = rhoint * exx0 * h0int + rhoint * u0int * dh0dx + drhodx * u0int * h0int;
        const double qy0dy = rhoint * eyy0 * h0int + rhoint * v0int * dh0dy + drhody * v0int * h0int;
        const double qterm = dt * (theta * qx1dx + (1 - theta) * qx0dx + theta * qy1dy + (1 - theta) * qy0dy);
        const double acc = dt * rhoint * ((1 - theta) * itp(F_A0) + theta * itp(F_A1));
        o[PR_TF] = make_double2(-rhoint * (h0int - hint) * w, (acc - qterm) * w);  // h0barr = h1barr = 0
      }
      __syncthreads();
      // (b) rows
      if (el < gn_) {
        const double2* q = pts + (size_t)el * kIpc * kPairs;
        for (int pi = 0; pi < kIpc; ++pi, q += kPairs) {
          const double* N = sN + (ip0 + pi) * 6;
          const double2* dr = sD + (ip0 + pi) * 6;
          const double2 da = dr[a];
          const double Na = N[a];
          double2 gu, gv, gh = make_double2(0, 0);  // row vectors against u, v, h columns
          double nu, nv, nh;
          if (c < 2) {
            const double2 t = q[PR_TX + c], f = q[PR_PX + c], tn = q[PR_TN], fn = q[PR_FN];
            T += t.x * da.x + t.y * da.y + (c ? tn.y : tn.x) * Na;
            F += f.x * da.x + f.y * da.y + (c ? fn.y : fn.x) * Na;
            if (!kw) continue;
            const double2 dd = q[c ? PR_VV : PR_UU], dc = q[c ? PR_VVC : PR_UUC], c1 = q[PR_UV1], c2 = q[PR_UV2];
            const double2 xh = q[PR_XH + c], ch = q[PR_CH];
            const double2 diag = make_double2(dd.x * da.x + dd.y * da.y, dd.y * da.x + dc.x * da.y);
            const double2 off = c ? make_double2(c1.x * da.x + c1.y * da.y, c2.x * da.x + c2.y * da.y)
                                  : make_double2(c1.x * da.x + c2.x * da.y, c1.y * da.x + c2.y * da.y);
            const double nd_ = dc.y * Na, no_ = q[PR_XV].x * Na;
            gu = c ? off : diag;
            gv = c ? diag : off;
            nu = c ? no_ : nd_;
            nv = c ? nd_ : no_;
            nh = xh.x * da.x + xh.y * da.y + (c ? ch.y : ch.x) * Na;
          } else {
            const double2 sp = q[PR_S], tf = q[PR_TF];
            const double su = Na + sp.x * da.x + sp.y * da.y;  // SUPG test function (:55)
            T += tf.x * su;
            F += tf.y * su;
            if (!kw) continue;
            const double2 hc = q[PR_HC], hu = q[PR_HU], hv = q[PR_HV], hh = q[PR_HH];
            gu = make_double2(su * hu.x, su * hu.y);
            gv = make_double2(su * hv.x, su * hv.y);
            gh = make_double2(su * hh.x, su * hh.y);
            nu = su * hc.x;
            nv = su * hc.y;
            nh = su * q[PR_XV].y;
          }
#pragma unroll
          for (int b = 0; b < 6; ++b) {
            const double2 db = dr[b];
            const double Nb = N[b];
            ku[b] += gu.x * db.x + gu.y * db.y + nu * Nb;
            kv[b] += gv.x * db.x + gv.y * db.y + nv * Nb;
            kh[b] += nh * Nb;
            if (c == 2) kh[b] += gh.x * db.x + gh.y * db.y;  // the same for a warp
          }
        }
      }
      __syncthreads();  // the points are rewritten
    }
    if (el < gn_) {
      const size_t row = 6 * (size_t)(eb + el) + a;
      rel[6 * row + 2 * c] = T;
      rel[6 * row + 2 * c + 1] = F;
      if (kw) {
#pragma unroll
        for (int b = 0; b < 6; ++b) {
          double* o = kel + (row * 6 + b) * 9 + 3 * c;
          o[0] = ku[b];
          o[1] = kv[b];
          o[2] = kh[b];
        }
      }
    }
  }
}

// The patches' non-zeros and residuals from the element rows, in increasing global element order.
template <bool KW>
__global__ void __launch_bounds__(256) uvh_p2_gather(DevMesh M, const int* active, UvOut out, const double* kel,
                                                     const double* rel) {
  const int p = blockIdx.x, s = M.patch_sys[p];
  if (active && !active[s]) return;
  const int no = M.sys_node_off[s], nn_s = M.sys_node_off[s + 1] - no;
  const int uoff = M.sys_dof_off[s] - no, voff = uoff + nn_s, hoff = voff + nn_s;
  const int e0 = M.patch_elem_ptr[p], ne = M.patch_elem_ptr[p + 1] - e0;
  (void)ne;  // bounds-checked build
  const int pn0 = M.patch_node_ptr[p], nr = M.patch_node_ptr[p + 1] - pn0;
  if (KW) {
    const int q1 = M.patch_q_ptr[p + 1];
    const int nbase = M.nodeptr[no], nnzn = M.sys_nnzn[s], kbase = M.sys_knz_off[s];
    double* Ko = reinterpret_cast<double*>(out.K);
    for (int q = M.patch_q_ptr[p] + threadIdx.x; q < q1; q += blockDim.x) {
      const uint32_t rk = __ldg(M.pq_rk + q);
      const int r = rk >> 16, k = rk & 0xffff;
      const int gnd = __ldg(M.patch_nodes + pn0 + r);
      const int np0 = __ldg(M.nodeptr + gnd), deg = __ldg(M.nodeptr + gnd + 1) - np0, lp = np0 - nbase;
      double v[9] = {};
      const int cend = __ldg(M.pq_cptr + q + 1);
      for (int c = __ldg(M.pq_cptr + q); c < cend; ++c) {
        const uint16_t code = __ldg(M.contrib + c);
        int ce = code >> 6;
        const int a = (code >> 3) & 7, b = code & 7;
        bool ok = true;
        UA_CHECK_INDEX(M.dbg, ce, 0, ne, BS_CONTRIB_ELEM, ok);
        if (!ok) continue;
        int e = __ldg(M.patch_elems + e0 + ce);
        UA_CHECK_INDEX(M.dbg, e, 0, M.ne, BS_GATHER_ELEM, ok);
        if (!ok) continue;
        const double* src = kel + ((size_t)36 * e + 6 * a + b) * 9;
#pragma unroll
        for (int i = 0; i < 9; ++i) v[i] += src[i];
      }
      size_t last = (size_t)kbase + 6 * (size_t)nnzn + 3 * (size_t)lp + 2 * (size_t)deg + k;  // largest index
      bool okk = true;
      UA_CHECK_INDEX(M.dbg, last, (size_t)kbase, (size_t)M.sys_knz_off[s + 1], BS_K_INDEX, okk);
      (void)last;
      if (!okk) continue;
#pragma unroll
      for (int cr = 0; cr < 3; ++cr) {
        const size_t base = (size_t)kbase + (size_t)cr * 3 * nnzn + 3 * (size_t)lp;
#pragma unroll
        for (int cc = 0; cc < 3; ++cc) Ko[base + (size_t)cc * deg + k] = v[cr * 3 + cc];
      }
    }
  }
  for (int r = threadIdx.x; r < nr; r += blockDim.x) {
    int gnd = __ldg(M.patch_nodes + pn0 + r);
    bool okr = true;
    UA_CHECK_INDEX(M.dbg, gnd, no, no + nn_s, BS_R_INDEX, okr);
    if (!okr) continue;
    const int q = __ldg(M.prow_diag + pn0 + r);
    double acc[6] = {};
    const int cend = __ldg(M.pq_cptr + q + 1);
    for (int c = __ldg(M.pq_cptr + q); c < cend; ++c) {
      const uint16_t code = __ldg(M.contrib + c);
      int ce = code >> 6;
      const int a = (code >> 3) & 7;
      bool ok = true;
      UA_CHECK_INDEX(M.dbg, ce, 0, ne, BS_CONTRIB_ELEM, ok);
      if (!ok) continue;
      int e = __ldg(M.patch_elems + e0 + ce);
      UA_CHECK_INDEX(M.dbg, e, 0, M.ne, BS_GATHER_ELEM, ok);
      if (!ok) continue;
      const double* src = rel + ((size_t)6 * e + a) * 6;
#pragma unroll
      for (int i = 0; i < 6; ++i) acc[i] += src[i];
    }
    out.R[uoff + gnd] = acc[0] - acc[1];
    out.R[voff + gnd] = acc[2] - acc[3];
    out.R[hoff + gnd] = acc[4] - acc[5];
    if (out.Tint) { out.Tint[uoff + gnd] = acc[0]; out.Tint[voff + gnd] = acc[2]; out.Tint[hoff + gnd] = acc[4]; }
    if (out.Fext) { out.Fext[uoff + gnd] = acc[1]; out.Fext[voff + gnd] = acc[3]; out.Fext[hoff + gnd] = acc[5]; }
  }
}

// Groups of the element kernel: 21 elements on 384 threads with the tangent (one CTA an SM), 14 on 252
// without (two).
static cudaError_t launch_p2h(ua_mesh* m, const UvhPhys& P, const UvhIn& in, const UvOut& out) {
  using namespace p2h;
  if (quad_table(6).nip != kIps) return cudaErrorInvalidConfiguration;
  const bool kw = out.K != nullptr;
  const int G = kw ? 21 : 14, rows = kw ? 128 : 84, nsys = (int)m->sys.size();
  UvhElemRows& B = m->uvh_rows;
  if (!B.blk[kw]) {
    std::vector<int4> v;
    for (int s = 0; s < nsys; ++s)
      for (int e = m->h_elem_off[s]; e < m->h_elem_off[s + 1]; e += G)
        v.push_back(make_int4(s, e, std::min(G, m->h_elem_off[s + 1] - e), 0));
    int4* d = (int4*)dev_alloc(m, sizeof(int4) * std::max<size_t>(v.size(), 1));
    if (!d) return cudaErrorMemoryAllocation;
    cudaError_t e = dev_write(m, d, v.data(), sizeof(int4) * v.size());
    if (e != cudaSuccess) return e;
    B.blk[kw] = d;
    B.n[kw] = (int)v.size();
  }
  if (!B.rel && !(B.rel = (double*)dev_alloc(m, sizeof(double) * 36 * (size_t)m->dm.ne))) return cudaErrorMemoryAllocation;
  if (kw && !B.kel && !(B.kel = (double*)dev_alloc(m, sizeof(double) * 324 * (size_t)m->dm.ne)))
    return cudaErrorMemoryAllocation;
  const size_t sm = (size_t)G * kPoint + (size_t)kIps * 18 * 8 + (size_t)F_COUNT * 6 * G * 8;
  const bool gen = P.uv.law != UA_SLIDING_WEERTMAN || P.uv.melange;
  auto kern = kw ? (gen ? uvh_p2_elements<true, true> : uvh_p2_elements<false, true>)
                 : (gen ? uvh_p2_elements<true, false> : uvh_p2_elements<false, false>);
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynSmem);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
  if (e != cudaSuccess) return e;
  if (B.n[kw]) kern<<<B.n[kw], kw ? 384 : 256, sm, m->stream>>>(m->dm, quad_table(6), P, in, B.blk[kw], G, rows, B.kel, B.rel);
  if (kw) uvh_p2_gather<true><<<m->dm.npatch, 256, 0, m->stream>>>(m->dm, in.active, out, B.kel, B.rel);
  else uvh_p2_gather<false><<<m->dm.npatch, 256, 0, m->stream>>>(m->dm, in.active, out, B.kel, B.rel);
  return cudaGetLastError();
}

template <bool WITHK, typename KT>
static cudaError_t launch_p1h(const ua_mesh* m, const UvhPhys& P, const UvhIn& in, const UvOut& out) {
  const int E = m->dm.max_patch_elems;
  const size_t k = WITHK ? (((size_t)9 * NOD * NOD * E * sizeof(KT) + 15) & ~(size_t)15) : 0;
  const size_t sm = k + (size_t)6 * NOD * E * 8 + (size_t)F_COUNT * E * NOD * 8;
  // the residual-only pass keeps the general build: without the tangent its Weertman-only build
  // spills more registers than the general one
  auto kern = uvh_patch_kernel<WITHK, KT, true>;
  if constexpr (WITHK) {
    if (P.uv.law == UA_SLIDING_WEERTMAN && !P.uv.melange) kern = uvh_patch_kernel<WITHK, KT, false>;
  }
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynSmem);
  if (e != cudaSuccess) return e;
  const int threads = ((E * NOD + 31) / 32) * 32;
  if (threads > kThreads) return cudaErrorInvalidConfiguration;
  kern<<<m->dm.npatch, threads, sm, m->stream>>>(m->dm, quad_table(NOD), P, in, out);
  return cudaGetLastError();
}

cudaError_t launch_uvh_assembly(ua_mesh* m, const UvhPhys& P, const UvhIn& in, const UvOut& out, bool withK) {
  if (m->nod == NOD) return withK ? launch_p1h<true, double>(m, P, in, out) : launch_p1h<false, double>(m, P, in, out);
  UvOut o = out;
  if (!withK) o.K = nullptr;
  return launch_p2h(m, P, in, o);
}

}  // namespace ua
