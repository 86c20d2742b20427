"""The calls that programs make of this framework, as cases to time and to compare.

Every case goes through the public entry points of ``uasource_b200`` on the ice stream / ice shelf of
``uasource_b200.synth`` (the diagnostic-solve workload), from the 21 x 11-vertex mesh of the smoke test to
meshes of 160,000 elements, linear (P1, nod 3) and quadratic (P2, nod 6), in FP64 and in the mixed form.  ``prepare`` holds what such
a program keeps: the resident mesh handle and host arrays of the fields.  ``run`` is one call; its outputs
are the arrays that the call returns.  ``exact`` restates the finite-element problem in plain torch in 64
bits (tangents by forward differentiation of the element residual) and solves it directly.
"""
import math

import numpy as np
import torch

import uasource_b200 as ua
from uasource_b200 import lib as L
from uasource_b200 import synth

TOL = 1e-20   # rForce at which a solve stops (the diagnostic-solve workload's tolerance)
DT = 0.1      # implicit step, years


def listed():
    return [
        # Drop-in of the MATLAB assembly (uvMatrixAssembly) on the smallest mesh in use: launches and latency.
        dict(name="asm_uv_p1_21x11", kind="asm", nod=3, nx=21, ny=11),
        # The same call for the transient tangent (uvhAssembly) on a quadratic mesh of ordinary size.
        dict(name="asm_uvh_p2_101x51", kind="asm_uvh", nod=6, nx=101, ny=51),
        # A diagnostic solve on the smallest mesh: test-sized problems, parameter studies.
        dict(name="uv_p1_21x11", kind="uv", nod=3, nx=21, ny=11, precision="fp64", warm=False),
        # The diagnostic-solve workload: one mesh of 19,600 elements from rest, plain FP64.
        dict(name="uv_p1_141x71", kind="uv", nod=3, nx=141, ny=71, precision="fp64", warm=False),
        # A run's next diagnostic solve: the velocities of the last one as the start, a changed slipperiness.
        dict(name="uv_p1_229x113_warm", kind="uv", nod=3, nx=229, ny=113, precision="mixed", warm=True),
        # Quadratic elements, the mixed form.
        dict(name="uv_p2_101x51_mixed", kind="uv", nod=6, nx=101, ny=51, precision="mixed", warm=False),
        # The largest single mesh here: 160,000 quadratic elements, 321,201 nodes, plain FP64.
        dict(name="uv_p2_401x201", kind="uv", nod=6, nx=401, ny=201, precision="fp64", warm=False),
        # Many meshes of uneven size in one handle (2k to 200k elements, log-uniform), pinned host arrays in and out.
        dict(name="batch16_mixed", kind="batch", count=16, lo=2000, hi=200000, precision="mixed"),
        # The same in plain FP64, with fewer and smaller meshes.
        dict(name="batch8", kind="batch", count=8, lo=2000, hi=100000, precision="fp64"),
        # One implicit thickness-velocity step from the diagnostic state, quadratic elements.
        dict(name="uvh_p2_101x51", kind="uvh", nod=6, nx=101, ny=51),
        # The same on linear elements.
        dict(name="uvh_p1_141x71", kind="uvh", nod=3, nx=141, ny=71),
        # One gradient of an inversion: adjoint solve and dI/dlog10(C) at a solved state.
        dict(name="adjoint_p1_141x71", kind="adjoint", nod=3, nx=141, ny=71),
    ]


def draw(rng):
    def grid(lo, hi):
        """Vertices of a rectangle of lo .. hi triangles, log-uniform, of uneven aspect."""
        ne = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        aspect = rng.uniform(1.6, 2.5)
        ny = max(10, round(math.sqrt(ne / (2 * aspect))) + 1)
        return dict(nx=max(18, round(aspect * (ny - 1)) + 1), ny=ny)

    kind = rng.choice(["asm", "asm_uvh", "uv", "uv", "uv", "batch", "batch", "uvh", "adjoint"])
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(3, 12), lo=rng.randint(1500, 4000), hi=rng.randint(20000, 100000),
                    precision=rng.choice(["fp64", "mixed"]))
    nod = rng.choice([3, 6])
    case = dict(kind=kind, nod=nod)
    if kind in ("asm", "asm_uvh"):
        case.update(grid(400 if nod == 3 else 4000, 20000 if kind == "asm" else 10000))
    elif kind == "uv":
        case.update(grid(400 if nod == 3 else 4000, 100000 if nod == 3 else 50000))
        case.update(precision=rng.choice(["fp64", "mixed"]), warm=rng.random() < 0.3)
    elif kind == "uvh":
        case.update(grid(1500 if nod == 3 else 4000, 20000 if nod == 3 else 10000))
    else:
        case.update(nod=3, **grid(800, 30000))
    return case


# --------------------------------------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------------------------------------

FIELDS = ("h", "S", "B", "rho", "AGlen", "n", "C", "m", "ub", "vb")


def _problem(case, seed):
    return synth.ice_stream_shelf(case["nx"], case["ny"], nod=case["nod"], seed=seed, transient=case["kind"] == "uvh")


def _batch_problems(case, seed):
    out = []
    for k, ne in enumerate(synth.batch_sizes(case["count"], case["lo"], case["hi"])):
        nx, ny = synth.elements_to_grid(int(ne))
        out.append(synth.ice_stream_shelf(nx, ny, nod=3, seed=1000 * seed + k))
    return out


def _assembly_state(P, seed):
    """A velocity field of the size and smoothness of a Newton iterate, and an evolving thickness."""
    rng = np.random.default_rng(seed)
    x, y = P.coordinates[:, 0] / 100e3, P.coordinates[:, 1] / 50e3
    a = rng.uniform(0.8, 1.2, 4)
    u = 900 * a[0] * x * (1 + 0.3 * np.sin(math.pi * y * a[1]))
    v = 60 * a[2] * np.sin(2 * math.pi * x) * np.sin(math.pi * y)
    h = P.h + 5 * np.sin(3 * math.pi * x * a[3]) * np.cos(math.pi * y)
    return u, v, h


def _ctrl(case):
    mixed = case.get("precision") == "mixed"
    c = ua.CtrlVar(precision=L.UA_PREC_MIXED if mixed else L.UA_PREC_FP64, krylov_rtol=1e-6 if mixed else 1e-12)
    return c.set_force_tolerance(TOL).set_uvh_force_tolerance(TOL)


def _changed_C(P, seed):
    """The slipperiness of a next solve: a smooth change of some 10 per cent."""
    rng = np.random.default_rng(seed + 77)
    x, y = P.coordinates[:, 0] / 100e3, P.coordinates[:, 1] / 50e3
    a = rng.uniform(0, 2 * math.pi, 2)
    return P.C * np.exp(0.1 * np.sin(4 * math.pi * x + a[0]) * np.sin(2 * math.pi * y + a[1]))


def _measured(P, u, v, seed):
    """Surface velocities as measured: the model's with noise, and their errors."""
    rng = np.random.default_rng(seed + 99)
    us = u * (1 + 0.05 * rng.standard_normal(P.Nnodes)) + rng.standard_normal(P.Nnodes)
    vs = v + 2 * rng.standard_normal(P.Nnodes)
    return us, vs, 1 + rng.random(P.Nnodes), 1 + rng.random(P.Nnodes)


def _pinned(a):
    t = torch.empty(a.size, dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy()
    t[:] = a
    return t


def prepare(case, seed):
    kind = case["kind"]
    st = dict(case=case, ctrl=_ctrl(case))
    if kind == "batch":
        Ps = _batch_problems(case, seed)
        st["mua"] = ua.CreateMUABatch([(P.coordinates, P.connectivity) for P in Ps])
        st["F"] = [ua.Fields(rhow=P.rhow, g=P.g, alpha=P.alpha, **{k: _pinned(getattr(P, k)) for k in FIELDS})
                   for P in Ps]
        st["bcs"] = [ua.BCs.from_problem(P) for P in Ps]
        st["out"] = [(_pinned(np.zeros(P.Nnodes)), _pinned(np.zeros(P.Nnodes))) for P in Ps]
        return st
    P = _problem(case, seed)
    F = ua.Fields.from_problem(P)
    bcs = ua.BCs.from_problem(P)
    st.update(F=F, bcs=bcs)
    if kind in ("asm", "asm_uvh"):
        st["mua"] = ua.CreateMUA(P.coordinates, P.connectivity, ndof=2 if kind == "asm" else 3)
        u, v, h = _assembly_state(P, seed)
        F.ub, F.vb = u, v
        if kind == "asm_uvh":
            F0 = F.copy()
            F0.ub, F0.vb = 0.97 * u, 0.97 * v
            F.h = h
            F0.as_ = F.as_ = np.full(P.Nnodes, 0.3)
            st["F0"] = F0
        return st
    if kind == "uv":
        st["mua"] = ua.CreateMUA(P.coordinates, P.connectivity)
        if case["warm"]:
            Fo = ua.uv(st["ctrl"], st["mua"], bcs, F)[0]
            F.ub, F.vb, F.C = Fo.ub, Fo.vb, _changed_C(P, seed)
        return st
    # an implicit step and an inversion start from a solved diagnostic state
    m2 = ua.CreateMUA(P.coordinates, P.connectivity)
    Fo = ua.uv(_ctrl(case), m2, bcs, F)[0]
    F.ub, F.vb = Fo.ub, Fo.vb
    if kind == "adjoint":
        st["mua"] = m2
        st["data"] = _measured(P, F.ub, F.vb, seed)
        return st
    m2.close()
    st["mua"] = ua.CreateMUA(P.coordinates, P.connectivity, ndof=3)
    st["bcs"] = ua.HBCs(ubFixedNode=bcs.ubFixedNode, ubFixedValue=bcs.ubFixedValue, vbFixedNode=bcs.vbFixedNode,
                        vbFixedValue=bcs.vbFixedValue)
    return st


def run(state):
    kind, ctrl, mua, F, bcs = (state["case"]["kind"], state["ctrl"], state["mua"], state["F"], state["bcs"])
    if kind == "asm":
        R, K = ua.uvMatrixAssembly(ctrl, mua, F, bcs)
        return dict(R=R, K=K.data)
    if kind == "asm_uvh":
        R, K = ua.uvhAssembly(ctrl, mua, state["F0"], F, DT)
        return dict(R=R, K=K.data)
    if kind == "uv":
        Fo = ua.uv(ctrl, mua, bcs, F)[0]
        return dict(ub=Fo.ub, vb=Fo.vb)
    if kind == "batch":
        res = ua.uv_batch(ctrl, mua, F, bcs, out=state["out"])
        return [dict(ub=r[0], vb=r[1]) for r in res]
    if kind == "uvh":
        Fo = ua.uvh(ctrl, mua, F, F, bcs, DT)[0]
        return dict(ub=Fo.ub, vb=Fo.vb, h=Fo.h)
    I, dIduv, lam, g, _ = ua.adjoint_gradient_C(ctrl, mua, F, bcs, *state["data"])
    return dict(I=I, dIduv=dIduv, lam=lam, dIdC=g)


# --------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# --------------------------------------------------------------------------------------------------------

def work(case):
    """Inputs read once and outputs written once, for a solve also its tangent once; the operations of one
    tangent at each of the least Newton steps that a solve takes (from rest 9, from a near state 4)."""
    def sizes(nx, ny, nod):
        ne = 2 * (nx - 1) * (ny - 1)
        return ne, nx * ny if nod == 3 else (2 * nx - 1) * (2 * ny - 1)

    if case["kind"] == "batch":
        parts = [(*sizes(*synth.elements_to_grid(int(ne)), 3), 3) for ne in
                 synth.batch_sizes(case["count"], case["lo"], case["hi"])]
    else:
        parts = [(*sizes(case["nx"], case["ny"], case["nod"]), case["nod"])]
    dof = 3 if case["kind"] in ("uvh", "asm_uvh") else 2
    steps = {"asm": 1, "asm_uvh": 1, "uvh": 4, "adjoint": 1}.get(case["kind"], 4 if case.get("warm") else 9)
    nbytes = flops = 0.0
    for ne, nn, nod in parts:
        nnz = dof * dof * nn * (7 if nod == 3 else 11.5)
        fields = {"uvh": 19, "asm_uvh": 17, "adjoint": 22}.get(case["kind"], 12)
        nbytes += 8 * (fields * nn + nnz) + 4 * nod * ne
        per_point = 60 + 12 * nod + 30 * dof + nod * nod * dof * dof * 8
        flops += steps * ne * (6 if nod == 3 else 16) * per_point
    return dict(bytes=nbytes, flops=flops)


# --------------------------------------------------------------------------------------------------------
# the same in plain torch, 64 bits
# --------------------------------------------------------------------------------------------------------

def _rule(nod):
    """Points (xi, eta) and weights of the fully symmetric rules of degree 4 (P1) and 8 (P2)."""
    if nod == 3:
        s = math.sqrt(38 - 44 * math.sqrt(0.4))
        t = math.sqrt(213125 - 53320 * math.sqrt(10))
        orbits = [(3, (8 - math.sqrt(10) + s) / 18, None, (620 + t) / 3720),
                  (3, (8 - math.sqrt(10) - s) / 18, None, (620 - t) / 3720)]
    else:
        orbits = [(1, 1 / 3, None, 0.1443156076777871682510911104890646),
                  (3, 0.1705693077517602066222935014914645, None, 0.1032173705347182502817915502921290),
                  (3, 0.0505472283170309754584235505965989, None, 0.0324584976231980803109259283417806),
                  (3, 0.4592925882927231560288155144941693, None, 0.0950916342672847246938961043885843),
                  (6, 0.2631128296346381134217857862846436, 0.0083947774099576053372138345392944,
                   0.0272303141744349942648446900739089)]
    pts, wts = [], []
    for m, p, q, w in orbits:
        q = p if q is None else q
        r = 1 - p - q
        ring = {1: [(p, q, r)], 3: [(p, q, r), (q, r, p), (r, p, q)],
                6: [(p, q, r), (q, r, p), (r, p, q), (p, r, q), (q, p, r), (r, q, p)]}[m]
        pts += [(b, c) for _, b, c in ring]
        wts += [0.5 * w] * m
    return pts, wts


def _shapes(nod, pts):
    N, D = [], []
    for a, b in pts:
        c = 1 - a - b
        if nod == 3:
            N.append([a, c, b])
            D.append([[1, -1, 0], [0, -1, 1]])
        else:
            N.append([(2 * a - 1) * a, 4 * c * a, (2 * c - 1) * c, 4 * b * c, (2 * b - 1) * b, 4 * a * b])
            D.append([[4 * a - 1, 4 * (c - a), -(4 * c - 1), -4 * b, 0, 4 * b],
                      [0, -4 * a, -(4 * c - 1), 4 * (c - b), 4 * b - 1, 4 * a]])
    return N, D


class _Exact:
    """The SSA problem of one mesh: residual, tangent and direct solves in torch, float64."""
    eps0, u0, eta0, kH, theta = 1e-10, 1e-4, 10.0, 1.0, 0.5

    def __init__(self, P, case):
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        t = lambda a: torch.as_tensor(np.asarray(a), dtype=torch.float64, device=self.dev)
        self.P, self.nn, self.nod = P, P.Nnodes, P.nod
        self.conn = torch.as_tensor(P.connectivity.astype(np.int64), device=self.dev)
        pts, wts = _rule(self.nod)
        N, D = _shapes(self.nod, pts)
        self.N, D = t(N), t(D)                                                  # [q, a], [q, 2, a]
        xy = t(P.coordinates)[self.conn]                                        # [e, a, 2]
        J = torch.einsum("qda,eac->eqdc", D, xy)
        det = J[..., 0, 0] * J[..., 1, 1] - J[..., 0, 1] * J[..., 1, 0]
        self.Dx = (J[..., 1, 1, None] * D[None, :, 0] - J[..., 0, 1, None] * D[None, :, 1]) / det[..., None]
        self.Dy = (-J[..., 1, 0, None] * D[None, :, 0] + J[..., 0, 0, None] * D[None, :, 1]) / det[..., None]
        self.w = det * t(wts)
        corner = xy if self.nod == 3 else xy[:, [0, 2, 4]]
        d1, d2 = corner[:, 1] - corner[:, 0], corner[:, 2] - corner[:, 0]
        self.area = 0.5 * (d1[:, 0] * d2[:, 1] - d1[:, 1] * d2[:, 0]).abs()
        self.f = {k: t(getattr(P, k)) for k in FIELDS}
        # nodes in vertical strips: an element reaches from its strip into the next one at most
        col = np.unique(np.round(P.coordinates[:, 0], 3), return_inverse=True)[1].ravel()
        per = 1 if self.nod == 3 else 2
        self.rows = int(np.bincount(col).max())
        self.strip0 = torch.as_tensor(col // per, device=self.dev)
        self.per = per

    def flotation(self, h):
        f, P = self.f, self.P
        hf = P.rhow * (f["S"] - f["B"]) / f["rho"]
        gf = 0.5 + 0.5 * torch.tanh(self.kH * (h - hf))
        return gf * f["B"] + (1 - gf) * (f["S"] - f["rho"] * h / P.rhow)

    def element_residual(self, x, b, prev, sel):
        """Residual [e, dof, a] at the element values x [e, dof, a] of (u, v) or (u, v, h); b: the nodal lower
        surface; prev: (u, v, h, a0, a1) of an implicit step, elements sel."""
        f, P, conn = self.f, self.P, self.conn[sel]
        Dx, Dy, w, N = self.Dx[sel], self.Dy[sel], self.w[sel], self.N
        at = lambda v: v @ N.T
        dx, dy = (lambda v: torch.einsum("eqa,ea->eq", Dx, v)), (lambda v: torch.einsum("eqa,ea->eq", Dy, v))
        u, v = x[:, 0], x[:, 1]
        h = x[:, 2] if prev is not None else self.h_el[sel]
        rho = at(f["rho"][conn])
        H = at(f["S"][conn]) - at(f["B"][conn])
        hi, ui, vi = at(h), at(u), at(v)
        hf = P.rhow * H / rho
        he = 0.5 + 0.5 * torch.tanh(self.kH * (hi - hf))
        hE = 0.5 + 0.5 * torch.tanh(self.kH * (hf - hi))
        d = hE * rho * hi / P.rhow + he * (0.5 + 0.5 * torch.tanh(self.kH * H)) * H
        exx, eyy, exy = dx(u), dy(v), 0.5 * (dx(v) + dy(u))
        n, m = at(f["n"][conn]), at(f["m"][conn])
        A, C = at(f["AGlen"][conn]).clamp_min(1e-20), at(f["C"][conn]).clamp_min(1e-20)
        e = torch.sqrt(self.eps0 ** 2 + exx ** 2 + eyy ** 2 + exx * eyy + exy ** 2)
        eta = 0.5 * A ** (-1 / n) * e ** ((1 - n) / n) + self.eta0
        beta = he * C ** (-1 / m) * torch.sqrt(ui ** 2 + vi ** 2 + self.u0 ** 2) ** (1 / m - 1)
        bn = b[conn]
        p1 = P.g * (rho * hi - P.rhow * d) * w
        p2 = 0.5 * P.g * (rho * hi ** 2 - P.rhow * d ** 2) * w
        s = hi * eta * w
        wx = lambda c: torch.einsum("eq,eqa->ea", c, Dx)
        wy = lambda c: torch.einsum("eq,eqa->ea", c, Dy)
        wn = lambda c: c @ N
        rx = wx(s * (4 * exx + 2 * eyy) - p2) + wy(2 * s * exy) + wn(beta * ui * w + p1 * dx(bn))
        ry = wy(s * (4 * eyy + 2 * exx) - p2) + wx(2 * s * exy) + wn(beta * vi * w + p1 * dy(bn))
        if prev is None:
            return torch.stack([rx, ry], 1)
        u0, v0, h0, a0, a1 = (p[conn] for p in prev)
        ui0, vi0, hi0 = at(u0), at(v0), at(h0)
        rx_, ry_ = dx(f["rho"][conn]), dy(f["rho"][conn])
        q1 = rho * exx * hi + rho * ui * dx(h) + rx_ * ui * hi + rho * eyy * hi + rho * vi * dy(h) + ry_ * vi * hi
        q0 = (rho * dx(u0) * hi0 + rho * ui0 * dx(h0) + rx_ * ui0 * hi0 + rho * dy(v0) * hi0 + rho * vi0 * dy(h0)
              + ry_ * vi0 * hi0)
        tau = torch.sqrt(2 * self.area[sel])[:, None] / (2 * torch.sqrt(ui0 ** 2 + vi0 ** 2 + self.u0 ** 2) + self.u0)
        th = self.theta
        c = (rho * (hi - hi0) + DT * (th * q1 + (1 - th) * q0) - DT * rho * ((1 - th) * at(a0) + th * at(a1))) * w
        rh = wn(c) + wx(0.5 * tau * ui0 * c) + wy(0.5 * tau * vi0 * c)
        return torch.stack([rx, ry, rh], 1)

    def element_parts(self, X, prev=None, tangent=True):
        """(residual vector of dof * nn, element tangents [e, dof * nod, dof * nod] or None) at X [dof, nn]."""
        ndof = X.shape[0]
        h = X[2] if prev is not None else self.f["h"]
        b = self.flotation(h)
        self.h_el = self.f["h"][self.conn]
        ne = self.conn.shape[0]
        R = torch.zeros(ndof, self.nn, dtype=torch.float64, device=self.dev)
        Ks = []
        for lo in range(0, ne, 40000):
            sel = slice(lo, min(ne, lo + 40000))
            x = X[:, self.conn[sel]].permute(1, 0, 2).contiguous()
            fun = lambda z: self.element_residual(z, b, prev, sel)
            r = fun(x)
            for c in range(ndof):
                R[c].index_add_(0, self.conn[sel].reshape(-1), r[:, c].reshape(-1))
            if tangent:
                cols = []
                for k in range(ndof * self.nod):
                    e = torch.zeros_like(x)
                    e[:, k // self.nod, k % self.nod] = 1
                    cols.append(torch.func.jvp(fun, (x,), (e,))[1].reshape(x.shape[0], -1))
                Ks.append(torch.stack(cols, 2))
        return R.reshape(-1), torch.cat(Ks) if tangent else None

    def dofs(self, ndof):
        """Global dof of each element dof [e, ndof * nod]."""
        return torch.cat([self.conn + c * self.nn for c in range(ndof)], 1)

    def csr_values(self, Ke, ndof):
        """Values on the structural pattern, rows and columns in order."""
        g, n = self.dofs(ndof), ndof * self.nn
        key = (g[:, :, None] * n + g[:, None, :]).reshape(-1)
        pos, inv = torch.unique(key, return_inverse=True)
        return torch.zeros(pos.numel(), dtype=torch.float64, device=self.dev).index_add_(0, inv, Ke.reshape(-1))

    def solver(self, Ke, ndof, fixed):
        """A direct solver of the constrained tangent (fixed: mask of dofs): block elimination over strips."""
        dev, nn = self.dev, self.nn
        merge = max(1, 700 // (self.per * self.rows * ndof))
        strip = self.strip0 // merge
        ns = int(strip.max()) + 1
        order = torch.argsort(strip, stable=True)
        count = torch.bincount(strip, minlength=ns)
        rank = torch.empty_like(order)
        rank[order] = torch.arange(nn, device=dev) - torch.repeat_interleave(torch.cumsum(count, 0) - count, count)
        width = int(count.max())
        m = width * ndof
        S = strip.repeat(ndof)
        Rk = torch.cat([rank + c * width for c in range(ndof)])
        A = torch.zeros(3, ns, m, m, dtype=torch.float64, device=dev)           # below, on, above the diagonal
        g = self.dofs(ndof)
        free = ~fixed
        K = Ke * (free[g][:, :, None] & free[g][:, None, :])
        si, sj = S[g][:, :, None].expand_as(K), S[g][:, None, :].expand_as(K)
        idx = (((sj - si + 1) * ns + si) * m + Rk[g][:, :, None]) * m + Rk[g][:, None, :]
        A.view(-1).index_add_(0, idx.reshape(-1), K.reshape(-1))
        ones = torch.ones(ns, m, dtype=torch.float64, device=dev)
        ones[S[free], Rk[free]] = 0                                              # fixed dofs and padding
        A[1].diagonal(dim1=1, dim2=2).add_(ones)
        lus = []
        for i in range(ns):
            D = A[1, i]
            if i:
                D = D - A[0, i] @ torch.linalg.lu_solve(*lus[-1], A[2, i - 1])
            lus.append(torch.linalg.lu_factor(D))

        def solve(b):
            y = torch.zeros(ns, m, dtype=torch.float64, device=dev)
            y[S, Rk] = b * free
            for i in range(1, ns):
                y[i] -= A[0, i] @ torch.linalg.lu_solve(*lus[i - 1], y[i - 1][:, None])[:, 0]
            y[-1] = torch.linalg.lu_solve(*lus[-1], y[-1][:, None])[:, 0]
            for i in range(ns - 2, -1, -1):
                y[i] = torch.linalg.lu_solve(*lus[i], (y[i] - A[2, i] @ y[i + 1])[:, None])[:, 0]
            return y[S, Rk]

        return solve

    def fixed(self, ndof):
        mask = torch.zeros(ndof * self.nn, dtype=torch.bool, device=self.dev)
        mask[torch.as_tensor(self.P.ubFixedNode.astype(np.int64), device=self.dev)] = True
        mask[torch.as_tensor(self.P.vbFixedNode.astype(np.int64), device=self.dev) + self.nn] = True
        return mask

    def newton(self, X, prev=None):
        """Newton with halved steps to the rounding of the residual; all boundary values are zero."""
        ndof = X.shape[0]
        fixed = self.fixed(ndof)
        X = X.clone()
        X.reshape(-1)[fixed] = 0
        R, Ke = self.element_parts(X, prev)
        norm, still = float((R * ~fixed).norm()), 0
        for _ in range(60):
            dx = self.solver(Ke, ndof, fixed)(-R).reshape(ndof, self.nn)
            step = 1.0
            while step > 1e-3:
                trial = X + step * dx
                r = float((self.element_parts(trial, prev, tangent=False)[0] * ~fixed).norm())
                if r < norm * (1 - 1e-3 * step) or float(dx.norm()) < 1e-9 * float(X.norm()):
                    break
                step *= 0.5
            small = float(dx.norm()) < 1e-9 * float(trial.norm())
            X, norm, still = trial, r, still + small
            if still >= 2:
                break
            R, Ke = self.element_parts(X, prev)
        return X


def _np(t):
    return t.cpu().numpy()


def _uv_state(P, case):
    E = _Exact(P, case)
    return E, E.newton(torch.stack([E.f["ub"], E.f["vb"]]))


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        Ps, out = _batch_problems(case, seed), []
        small = sorted(range(len(Ps)), key=lambda k: Ps[k].Nnodes)[:4]           # direct solves of the smallest
        for k, P in enumerate(Ps):
            X = _uv_state(P, case)[1] if k in small else None
            out.append(None if X is None else dict(ub=_np(X[0]), vb=_np(X[1])))
        return out
    if kind == "uv" and case["nx"] * case["ny"] * case["nod"] > 160000:
        return None
    P = _problem(case, seed)
    if kind in ("asm", "asm_uvh"):
        u, v, h = _assembly_state(P, seed)
        E = _Exact(P, case)
        t = lambda a: torch.as_tensor(a, dtype=torch.float64, device=E.dev)
        prev, X = None, torch.stack([t(u), t(v)])
        if kind == "asm_uvh":
            a = torch.full_like(X[0], 0.3)
            prev, X = (t(0.97 * u), t(0.97 * v), t(P.h), a, a), torch.stack([t(u), t(v), t(h)])
        R, Ke = E.element_parts(X, prev)
        return dict(R=_np(R), K=_np(E.csr_values(Ke, X.shape[0])))
    if kind == "uv" and case["warm"]:
        P.C = _changed_C(P, seed)
    E, X = _uv_state(P, case)
    if kind == "uv":
        return dict(ub=_np(X[0]), vb=_np(X[1]))
    if kind == "uvh":
        t = lambda a: torch.as_tensor(a, dtype=torch.float64, device=E.dev)
        a = t(P.as_ + P.ab)
        X = E.newton(torch.stack([X[0], X[1], E.f["h"]]), (X[0], X[1], E.f["h"], a, a))
        return dict(ub=_np(X[0]), vb=_np(X[1]), h=_np(X[2]))
    # the adjoint gradient: misfit with the mass matrix, adjoint velocities, dI/dlog10(C), mass-matrix solve
    u, v = X
    us, vs, ue, ve = (torch.as_tensor(a, dtype=torch.float64, device=E.dev) for a in
                      _measured(P, _np(u), _np(v), seed))
    Me = torch.einsum("eq,qa,qb->eab", E.w, E.N, E.N)
    area = float(E.area.sum())
    mass = lambda z: torch.zeros_like(z).index_add_(0, E.conn.reshape(-1), (Me @ z[E.conn][..., None]).reshape(-1))
    ru, rv = (u - us) / ue, (v - vs) / ve
    mu, mv = mass(ru), mass(rv)
    I = float(ru @ mu + rv @ mv) / 2 / area
    dI = torch.cat([mu / ue, mv / ve]) / area
    lam = E.solver(E.element_parts(X)[1], 2, E.fixed(2))(dI)
    f, N, conn = E.f, E.N, E.conn
    at = lambda z: z[conn] @ N.T
    hf = P.rhow * (f["S"] - f["B"]) / f["rho"]
    he = 0.5 + 0.5 * torch.tanh(at(f["h"]) - at(hf))
    ui, vi, m = at(u), at(v), at(f["m"])
    c = (he / m * at(f["C"]).clamp_min(1e-20) ** (-1 / m - 1) * torch.sqrt(ui ** 2 + vi ** 2 + E.u0 ** 2) ** (1 / m - 1)
         * (ui * at(lam[:E.nn]) + vi * at(lam[E.nn:])) * E.w)
    g = torch.zeros_like(u).index_add_(0, conn.reshape(-1), (c @ N).reshape(-1)) * math.log(10) * f["C"]
    none = torch.zeros(E.nn, dtype=torch.bool, device=E.dev)
    g = E.solver(Me / area, 1, none)(g)
    return dict(I=I, dIduv=_np(dI), lam=_np(lam), dIdC=_np(g))
