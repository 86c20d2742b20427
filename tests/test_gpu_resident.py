"""The resident Krylov solves (PCG of the uv step, GMRES of the uvh step) against the launched ones.

The two use the same preconditioner in different forms (collapsed and plain V-cycle) and different
summation orders, and stop at the same tolerance, so the converged velocities agree within the
tolerances of the Newton solves (force tolerance 1e-20, i.e. a relative residual of 1e-10) and the
iteration counts nearly.
"""
import threading

import numpy as np
import pytest

import uasource_b200 as ua
from uasource_b200 import lib as L
from uasource_b200 import synth

pytestmark = pytest.mark.gpu
# as in the CSR comparison of the node slices
FORMS = {"fp64": (dict(precision=L.UA_PREC_FP64, krylov_rtol=1e-12), 1e-10),
         "mixed": (dict(precision=L.UA_PREC_MIXED, krylov_rtol=1e-6), 1e-7),
         "mixed_fp32_cycle": (dict(precision=L.UA_PREC_MIXED, krylov_rtol=1e-6, precond_bf16=0), 1e-7)}


def _uv(P, bcs=None, F=None, **kw):
    mua = ua.CreateMUA(P.coordinates, P.connectivity)
    ctrl = ua.CtrlVar(**kw).set_force_tolerance(1e-20)
    Fo, _, _, _, info = ua.uv(ctrl, mua, bcs or ua.BCs.from_problem(P), F or ua.Fields.from_problem(P))
    assert info.converged
    return np.concatenate([Fo.ub, Fo.vb]), info


# one CTA and a ragged slice; two CTAs; a P1 mesh of three levels and one of four (solo levels); P2 with
# linear and aggregated transfers
@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("nod,nx,ny,seed", [(3, 10, 7, 3), (3, 17, 9, 3), (3, 61, 43, 3), (3, 141, 71, 3), (6, 9, 6, 0),
                                            (6, 33, 17, 3)])
def test_resident_pcg_agrees_with_the_launched_one(nod, nx, ny, seed, form):
    P = synth.ice_stream_shelf(nx, ny, nod=nod, seed=seed)
    kw, tol = FORMS[form]
    a, ia = _uv(P, **kw)
    b, ib = _uv(P, krylov_sell=0, **kw)
    assert np.linalg.norm(a - b) <= tol * np.linalg.norm(b)
    # per Newton step a few iterations apart: rounding and the place of the BF16 values
    assert abs(ia.krylov_its_total - ib.krylov_its_total) <= 3 * ib.iterations + 0.1 * ib.krylov_its_total
    # a profiled solve reads its counts at once instead of with the costs
    c, ic = _uv(P, profile=1, **kw)
    assert np.array_equal(a, c) and ic.krylov_its_total == ia.krylov_its_total


def _fan(spokes=48, rings=9):
    """A disc whose centre touches `spokes` triangles: rows longer than the set-up's stage of 32."""
    r = np.arange(1, rings + 1) * 4e3
    th = 2 * np.pi * np.arange(spokes) / spokes
    xy = np.vstack([[0.0, 0.0], np.column_stack([np.outer(r, np.cos(th)).ravel(), np.outer(r, np.sin(th)).ravel()])])
    k = np.arange(spokes)
    k1 = (k + 1) % spokes
    tri = [np.column_stack([np.zeros(spokes, int), 1 + k, 1 + k1])]
    for q in range(rings - 1):
        a, b = 1 + q * spokes, 1 + (q + 1) * spokes
        tri += [np.column_stack([a + k, b + k, b + k1]), np.column_stack([a + k, b + k1, a + k1])]
    conn = np.vstack(tri)
    n = xy.shape[0]
    one = np.ones(n)
    B = 300.0 - 2e-3 * xy[:, 0]
    F = ua.Fields(h=1000.0 * one, S=0 * one, B=B, rho=917.0 * one, AGlen=1e-8 * one, n=3 * one, C=1e-4 * one, m=3 * one,
                  ub=0 * one, vb=0 * one)
    edge = np.arange(n - spokes, n)
    return xy, conn, F, ua.BCs(ubFixedNode=edge, ubFixedValue=np.zeros(spokes), vbFixedNode=edge,
                               vbFixedValue=np.zeros(spokes))


def test_setup_of_rows_longer_than_a_stage():
    xy, conn, F, bcs = _fan()
    mua = ua.CreateMUA(xy, conn)
    out = []
    for kw in (dict(), dict(krylov_sell=0), dict(krylov_precond=L.UA_PC_JACOBI)):
        Fo, _, _, _, info = ua.uv(ua.CtrlVar(**kw).set_force_tolerance(1e-20), mua, bcs, F.copy())
        assert info.converged
        out.append((np.concatenate([Fo.ub, Fo.vb]), info))
    for x, _ in out[:2]:
        assert np.linalg.norm(x - out[2][0]) <= 1e-10 * np.linalg.norm(out[2][0])
    # a wrong hierarchy would still converge, but in about the count of point Jacobi
    assert out[0][1].krylov_its_total < 0.5 * out[2][1].krylov_its_total


# 80 systems: two CTAs a team and several systems a queue; 30: teams of their own, some of one CTA.  The
# last system alone runs on ten CTAs with its coarse levels solo.
@pytest.mark.parametrize("form", ["fp64", "mixed"])
@pytest.mark.parametrize("count", [30, 80])
def test_team_size_does_not_change_a_result(count, form):
    kw, _ = FORMS[form]
    shapes = [(9 + k % 7, 6 + k % 4) for k in range(count - 2)] + [(45, 33), (41, 31)]
    probs = [synth.ice_stream_shelf(nx, ny, seed=k) for k, (nx, ny) in enumerate(shapes)]
    mua = ua.CreateMUABatch([(P.coordinates, P.connectivity) for P in probs])
    out = ua.uv_batch(ua.CtrlVar(**kw).set_force_tolerance(1e-20), mua, [ua.Fields.from_problem(P) for P in probs],
                      [ua.BCs.from_problem(P) for P in probs])
    for k in (0, 1, count - 2, count - 1):
        a, info = _uv(probs[k], **kw)
        assert np.array_equal(a, np.concatenate(out[k][:2])) and info.krylov_its_total == out[k][2].krylov_its_total


# sweeps: the default, one, an even count, more than the polynomial's sixteen; restart: several cycles,
# the longest resident one, and one past it (launched)
@pytest.mark.parametrize("nod,nx,ny,sweeps,restart", [(3, 10, 7, 0, 40), (3, 61, 43, 0, 40), (3, 61, 43, 1, 40),
                                                      (3, 33, 17, 4, 7), (3, 33, 17, 17, 48), (3, 33, 17, 0, 60),
                                                      (6, 9, 5, 0, 40), (6, 33, 17, 6, 12)])
def test_resident_gmres_agrees_with_the_launched_one(nod, nx, ny, sweeps, restart):
    P = synth.ice_stream_shelf(nx, ny, nod=nod, seed=4, transient=True)
    bcs = ua.BCs.from_problem(P)
    m2, m3 = (ua.CreateMUA(P.coordinates, P.connectivity, ndof=d) for d in (2, 3))
    F0 = ua.uv(ua.CtrlVar().set_force_tolerance(1e-20), m2, bcs, ua.Fields.from_problem(P))[0]
    out = []
    for sell in (1, 0):
        ctrl = ua.CtrlVar(krylov_sell=sell, uvh_h_sweeps=sweeps, krylov_restart=restart).set_force_tolerance(1e-20)
        F1, _, info = ua.uvh(ctrl.set_uvh_force_tolerance(1e-20), m3, F0, F0.copy(), bcs, 0.1)
        assert info.converged
        out.append((np.concatenate([F1.ub, F1.vb, F1.h]), info))
    (a, ia), (b, ib) = out
    assert np.linalg.norm(a - b) <= 1e-10 * np.linalg.norm(b)
    assert abs(ia.krylov_its_total - ib.krylov_its_total) <= 3 * ib.iterations + 0.1 * ib.krylov_its_total


# groups of elements and patches with remainders: one node a patch, a few, the default
@pytest.mark.parametrize("ndof", [2, 3], ids=["uv", "uvh"])
def test_p2_assembly_does_not_depend_on_the_patches(ndof):
    P = synth.ice_stream_shelf(14, 9, nod=6, seed=2, transient=True)
    rng = np.random.default_rng(1)
    mua = ua.CreateMUA(P.coordinates, P.connectivity, ndof=ndof)
    F = ua.Fields.from_problem(P)
    F.ub, F.vb = 100 + 200 * rng.random(P.Nnodes), 30 * rng.standard_normal(P.Nnodes)
    out = []
    for pn in (0, 1, 5, 29, 300):
        ctrl = ua.CtrlVar(patch_nodes=pn)
        if ndof == 2:
            Rv, K = ua.uvMatrixAssembly(ctrl, mua, F)
            Rr, _ = ua.uvMatrixAssembly(ctrl, mua, F, Ronly=True)
        else:
            Rv, K = ua.uvhAssembly(ctrl, mua, F, F.copy(), 0.1)
            Rr, _ = ua.uvhAssembly(ctrl, mua, F, F.copy(), 0.1, Ronly=True)
        assert np.array_equal(Rr, Rv)
        out.append((Rv, K.data.copy()))
    for Rv, Kd in out[1:]:
        assert np.array_equal(Rv, out[0][0]) and np.array_equal(Kd, out[0][1])


def test_solves_from_several_threads():
    """Handles of different sizes, each with its own stream: resident launches of two solves overlap, and no
    launch depends on what another thread set for its own."""
    probs = [synth.ice_stream_shelf(141, 71, seed=1), synth.ice_stream_shelf(101, 51, seed=2),
             synth.ice_stream_shelf(33, 17, nod=6, seed=3), synth.ice_stream_shelf(21, 11, seed=4)]
    ref = [_uv(P)[0] for P in probs]
    bad = []

    def run(k):
        try:
            bad.extend((k, r) for r in range(8) if not np.array_equal(_uv(probs[k])[0], ref[k]))
        except Exception as e:  # noqa: BLE001 - reported below
            bad.append((k, repr(e)))

    threads = [threading.Thread(target=run, args=(k,)) for k in range(len(probs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
