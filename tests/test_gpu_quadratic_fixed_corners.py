"""Quadratic meshes whose corner nodes are all held in a component, mid nodes between them free.  In exact
arithmetic a Krylov solve ends after as many steps as there are free dofs; a preconditioner that is no worse than
none stays below twice that with rounding.  (With held corners as coarse dofs the coarse operator was singular:
40206 iterations, and uvh steps that did not converge.)"""
import numpy as np
import pytest

import uasource_b200 as ua
from uasource_b200 import lib as L
from uasource_b200 import synth

pytestmark = pytest.mark.gpu
MESHES = [(2, 2), (3, 2)]


def _free(P, comps):
    return comps * P.Nnodes - len(P.ubFixedNode) - len(P.vbFixedNode)


@pytest.mark.parametrize("sell", [1, 0], ids=["resident", "launched"])
@pytest.mark.parametrize("form", ["fp64", "mixed"])
@pytest.mark.parametrize("nx,ny", MESHES)
def test_uv(nx, ny, form, sell):
    P = synth.ice_stream_shelf(nx, ny, nod=6, seed=0)
    mua, bcs = ua.CreateMUA(P.coordinates, P.connectivity), ua.BCs.from_problem(P)
    kw = dict(precision=L.UA_PREC_MIXED, krylov_rtol=1e-6) if form == "mixed" else {}

    def solve(**k):
        F, _, _, _, info = ua.uv(ua.CtrlVar(**k).set_force_tolerance(1e-20), mua, bcs, ua.Fields.from_problem(P))
        assert info.converged
        return np.concatenate([F.ub, F.vb]), info

    x, info = solve(krylov_sell=sell, **kw)
    ref, _ = solve(krylov_precond=L.UA_PC_JACOBI)
    assert info.krylov_its_total <= 2 * _free(P, 2) * info.iterations
    assert np.linalg.norm(x - ref) <= (1e-7 if kw else 1e-10) * np.linalg.norm(ref)


@pytest.mark.parametrize("sell", [1, 0], ids=["resident", "launched"])
@pytest.mark.parametrize("nx,ny", MESHES)
def test_uvh(nx, ny, sell):
    P = synth.ice_stream_shelf(nx, ny, nod=6, seed=4, transient=True)
    bcs = ua.BCs.from_problem(P)
    m2, m3 = (ua.CreateMUA(P.coordinates, P.connectivity, ndof=d) for d in (2, 3))
    F0 = ua.uv(ua.CtrlVar().set_force_tolerance(1e-20), m2, bcs, ua.Fields.from_problem(P))[0]
    ctrl = ua.CtrlVar(krylov_sell=sell).set_uvh_force_tolerance(1e-20)
    info = ua.uvh(ctrl, m3, F0, F0.copy(), bcs, 0.1)[2]
    assert info.converged
    assert info.krylov_its_total <= 2 * _free(P, 3) * info.iterations
