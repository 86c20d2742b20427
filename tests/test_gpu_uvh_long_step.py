"""Implicit steps of several cells' advection: the thickness block is far from symmetric there.  More l1-Jacobi
sweeps on it make a better preconditioner, and the default ones take no more than half as many iterations again
as eight (plain sweeps: 533 and 513, 675 and 469, 631 and 593; weighted ones 2514 and 545, 566 and 4752)."""
import pytest

import uasource_b200 as ua
from uasource_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sell", [1, 0], ids=["resident", "launched"])
@pytest.mark.parametrize("nod,nx,ny,dt", [(3, 61, 43, 0.5), (6, 33, 17, 0.5), (3, 141, 71, 0.3)])
def test_sweeps_at_long_steps(nod, nx, ny, dt, sell):
    P = synth.ice_stream_shelf(nx, ny, nod=nod, seed=1, transient=True)
    bcs = ua.BCs.from_problem(P)
    m2, m3 = (ua.CreateMUA(P.coordinates, P.connectivity, ndof=d) for d in (2, 3))
    F0 = ua.uv(ua.CtrlVar().set_force_tolerance(1e-20), m2, bcs, ua.Fields.from_problem(P))[0]
    its = []
    for sweeps in (0, 8):
        ctrl = ua.CtrlVar(uvh_h_sweeps=sweeps, krylov_maxit=2000, krylov_sell=sell).set_uvh_force_tolerance(1e-20)
        info = ua.uvh(ctrl, m3, F0, F0.copy(), bcs, dt)[2]
        assert info.converged
        its.append(info.krylov_its_total)
    assert its[1] <= its[0] <= 1.5 * its[1]
