"""precond_bf16 = 0 keeps the whole V-cycle of the mixed form in FP32 beside its prolongator: the collapsed
cycle of the resident PCG then is the launched cycle up to FP32 rounding, which moves the iteration at which a
system passes its tolerance by one at most.  (Its transfer held in BF16 took two more.)"""
import pytest

import uasource_b200 as ua
from uasource_b200 import lib as L
from uasource_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nod,nx,ny", [(3, 61, 43), (6, 101, 51)])
def test_the_fp32_cycle_takes_the_launched_one_s_iterations(nod, nx, ny):
    P = synth.ice_stream_shelf(nx, ny, nod=nod, seed=3)
    mua = ua.CreateMUA(P.coordinates, P.connectivity)
    info = []
    for sell in (1, 0):
        ctrl = ua.CtrlVar(precision=L.UA_PREC_MIXED, krylov_rtol=1e-6, precond_bf16=0, krylov_sell=sell)
        info.append(ua.uv(ctrl.set_force_tolerance(1e-20), mua, ua.BCs.from_problem(P), ua.Fields.from_problem(P))[4])
        assert info[-1].converged
    a, b = info
    assert a.iterations == b.iterations
    assert a.krylov_its_total <= b.krylov_its_total + b.iterations
