"""assembly_ms and solve_ms are the times of those phases, although the host only enqueues them: the assembly
holds its tangent kernels, the solve its set-up and Krylov iterations and nothing of the costs that follow, and
the two lie apart in the call's device time."""
import pytest

import uasource_b200 as ua
from uasource_b200 import synth

pytestmark = pytest.mark.gpu
EVENT = 0.002  # resolution of an event, ms


def _check(info):
    k = info.kernels
    spans = 2 * EVENT * (k["asmK_n"] + k["asmR_n"] + k["setup_n"] + k["krylov_n"])
    assert info.converged and info.assembly_ms > 0
    assert info.solve_ms >= k["setup_ms"] + k["krylov_ms"] - spans
    # residual assemblies belong to the costs, but one before the first step
    assert info.assembly_ms + info.solve_ms + k["asmR_ms"] <= info.device_ms + spans
    return k["asmK_ms"] - spans


@pytest.mark.parametrize("nod", [3, 6])
def test_uv(nod):
    P = synth.ice_stream_shelf(141, 71, nod=nod, seed=1)
    mua = ua.CreateMUA(P.coordinates, P.connectivity)
    info = ua.uv(ua.CtrlVar(profile=1).set_force_tolerance(1e-20), mua, ua.BCs.from_problem(P),
                 ua.Fields.from_problem(P))[4]
    _check(info)
    # one of the tangents is assembled in its step, the others ahead
    assert info.assembly_ms >= 0.5 * info.kernels["asmK_ms"] / info.kernels["asmK_n"]


@pytest.mark.parametrize("nod", [3, 6])
def test_uvh(nod):
    P = synth.ice_stream_shelf(141, 71, nod=nod, seed=1, transient=True)
    bcs = ua.BCs.from_problem(P)
    m2, m3 = (ua.CreateMUA(P.coordinates, P.connectivity, ndof=d) for d in (2, 3))
    F0 = ua.uv(ua.CtrlVar().set_force_tolerance(1e-20), m2, bcs, ua.Fields.from_problem(P))[0]
    info = ua.uvh(ua.CtrlVar(profile=1).set_uvh_force_tolerance(1e-20), m3, F0, F0.copy(), bcs, 0.1)[2]
    assert info.assembly_ms >= _check(info)  # every tangent in its step
