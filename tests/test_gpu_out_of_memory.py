"""Calls that run out of device memory say so and leave the handle usable.

Another allocation takes all but a set number of bytes of the device; the library's next cudaMalloc then
fails with an error, nothing more.
"""
import contextlib

import numpy as np
import pytest

import uasource_b200 as ua
from uasource_b200 import lib as L
from uasource_b200 import synth

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def _left(nbytes):
    """Only nbytes of the device are free inside."""
    torch = pytest.importorskip("torch")
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    hold = torch.empty(torch.cuda.mem_get_info()[0] - int(nbytes), dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del hold
        torch.cuda.empty_cache()


def test_quadratic_assembly_without_room_for_its_element_rows():
    P = synth.ice_stream_shelf(141, 101, nod=6, seed=2, transient=True)
    mua = ua.CreateMUA(P.coordinates, P.connectivity, ndof=3)
    F = ua.Fields.from_problem(P)
    F.ub, F.vb = 100 * np.sin(P.coordinates[:, 0] / 2e4), 10 * np.cos(P.coordinates[:, 1] / 2e4)
    R0, _ = ua.uvhAssembly(ua.CtrlVar(), mua, F, F.copy(), 0.1, Ronly=True)  # everything but the tangent
    nnz, rows = mua.nnz(), P.connectivity.shape[0] * 36 * 9  # values of the tangent and of its element rows
    with _left(8 * nnz + 4 * rows):  # the first fit, the second do not
        with pytest.raises(L.UaError) as ei:
            ua.uvhAssembly(ua.CtrlVar(), mua, F, F.copy(), 0.1)
        assert ei.value.code == L.UA_ERR_OOM
    R1, K = ua.uvhAssembly(ua.CtrlVar(), mua, F, F.copy(), 0.1)
    assert np.array_equal(R0, R1) and np.isfinite(K.data).all() and K.nnz == nnz


def test_gmres_restart_without_room_for_its_basis():
    P = synth.ice_stream_shelf(141, 101, seed=2, transient=True)
    bcs = ua.BCs.from_problem(P)
    m2, m3 = (ua.CreateMUA(P.coordinates, P.connectivity, ndof=d) for d in (2, 3))
    F0 = ua.uv(ua.CtrlVar().set_force_tolerance(1e-20), m2, bcs, ua.Fields.from_problem(P))[0]

    def step(restart):
        ctrl = ua.CtrlVar(krylov_restart=restart).set_uvh_force_tolerance(1e-20)
        F1, _, info = ua.uvh(ctrl, m3, F0, F0.copy(), bcs, 0.1)
        assert info.converged
        return np.concatenate([F1.ub, F1.vb, F1.h])

    a = step(20)
    with _left(4 << 20):  # the basis of 48 takes 19 MB, the work space of 20 gives back 18
        with pytest.raises(L.UaError) as ei:
            step(48)
        assert ei.value.code == L.UA_ERR_OOM
    assert np.array_equal(a, step(20))
    assert np.linalg.norm(a - step(48)) <= 1e-9 * np.linalg.norm(a)


def test_setup_lists_without_room_are_given_back():
    P = synth.ice_stream_shelf(161, 121, seed=2)
    bcs = ua.BCs.from_problem(P)

    def solve(mua, **kw):
        F, _, _, _, info = ua.uv(ua.CtrlVar(**kw).set_force_tolerance(1e-20), mua, bcs, ua.Fields.from_problem(P))
        return np.concatenate([F.ub, F.vb]), info

    def failure(mua):
        try:
            solve(mua)
        except L.UaError as e:
            return str(e)
        return ""

    solve(ua.CreateMUA(P.coordinates, P.connectivity))  # kernels are loaded
    tried = []
    for left in range(64, 0, -3):  # MB: down to where the lists are what does not fit
        mua = ua.CreateMUA(P.coordinates, P.connectivity)
        solve(mua, krylov_precond=L.UA_PC_JACOBI)
        with _left(left << 20):
            tried.append(failure(mua))
            if "set-up lists" in tried[-1]:
                held = mua.device_bytes()
                for _ in range(3):
                    assert "set-up lists" in failure(mua)
                    assert mua.device_bytes() == held
                break
    else:
        pytest.fail(f"no size at which the lists alone do not fit: {tried}")
    x, info = solve(mua)
    assert info.converged and np.array_equal(x, solve(mua)[0])
