"""The bounds-checked build checks what the default solves gather through: a clean flag counts only where the
checks were reached.  The sites: 2 element nodes, 3 contributions, 6 node-slice columns of a launched solve
(a tied pair of nodes), 7 those of the resident solves, 8 coarse operators and transfers, 9 the uvh tangent,
10 the elements of the quadratic gathers.  Each case runs in a child process that loads the debug library."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DEBUG_LIB = os.path.join(ROOT, "uasource_b200", "libuassa_debug.so")

CHILD = r'''
import ctypes as C, json, sys
import numpy as np
sys.path.insert(0, sys.argv[1])
import uasource_b200 as ua
from uasource_b200 import lib as L, synth
out = {}

def seen(mua):
    lib, en, site, idx, sites = L.load(), C.c_int32(), C.c_int32(), C.c_int64(), C.c_uint64()
    L.check(lib.ua_debug_bounds(mua.handle, C.byref(en), C.byref(site), C.byref(idx)))
    L.check(lib.ua_debug_sites(mua.handle, C.byref(en), C.byref(sites)))
    return en.value, site.value, idx.value, [s for s in range(64) if sites.value >> s & 1]

# staged and streamed rows (the second mesh of each kind does not fit the shared memory of its CTAs), solo
# levels and one CTA
for nod, nx, ny in ((3, 21, 11), (3, 141, 71), (6, 13, 7), (6, 101, 51)):
    P = synth.ice_stream_shelf(nx, ny, nod=nod, seed=1, transient=True)
    b = ua.BCs.from_problem(P)
    for prec, bf16 in ((L.UA_PREC_FP64, 1), (L.UA_PREC_MIXED, 1), (L.UA_PREC_MIXED, 0)):
        m = ua.CreateMUA(P.coordinates, P.connectivity)
        ctrl = ua.CtrlVar(precision=prec, krylov_rtol=1e-6 if prec else 1e-12, precond_bf16=bf16)
        Fo = ua.uv(ctrl.set_force_tolerance(1e-20), m, b, ua.Fields.from_problem(P))[0]
        out[f"uv {nod} {nx} {prec} {bf16}"] = seen(m)
    m3 = ua.CreateMUA(P.coordinates, P.connectivity, ndof=3)
    ua.uvh(ua.CtrlVar().set_uvh_force_tolerance(1e-20), m3, Fo, Fo.copy(), b, 0.1)
    out[f"uvh {nod} {nx}"] = seen(m3)
P = synth.ice_stream_shelf(21, 11, seed=0)
b = ua.BCs.from_problem(P)
x, y = P.coordinates[:, 0], P.coordinates[:, 1]
lo, hi = (np.flatnonzero((y == e) & (x > x.min()) & (x < x.max())) for e in (y.min(), y.max()))
b.ubTiedNodeA, b.ubTiedNodeB = lo.astype(np.int32), hi.astype(np.int32)
m = ua.CreateMUA(P.coordinates, P.connectivity)
ua.uv(ua.CtrlVar().set_force_tolerance(1e-20), m, b, ua.Fields.from_problem(P))
out["tied"] = seen(m)
print(json.dumps(out))
'''


def test_the_default_solves_are_checked_and_clean():
    if not os.path.exists(DEBUG_LIB):
        pytest.fail("libuassa_debug.so is missing: build it with `make -C uasource_b200/csrc debug`")
    env = dict(os.environ, UASOURCE_B200_LIBRARY=DEBUG_LIB)
    r = subprocess.run([sys.executable, "-c", CHILD, ROOT], capture_output=True, text=True, env=env, timeout=900)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
    for case, (enabled, site, index, sites) in json.loads(r.stdout.strip().splitlines()[-1]).items():
        assert enabled == 1, case
        assert site == 0, f"{case}: bounds violation at site {site}, index {index}"
        want = {2, 3} | ({6} if case == "tied" else {7, 8})
        want |= ({9} if case.startswith("uvh") else set()) | ({10} if case.split()[1:2] == ["6"] else set())
        assert want <= set(sites), f"{case}: checked {sites}"
