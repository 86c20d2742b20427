"""The barriers of the resident solves wait for a bounded time: a team that does not meet ends its kernel with a
flag, which the host turns into UA_ERR_TIMEOUT, and the handle and the context go on.  The debug library has the
same barrier with a short wait; a team of two is launched whole and with one CTA missing."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DEBUG_LIB = os.path.join(ROOT, "uasource_b200", "libuassa_debug.so")

CHILD = r'''
import sys
sys.path.insert(0, sys.argv[1])
import uasource_b200 as ua
from uasource_b200 import lib as L, synth
lib = L.load()
P = synth.ice_stream_shelf(61, 43, seed=3)
m = ua.CreateMUA(P.coordinates, P.connectivity)
for _ in range(2):
    assert lib.ua_debug_team_wait(m.handle, 2) == L.UA_OK
    assert lib.ua_debug_team_wait(m.handle, 1) == L.UA_ERR_TIMEOUT
    assert b"barrier" in lib.ua_last_error()
    assert ua.uv(ua.CtrlVar().set_force_tolerance(1e-20), m, ua.BCs.from_problem(P),
                 ua.Fields.from_problem(P))[4].converged
assert lib.ua_debug_team_wait(m.handle, 3) == L.UA_ERR_INVALID
print("ok")
'''


def test_a_team_that_does_not_meet_is_an_error_and_no_more():
    if not os.path.exists(DEBUG_LIB):
        pytest.fail("libuassa_debug.so is missing: build it with `make -C uasource_b200/csrc debug`")
    env = dict(os.environ, UASOURCE_B200_LIBRARY=DEBUG_LIB)
    r = subprocess.run([sys.executable, "-c", CHILD, ROOT], capture_output=True, text=True, env=env, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout[-2000:] + r.stderr[-4000:]
