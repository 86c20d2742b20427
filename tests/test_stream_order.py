"""The library's streams are non-blocking, so nothing that it puts on the legacy stream is ordered before its
kernels: index lists, counters and fields must reach the device on the handle's own stream (a kernel that
read a list before its copy landed would index with whatever the memory held)."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "uasource_b200", "csrc")
# copies and clears that name no stream
LEGACY = re.compile(r"\bcudaMem(?:cpy|set)(?:2D|3D|ToSymbol|FromSymbol|ToArray|FromArray|Peer)?\s*\(")


def _code(path):
    return re.sub(r"//[^\n]*", "", open(path).read())


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu*")) + glob.glob(os.path.join(CSRC, "*.h"))),
                         ids=os.path.basename)
def test_no_copy_or_clear_on_the_legacy_stream(path):
    code = _code(path)
    assert [m.group(0) for m in LEGACY.finditer(code)] == []
    # every launch names a stream: <<<grid, block, shared, stream>>>
    for m in re.finditer(r"<<<(.*?)>>>", code, re.S):
        depth, commas = 0, 0
        for ch in m.group(1):
            depth += ch in "([{"
            depth -= ch in ")]}"
            commas += ch == "," and depth == 0
        assert commas == 3, m.group(0)
