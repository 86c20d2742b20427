"""Buffers that belong together are allocated together (csrc/ua_alloc.h): a failure between two of them leaves
none, and a later call for the old size does not take what is left for its own.  The GMRES work space of the
uvh step relies on it: with the basis there and the partials missing its kernel would write through null."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "uasource_b200", "csrc")

PROGRAM = r'''
#include <cassert>
#include <cstdio>
#include <cstdlib>
#include <set>
#include "ua_alloc.h"
int main() {
  std::set<void*> live;
  int left = 0;  // allocations that still succeed
  auto alloc = [&](size_t n) -> void* {
    if (left-- <= 0) return nullptr;
    void* p = std::malloc(n);
    live.insert(p);
    return p;
  };
  auto release = [&](void* p) { assert(live.erase(p) == 1); std::free(p); };
  for (int ok = 0; ok <= 4; ++ok) {  // the second size fails after ok buffers
    void* b[4] = {};
    int have = 0;
    auto get = [&](int key) {
      return ua::alloc_for(have, key, {{&b[0], 8u * key}, {&b[1], 16u * key}, {&b[2], 24}, {&b[3], 32}}, alloc, release);
    };
    left = 4;
    assert(get(30) && have == 30 && live.size() == 4);
    assert(get(30) && left == 0);  // nothing to do
    left = ok;
    const bool got = get(48);
    assert(got == (ok == 4) && have == (got ? 48 : 0) && live.size() == (got ? 4u : 0u));
    for (void* p : b) assert((p != nullptr) == got);
    left = 4;
    assert(get(30) && have == 30 && live.size() == 4);
    for (void* p : b) { assert(p && live.count(p)); release(p); }
  }
  assert(live.empty());
  std::puts("ok");
}
'''


def test_all_or_none(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no g++")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-Wall", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout == "ok\n"


def test_the_gmres_work_space_is_allocated_together():
    src = open(os.path.join(CSRC, "ua_gmres.cu")).read()
    assert "dev_alloc(m, sizeof" not in src  # no buffer of its own beside alloc_for
    assert "alloc_for(C.gm_mr" in src
