"""The rule of the device workspace (csrc/workspace.h) against a fake allocator:
compiled with the host compiler, no device."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "ht_tensor_learning_using_gpu_tensor_cores_gb300", "csrc")

PROGRAM = r"""
#include <cassert>
#include <cstdio>
#include <cstdlib>
#include <map>
#include "workspace.h"
using namespace htgb;

struct Fake {
  size_t total, used = 0, others = 0;   // device memory; held here; held by other users
  size_t hole = ~size_t(0);             // the largest allocation that succeeds
  int allocations = 0, failures = 0, releases = 0, asked = 0;
  bool take_freed = false;              // another user takes whatever is freed
  std::map<void *, size_t> live;
  explicit Fake(size_t t) : total(t) {}
  bool room(size_t *b) { ++asked; *b = total - used - others; return true; }
  bool allocate(void **p, size_t n) {
    if (n > total - used - others || n > hole) { ++failures; return false; }
    *p = std::malloc(1);
    live[*p] = n;
    used += n;
    ++allocations;
    return true;
  }
  bool release(void *p) {
    assert(live.count(p));
    used -= live[p];
    if (take_freed) others += live[p];
    live.erase(p);
    std::free(p);
    ++releases;
    return true;
  }
};

static Granted call(WorkspaceBlock &w, Fake &m, size_t want, size_t least, bool optional = true) {
  const Granted g = grant_workspace(w, want, least, optional, m);
  if (g != Granted::none) {
    assert(w.ptr && m.live.count(w.ptr) && m.live[w.ptr] == w.bytes);
    assert(w.bytes >= (g == Granted::want ? want : least));
  }
  assert(m.live.size() == (w.ptr ? 1u : 0u));   // nothing leaks
  return g;
}

int main() {
  {   // room for everything: one block, then no call of the allocator at all
    Fake m(1000); WorkspaceBlock w;
    assert(call(w, m, 300, 100) == Granted::want && w.bytes == 300);
    const int asked = m.asked;
    for (int i = 0; i < 5; ++i) assert(call(w, m, 300, 100) == Granted::want && call(w, m, 50, 50) == Granted::want);
    assert(m.allocations == 1 && m.releases == 0 && m.asked == asked);
    assert(call(w, m, 600, 200) == Granted::want && w.bytes == 600 && m.releases == 1);
  }
  {   // no room for the planes: the small block is made once and stays, call after call
    Fake m(1000); WorkspaceBlock w;
    m.others = 700;
    for (int i = 0; i < 5; ++i) assert(call(w, m, 500, 100) == Granted::least && w.bytes == 100);
    assert(m.allocations == 1 && m.releases == 0 && m.failures == 0);
    m.others = 0;   // and when there is room, the planes come back
    assert(call(w, m, 500, 100) == Granted::want && w.bytes == 500);
  }
  {   // a block that was enough at least is not given up, whoever waits for the memory
    Fake m(1000); WorkspaceBlock w;
    m.others = 500;
    assert(call(w, m, 150, 150) == Granted::want);
    m.take_freed = true;
    for (int i = 0; i < 3; ++i) assert(call(w, m, 600, 150) == Granted::least && w.bytes == 150);
    assert(m.releases == 0 && m.failures == 0);
  }
  {   // only both together make the room
    Fake m(1000); WorkspaceBlock w;
    assert(call(w, m, 600, 600) == Granted::want);
    assert(call(w, m, 900, 650) == Granted::want && w.bytes == 900 && m.releases == 1);
  }
  {   // room that is none (no allocation that large succeeds): tried once, and again only with more room
    Fake m(1000); WorkspaceBlock w;
    m.others = 200; m.hole = 300;
    for (int i = 0; i < 4; ++i) assert(call(w, m, 400, 100) == Granted::least && w.bytes == 100);
    assert(m.failures == 1 && m.allocations == 1 && m.releases == 0);
    m.others = 100;
    assert(call(w, m, 400, 100) == Granted::least && m.failures == 2);
    m.others = 0; m.hole = ~size_t(0);
    assert(call(w, m, 400, 100) == Granted::want);
  }
  {   // inside a capture nothing is allocated that the call can do without
    Fake m(1000); WorkspaceBlock w;
    assert(call(w, m, 200, 200) == Granted::want);
    assert(call(w, m, 500, 200, false) == Granted::least && m.allocations == 1 && m.releases == 0);
    assert(call(w, m, 500, 200) == Granted::want);
  }
  {   // and what does not fit at all is refused, now and later
    Fake m(100); WorkspaceBlock w;
    assert(call(w, m, 500, 200) == Granted::none && !w.ptr && w.bytes == 0);
    assert(call(w, m, 80, 80) == Granted::want);
    assert(call(w, m, 500, 200) == Granted::none);
  }
  std::puts("ok");
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_grant_workspace(tmp_path):
    src = tmp_path / "workspace.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "workspace"
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout == "ok\n"
