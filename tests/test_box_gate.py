"""BoxGate (box_gate.h) on the host: when a step looks for its boxes."""
import shutil
import subprocess

import pytest

from fall3d_b200 import build as B

HARNESS = r"""
#include "box_gate.h"
#include <cstdio>
using f3d::BoxGate;
static unsigned int pub[f3d::kGateWords];
static void leave(int dirs, unsigned int mx, unsigned int my, unsigned int mz, unsigned int blocks) {
  const unsigned int m[3] = {mx, my, mz};
  for (int d = 0; d < 3; ++d) {
    pub[1 + d] = dirs >> d & 1 ? m[d] : 0;
    pub[4 + d] = dirs >> d & 1 ? m[d] * blocks : 0;
  }
  pub[7] = dirs;
  pub[0] += 1;
}
#define CHECK(x) if (!(x)) { printf("line %d: %s\n", __LINE__, #x); return 1; }
int main() {
  const int n[3] = {400, 300, 60}, tiny[3] = {9, 8, 7};
  const long long blocks = 100, tot[3] = {400 * blocks, 300 * blocks, 60 * blocks}, few[3] = {9, 8, 7};
  BoxGate off, g;
  CHECK(!off.use(7, n, tot));          // nothing attached
  g.attach(pub, true);
  CHECK(!g.use(7, tiny, few));         // too short ever to pay
  CHECK(g.use(7, n, tot) && g.use(7, n, tot));  // no result yet
  leave(7, 40, 40, 40, 20);
  for (int q = 0; q < 100; ++q) CHECK(g.use(7, n, tot));
  leave(7, 400, 300, 60, 100);         // full
  int looks = 0;
  for (int q = 0; q < 160; ++q) looks += g.use(7, n, tot);
  CHECK(looks == 5);
  CHECK(g.use(1, n, tot));             // x alone has its own state
  leave(1, 400, 0, 0, 100);
  CHECK(!g.use(1, n, tot));
  leave(7, 0, 0, 0, 0);                // empty
  CHECK(g.use(7, n, tot) && g.use(7, n, tot) && !g.use(1, n, tot));
  leave(7, 350, 290, 60, 100);         // not enough left out
  CHECK(!g.use(7, n, tot));
  leave(7, 400, 300, 60, 100);
  g.reset();                           // what was left before the reset is not read
  CHECK(g.use(7, n, tot) && g.use(7, n, tot) && g.use(1, n, tot));
  // many blocks: the sum decides
  const long long many[3] = {400 * 50000ll, 300 * 50000ll, 60 * 50000ll};
  leave(7, 400, 300, 60, 50000 / 2);
  CHECK(g.use(7, n, many) && g.use(7, n, many));
  leave(7, 400, 300, 60, 49000);
  CHECK(!g.use(7, n, many));
  return 0;
}
"""


def test_box_gate(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("needs g++")
    src, exe = tmp_path / "gate.cpp", tmp_path / "gate"
    src.write_text(HARNESS)
    subprocess.run([cxx, "-std=c++17", "-Wall", "-Werror", "-I" + B.CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
