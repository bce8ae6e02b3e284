"""The per-device buffers of the convolution entry points (csrc/xtg_per_device.h),
compiled for the host with a counting stand-in for the CUDA runtime: a buffer of
one device is never handed out on another, grows in place of a smaller one, and a
failed allocation leaves nothing behind."""
import os
import subprocess

import common

CSRC = os.path.join(common.ROOT, "timbir-python_b200", "csrc")
PROGRAM = r"""
#include <cassert>
#include <cstdlib>
#include <set>
#include "xtg_per_device.h"
static int cur, fail_next;
static std::set<void *> live;
struct Fake {
  typedef int Error;
  static constexpr int ok = 0;
  static int device(int *d) { if (cur < 0) return 7; *d = cur; return 0; }
  static int allocate(void **p, size_t n) { if (fail_next) return 2; *p = malloc(n); live.insert(*p); return 0; }
  static void release(void *p) { assert(live.erase(p) == 1); free(p); }
};
int main() {
  xtg::PerDevice<Fake> b;
  void *p0 = nullptr, *p1 = nullptr, *q = nullptr;
  bool fresh = false;
  assert(b.get(100, &p0, &fresh) == 0 && p0 && fresh);
  cur = 1;
  assert(b.get(50, &p1, &fresh) == 0 && p1 && p1 != p0 && fresh && live.size() == 2);
  cur = 0;
  assert(b.get(80, &q, &fresh) == 0 && q == p0 && !fresh);
  assert(b.get(200, &q, &fresh) == 0 && fresh && live.size() == 2 && live.count(p1));
  cur = 1;
  void *r = nullptr;
  assert(b.get(50, &r, &fresh) == 0 && r == p1 && !fresh);
  fail_next = 1;
  r = nullptr;
  assert(b.get(500, &r) == 2 && r == nullptr && live.size() == 1);
  fail_next = 0;
  assert(b.get(10, &r, &fresh) == 0 && fresh && live.size() == 2);
  cur = -1;
  assert(b.get(10, &r) == 7);
  return 0;
}
"""


def test_buffers_per_device(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    subprocess.run([str(exe)], check=True)
