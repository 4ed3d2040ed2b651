"""The growing device list (far cells of the strip drift) when an allocation
fails: the list then holds nothing, so that the next call allocates again
instead of writing past a shorter list."""

import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include <cstdio>
#include <cstdlib>
#include <map>
#include "vls_devlist.h"
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)
int main() {
  std::map<int *, size_t> live;  // what is allocated, and its length
  bool fail = false;
  auto alloc = [&](int **q, size_t n) {
    if (fail) return 7;
    *q = (int *)std::malloc(n * sizeof(int));
    live[*q] = n;
    return 0;
  };
  auto release = [&](int *q, size_t n) {
    if (live.at(q) != n) return 9;
    live.erase(q);
    std::free(q);
    return 0;
  };
  vls::DeviceList<int> l;
  CHECK(l.reserve(4, alloc, release) == 0 && l.p && l.cap == 4);
  int *const first = l.p;
  CHECK(l.reserve(3, alloc, release) == 0 && l.p == first && l.cap == 4);
  fail = true;
  CHECK(l.reserve(9, alloc, release) == 7);
  CHECK(l.p == nullptr && l.cap == 0 && live.empty());
  CHECK(l.reserve(9, alloc, release) == 7 && l.p == nullptr && l.cap == 0);
  fail = false;
  CHECK(l.reserve(2, alloc, release) == 0 && l.p && live.at(l.p) == 2 && l.cap == 2);
  // rising lengths keep one list only
  for (size_t n = 3; n < 50; ++n) CHECK(l.reserve(n, alloc, release) == 0 && live.size() == 1);
  CHECK(live.at(l.p) == l.cap && l.cap == 49);
  return 0;
}
"""


def test_failed_growth_leaves_no_capacity(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    src = tmp_path / "t.cpp"
    src.write_text(SRC)
    exe = str(tmp_path / "t")
    subprocess.check_call(["g++", "-std=c++17", "-Wall", "-Werror",
                           "-I" + os.path.join(REPO, "vlasolve_b200", "csrc"), str(src), "-o", exe])
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
