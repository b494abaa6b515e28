"""host_parallel (csrc/tree.h) when memory runs out: every share of the work is done or
an exception is passed on with all threads joined; the program never aborts."""
import os
import subprocess

import cabi

CSRC = os.path.join(cabi.LIB_PATH.rsplit(os.sep, 1)[0], "csrc")
MAIN = r"""
#include <cstdio>
#include <cstdlib>
#include <new>
#include "tree.h"
static thread_local long left = -1;  // allocations of this thread until one fails
void* operator new(std::size_t n) {
  if (left >= 0 && left-- == 0) throw std::bad_alloc();
  if (void* p = std::malloc(n)) return p;
  throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }
int main() {
  for (int fail = 0; fail < 40; ++fail) {
    long done[8] = {};
    bool threw = false;
    left = fail;
    try {
      cg::host_parallel(8, 80, [&](int t, long b, long e) { done[t] += e - b; });
    } catch (const std::bad_alloc&) {
      threw = true;
    }
    left = -1;
    long sum = 0;
    for (long d : done) sum += d;
    if (!threw && sum != 80) return 1;
  }
  // an exception of one share
  try {
    cg::host_parallel(8, 80, [&](int t, long, long) { if (t == 5) throw 5; });
    return 2;
  } catch (int) {
  }
  std::puts("ok");
}
"""


def test_out_of_memory(tmp_path):
    (tmp_path / "main.cc").write_text(MAIN)
    exe = str(tmp_path / "main")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, "-o", exe,
                    str(tmp_path / "main.cc")], check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stderr
