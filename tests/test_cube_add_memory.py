"""The host pass that adds an inserted cube when memory runs out: mg_cube_add
compiled alone with an allocator that fails at each of its allocations in turn
(the row sums, the pool, every thread's start).  It must return, with the whole
cube added if it reports success and with the array untouched if not, and never
end the process (CPU only)."""

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HARNESS = r"""
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <new>
#include <string>
#include <vector>
#include "martini_gb300.h"
namespace mg { void set_last_error(const std::string&) {} }
static std::atomic<int> left{-1};  // allocations until one fails; negative: none does
void* operator new(std::size_t n) {
  if (left.load() >= 0 && left.fetch_sub(1) == 0) throw std::bad_alloc();
  if (void* p = std::malloc(n ? n : 1)) return p;
  throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }
int main() {
  const long nx = 64, ny = 64, nc = 256, n = nx * ny * nc;  // enough for every thread
  std::vector<float> add(n, 0.5f);
  std::vector<double> a(n), sums(nc);
  int failures = 0;
  for (int k = 0; k < 40; ++k) {
    for (double& v : a) v = 1.0;
    left = k;
    const int rc = mg_cube_add(a.data(), add.data(), nx, ny, nc, 0, 0, 2.0, 1, sums.data());
    const bool hit = left.exchange(-1) < 0;
    const double want = rc == MG_OK ? 0.75 : 1.0;
    for (double v : a) if (v != want) return 2;
    if (rc != MG_OK && rc != MG_ERR_WORKSPACE) return 3;
    if (rc == MG_OK && sums[7] != 1.5 * nx * ny) return 4;
    if (rc != MG_OK) ++failures;
    if (!hit && k > 0) break;
  }
  std::printf("%d\n", failures);
  return failures > 0 ? 0 : 5;
}
"""


def test_failing_allocations_never_end_the_process(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    (tmp_path / "harness.cpp").write_text(HARNESS)
    exe = tmp_path / "harness"
    subprocess.run([cxx, "-O1", "-std=c++17", "-pthread", "-I", os.path.join(ROOT, "include"),
                    "-x", "c++", os.path.join(ROOT, "martini_gb300", "csrc", "mg_host.cu"),
                    str(tmp_path / "harness.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], timeout=120, capture_output=True, text=True)
    assert r.returncode == 0, (r.returncode, r.stderr)
