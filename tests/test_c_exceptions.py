"""No C++ exception crosses the C boundary: sns_fft3d_create with the k-th host allocation failing,
for every k, returns an error code.  The call is one that is refused (an axis too long) after
all three axes were planned, so it needs no device."""
import os
import subprocess

PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "spectral_solver_b200")

SOURCE = r"""
#include "sns_b200.h"
#include <cstdio>
#include <cstdlib>
#include <new>
static long countdown = -1;
void* operator new(std::size_t n) {
  if (countdown >= 0 && countdown-- == 0) throw std::bad_alloc();
  void* p = std::malloc(n ? n : 1);
  if (!p) throw std::bad_alloc();
  return p;
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }
int main() {
  for (long k = 0; k < 100000; ++k) {
    sns_fft3d* h = nullptr;
    int rc = -1;
    countdown = k;
    try {
      rc = sns_fft3d_create(48, 60, 7000, 1.0, 1.0, 1.0, &h);
    } catch (...) {
      std::printf("escaped at allocation %ld\n", k);
      return 1;
    }
    const bool failed = countdown < 0;
    countdown = -1;
    if (h != nullptr || (rc != SNS_ERR_UNSUPPORTED && !(failed && rc == SNS_ERR_NOMEM))) {
      std::printf("code %d at allocation %ld\n", rc, k);
      return 1;
    }
    if (!failed) {
      std::printf("%ld allocations\n", k);
      return 0;
    }
  }
  return 1;
}
"""


def test_failed_allocations_become_error_codes(tmp_path):
    src, exe = tmp_path / "alloc.cpp", tmp_path / "alloc"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", os.path.join(PKG, "..", "include"), str(src), "-o", str(exe),
                    "-L", PKG, "-lsns_b200", f"-Wl,-rpath,{PKG}"], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
    assert int(r.stdout.split()[0]) > 3  # the planner's vectors were among them
