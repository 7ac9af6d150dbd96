"""Host loops over all cores (parallel_for): an exception in one of the threads, such as a host
allocation that fails while a tree is packed or a plan is built, reaches the caller, whose C entry
point turns it into a status.  CPU only."""
import importlib
import os
import subprocess

PROGRAM = r"""
#include <cstdio>
#include <new>
#include <stdexcept>
#include "nrt_internal.h"
int main() {
  // a worker, the calling thread, several at once, and none
  std::atomic<int64_t> seen(0);
  nrt::parallel_for(5000, [&](int64_t) { seen++; });
  if (seen != 5000) return 1;
  for (int64_t at : {0, 4999, 2500}) {
    try {
      nrt::parallel_for(5000, [&](int64_t i) {
        if (i == at || (at == 2500 && i > 2500)) throw std::bad_alloc();
      });
      return 2;
    } catch (const std::bad_alloc &) {
    }
  }
  try {
    nrt::parallel_ranges((int64_t)5 << 20, [&](int64_t a, int64_t) {
      if (a > 0) throw std::runtime_error("range");
    });
    return 3;
  } catch (const std::runtime_error &) {
  }
  puts("caught");
  return 0;
}
"""


def test_exceptions_reach_the_caller(tmp_path):
    build = importlib.import_module("168861_gb300.build")
    src, exe = tmp_path / "pf.cu", tmp_path / "pf"
    src.write_text(PROGRAM)
    subprocess.run([build.nvcc(), "-std=c++17", "-O1", "-I", build.CSRC, "-I",
                    os.path.join(build.ROOT, "include"), *build.ARCH, str(src), "-o", str(exe),
                    "-Xcompiler", "-pthread"], check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout == "caught\n", (r.returncode, r.stderr)
