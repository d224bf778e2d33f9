"""A launch of the tile engine that fails says so, so that a loop body without it is never run.  Here it
fails on the host: without a device any launch does, with one an empty grid does."""
import os
import subprocess

from conftest import ROOT

PROGRAM = r"""
#include <cstdio>
#include "tile_engine.h"
int main() {
  int bad = 0;
  for (int overlap = 0; overlap < 2; ++overlap) {
    for (int stage = 1; stage <= 3; ++stage)
      bad += acs::te_launch_uv(stage, nullptr, nullptr, nullptr, 0, nullptr, nullptr, overlap != 0, nullptr) != cudaSuccess;
    bad += acs::te_launch_ptc(nullptr, nullptr, nullptr, 0, nullptr, nullptr, overlap != 0, nullptr) != cudaSuccess;
  }
  std::printf("%d\n", bad);
  return bad == 8 ? 0 : 1;
}
"""


def test_tile_launches_report_errors(pkg, tmp_path):
    import __graft_entry__ as entry
    (tmp_path / "launch.cu").write_text(PROGRAM)
    pkg_dir = os.path.join(ROOT, "solver-cfd_b200")
    lib = os.path.join(pkg_dir, "libacs_b200.so")
    exe = str(tmp_path / "launch")
    subprocess.run([entry._load_build_module().nvcc(), "-std=c++17", "-I", os.path.join(pkg_dir, "csrc"), "-o", exe,
                    str(tmp_path / "launch.cu"), lib, "-Xlinker", "-rpath=" + pkg_dir], check=True)
    assert subprocess.run([exe], capture_output=True, text=True).stdout.strip() == "8"
