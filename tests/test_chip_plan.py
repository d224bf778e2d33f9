"""The split of cases into clusters of the on-chip engine (csrc/chip_plan.h), on the CPU with a given
device: how many clusters of each size it holds at once."""
import os
import subprocess

import pytest

from conftest import ROOT

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "chip_plan.h"
// arguments: fast, largest cluster size of the device, then nx ny scalars want per case
int main(int argc, char** argv) {
  std::vector<acs::PlanCase> cases;
  for (int q = 3; q + 3 < argc; q += 4) {
    const int nx = atoi(argv[q]), ny = atoi(argv[q + 1]);
    cases.push_back({nx, ny, (nx + 4) / 4 * 4, atoi(argv[q + 2]) != 0, true, atoi(argv[q + 3])});
  }
  const int most = atoi(argv[2]);
  const acs::ChipPlan p = acs::plan_chip(cases, atoi(argv[1]) != 0, [&](int K) { return K > most ? 0 : 148 / K; });
  for (int k : p.k) std::printf("%d ", k);
  std::printf("%.3f\n", p.us);
  for (size_t c = 0; c < cases.size(); ++c)
    if (p.k[c] && (p.k[c] > most || !acs::chip_bytes(cases[c], p.k[c], false))) return 1;
  return 0;
}
"""


@pytest.fixture(scope="module")
def plan(pkg, tmp_path_factory):
    import __graft_entry__ as entry
    where = tmp_path_factory.mktemp("plan")
    src, exe = where / "plan.cu", where / "plan"
    src.write_text(PROGRAM)
    csrc = os.path.join(ROOT, "solver-cfd_b200", "csrc")
    subprocess.run([entry._load_build_module().nvcc(), "-std=c++17", "-I", csrc, "-o", str(exe), str(src)], check=True)

    def run(cases, fast=1, most=16):
        args = [str(v) for c in cases for v in c]
        out = subprocess.run([str(exe), str(fast), str(most)] + args, check=True, capture_output=True, text=True).stdout.split()
        return [int(k) for k in out[:-1]], float(out[-1])
    return run


def test_sizes_that_the_device_cannot_hold_are_left_out(plan):
    """A device (or a share of one) that holds no cluster above 4 CTAs, or none at all: smaller splits are
    taken, and cases that do not fit in them are left to the cluster engine, as are all without any."""
    full = (153, 153, 1, 0)   # fits in 16 CTAs only
    small = (51, 51, 1, 0)    # fits in 4
    assert plan([full])[0] == [16] and plan([full])[1] > 0
    assert plan([full], most=8) == ([0], 0.0)
    k, us = plan([small, full], most=4)
    assert 0 < k[0] <= 4 and k[1] == 0 and us == 0.0
    k, us = plan([small, small], most=4)
    assert all(0 < x <= 4 for x in k) and us > 0
    for most in range(1, 17):
        plan([small, full, (30, 22, 0, 0), (40, 9, 1, 0)], most=most)
    assert plan([small, (30, 22, 0, 0)], most=0) == ([0, 0], 0.0)
    assert plan([(51, 51, 1, 9)], most=8)[0] == [8]


def test_a_caller_s_split_does_not_move_a_case_off_the_chip(plan):
    """The size asked for where the case fits in it, else the next larger one that it fits in."""
    assert [plan([(51, 51, 1, K)])[0][0] for K in (4, 9, 12)] == [4, 9, 12]
    least = next(K for K in range(1, 17) if plan([(102, 102, 1, K)])[0] == [K])
    assert least > 4
    for K in range(1, 17):
        assert plan([(102, 102, 1, K)])[0] == [max(K, least)]
        assert plan([(153, 153, 1, K)])[0] == [16]
        assert plan([(300, 300, 1, K)])[0] == [0]          # too large for any cluster
    k, us = plan([(51, 51, 1, 4), (51, 51, 1, 0)])
    assert k[0] == 4 and k[1] > 0 and us > 0
