"""Group sizes of the attention kernels' block order and the choice of grids that start early (csrc/tile_order.h), as a host
program; who passes what to that choice, from the sources."""
import os
import shutil
import subprocess
import tempfile

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROGRAM = r"""
#include <cstdio>
#include "tile_order.h"
// at most `per_sm` blocks an SM; clusters always
static_assert(tlm::starts_early(148, 1, 1, 148) && !tlm::starts_early(149, 1, 1, 148), "");
static_assert(tlm::starts_early(149, 1, 2, 148) && tlm::starts_early(296, 1, 2, 148) && !tlm::starts_early(297, 1, 2, 148), "");
static_assert(tlm::starts_early(148, 2, 1, 148) && tlm::starts_early(1 << 20, 8, 1, 148), "");
int main() {
  for (int n = 1; n <= 300; ++n)
    for (int most = 1; most <= n; ++most) {
      const int g = tlm::even_group(n, most), groups = (n + most - 1) / most;
      if (g < 1 || g > most || (n + g - 1) / g > groups || (g > 1 && (n + g - 2) / (g - 1) <= groups)) { std::printf("%d %d -> %d\n", n, most, g); return 1; }
    }
  std::printf("ok\n");
}
"""


def test_groups_of_heads_are_as_even_as_their_number_allows():
    """No more heads a group than allowed, no more groups than needed, and the smallest size for which that holds."""
    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    d = tempfile.mkdtemp(prefix="tlm_group_")
    src, out = os.path.join(d, "t.cpp"), os.path.join(d, "t")
    with open(src, "w") as f:
        f.write(PROGRAM)
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "train_large_model_from_scratch_b200", "csrc"), "-o", out, src],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([out], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr


def test_small_tile_gemms_start_early_with_two_blocks_per_sm():
    """Their plans take up to two blocks per SM (`slots` in gemm_cost.h); launched as ordinary kernels above one, products of a
    few microseconds lost the launch that is hidden behind the kernel in front."""
    csrc = os.path.join(ROOT, "train_large_model_from_scratch_b200", "csrc")
    def text(name):
        with open(os.path.join(csrc, name)) as f:
            return f.read()
    assert "slots = 2LL * sms" in text("gemm_cost.h")
    assert text("gemm_split.cu").count("launch_overlapped<2>(") == 1 and "launch_overlapped(" not in text("gemm_split.cu")
    assert "starts_early(grid.x, cluster, PER_SM, num_sms())" in text("common.cuh")
