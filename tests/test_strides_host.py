"""Sizes that the one-launch traversals accept (strides_fit, csrc/rg_host.h), on the CPU:
a 32-bit loop over ids that steps by every thread of a launch ends at the largest
size accepted, and would not at the largest size a graph may have."""

import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include <stdint.h>
#include "rg_host.h"
// Does `for (uint32_t i = first; i < n; i += step)` end?  (Its last index is below n,
// so the step after it is what may wrap.)
static bool ends(uint32_t n, uint32_t step) { return (uint64_t)(n - 1) + step <= 0xFFFFFFFFull; }
int main() {
  const uint32_t threads = 152 * 1024;  // a CTA of 1024 threads per SM
  const int64_t most = rg::kMostStrided, largest = 0xFFFFFFFEll;  // the builders' limit
  if (!rg::strides_fit(most, most) || !ends((uint32_t)most, threads)) return 1;
  // groups of 128 edges, four a lane, past the last edge
  if (!ends((uint32_t)most, 4 * threads)) return 2;
  if (rg::strides_fit(most + 1, 0) || rg::strides_fit(1, most + 1)) return 3;
  if (rg::strides_fit(largest, 0) || ends((uint32_t)largest, threads)) return 4;
  return 0;
}
"""


def test_loops_end_at_the_largest_sizes(tmp_path):
    (tmp_path / "t.cc").write_text(SRC)
    exe = tmp_path / "t"
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "radar-graph_gb300", "csrc"), str(tmp_path / "t.cc"),
                    "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0
