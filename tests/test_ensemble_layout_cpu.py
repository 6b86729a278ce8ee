"""The shared memory that the persistent ensemble step's blocks count on, for every
wave-vector cube and every number of columns it can keep: within the block's
allocation, whole rounds of the warps where the columns come in parts."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "md-lab_gb300", "csrc")

PROBE = r"""
#include <cstdio>
#include "xmd_ens_layout.h"
using namespace xk;
int main() {
  std::printf("%zu %d %d\n", ENS_SMEM, ENS_NSMAX, ENS_W);
  for (int ns = 1; ns <= ENS_NSMAX; ++ns)
    for (int ncol = 0; ncol <= ns * (2 * ns + 1) + ns + 1; ++ncol)
      std::printf("%d %d %d %zu\n", ns, ncol, ens_recip_columns(ns, ncol), ens_recip_bytes(ns, ncol));
}
"""


def test_reciprocal_forces_fit(tmp_path):
    src, exe = tmp_path / "probe.cpp", tmp_path / "probe"
    src.write_text(PROBE)
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    lines = [list(map(int, line.split())) for line in
             subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.splitlines()]
    (smem, nsmax, warps), rows = lines[0], lines[1:]
    assert (smem, nsmax, warps) == (65536, 11, 8)
    parts = 0
    for ns, ncol, cap, nbytes in rows:
        # a float4 per harmonic 0..ns and a 32-byte record a column; two rows of ns + 1 and the sums' 8 x 3 rows of 32 float2
        assert nbytes == cap * (16 * (ns + 1) + 32) + 32 * 8 * (2 * (ns + 1) + 24)
        assert nbytes <= smem
        if cap < ncol:
            parts += 1
            assert cap >= warps and cap % warps == 0
            assert nbytes + (ncol - cap) * (16 * (ns + 1) + 32) > smem, "all columns would fit"
        else:
            assert cap == ncol
    assert parts == 265 - 237  # n_sum = 11 alone
