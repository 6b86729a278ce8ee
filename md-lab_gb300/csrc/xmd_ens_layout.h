// xmd_ens_layout.h -- the dynamic shared memory of a block of the persistent
// ensemble step, in plain C++ (the kernel, the host's checks and a test without a
// GPU count the same bytes).
#pragma once

#include <cstddef>

namespace xk {

constexpr size_t ENS_SMEM = 64 * 1024;  // per block: two or three blocks an SM
constexpr int ENS_NSMAX = 11;           // largest Ewald n_sum
constexpr int ENS_W = 8;                // warps per block

// Reciprocal forces of 32 particles: force tables (a float4 per harmonic 0..ns)
// and a 32-byte record per staged column, x and y phase factors of the
// particles, the warps' sums
constexpr size_t ens_recip_column(int ns) { return 16 * (size_t)(ns + 1) + 32; }
constexpr size_t ens_recip_rest(int ns) { return 8 * (size_t)(2 * (ns + 1) * 32) + 8 * (size_t)(ENS_W * 3 * 32); }
// Columns staged at a time: all of them where they fit (always up to n_sum = 10;
// at 11 up to 237, in a cubic box those of alpha L below about 6.7), else as many
// whole rounds of the warps as fit, so that each warp keeps its columns and
// their order.
constexpr int ens_recip_columns(int ns, int ncol) {
  const size_t room = (ENS_SMEM - ens_recip_rest(ns)) / ens_recip_column(ns);
  return (size_t)ncol <= room ? ncol : (int)(room / ENS_W * ENS_W);
}
constexpr size_t ens_recip_bytes(int ns, int ncol) {
  return ens_recip_rest(ns) + ens_recip_column(ns) * (size_t)ens_recip_columns(ns, ncol);
}

// the recursions' block solve (mantissas and exponents; rows of `chunk`)
constexpr size_t ens_solve_bytes(int N, int chunk) { return 12 * ((size_t)N + 1 + 2 * chunk + 2 * (size_t)chunk * (chunk + 1)); }

}  // namespace xk
