// Which form assembles A's rows: in shared memory (a warp of 32 rows a CTA, 33
// entries of 76 bytes a block of the longest row) or in global memory.  Host
// arithmetic alone, so that a CPU test can run it.
#pragma once
#include <algorithm>

namespace mprgp {

constexpr int kRowPad = 33;
constexpr int kRowSmemMax = 220 * 1024;  // rows of up to 89 blocks
constexpr int row_smem(int max_len) { return kRowPad * max_len * (9 * 8 + 4); }

// The sums in shared memory need four warps an SM, or all that the mesh has
// for it, to keep the FP64 units busy; one long row costs every CTA its room.
// 348,480 vertices, whole call, by the longest row that shared memory is sized
// for (global memory: 4.84 ms): 15 blocks, six CTAs an SM 3.38, 22 and four 4.14,
// 24 and three 5.40, 32 and two 7.83, 56 and one 15.3.  17,856 vertices, four
// warps an SM (0.38): 22 blocks 0.27, 24 0.47.  1,700, one warp an SM (0.32):
// 0.24 up to 80 blocks.  A tetrahedral grid has 15 blocks a row, an irregular
// mesh 16 on average and 30 to 50 at most (85,184 vertices, 52 blocks: 2.8 ms in
// global memory, 7.2 in shared).
inline bool rows_in_smem(int max_len, int nv, int nsm, int sm_smem) {
  if (max_len > kRowSmemMax / row_smem(1)) return false;
  const int resident = sm_smem / (row_smem(max_len) + 1024);  // (1 KB a CTA is the system's)
  const int warps = ((nv + 31) / 32 + nsm - 1) / nsm;
  return resident >= std::min(4, warps);
}

}  // namespace mprgp
