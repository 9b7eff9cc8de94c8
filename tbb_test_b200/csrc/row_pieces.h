// Stores of result rows in 32-byte groups (step_kernel.cu).
#pragma once

#ifdef __CUDACC__
#define B2_HD __host__ __device__
#else
#define B2_HD
#endif

namespace b2 {

// How many of the two 16-byte pieces of a group lie in the matrix: `left` elements from the group's first to the row's
// end, `per` elements in a piece (a piece that the row ends in counts: rows are padded to whole pieces).
B2_HD inline int pieces_of_32(int left, int per) {
  const int n = (left + per - 1) / per;
  return n < 0 ? 0 : n > 2 ? 2 : n;
}

}  // namespace b2
