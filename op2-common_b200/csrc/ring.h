// The stages of a ring of shared memory that several warps fill in turn (warp w
// of `turns` the stages w, w + turns, ...) and that are used in order, stage n
// in slot n % ring after stage n - ring has been used.  Plain C++.  Internal.
#pragma once

#ifdef __CUDACC__
#define OP2B_HD __host__ __device__
#else
#define OP2B_HD
#endif

namespace op2b {

// What a kernel that gives up has to wait for before it leaves: the newest stage
// that may still be on its way into `slot`, or -1.  last[w]: the last stage that
// warp w began to load (below 0: none).  Of warp w, the stages up to last[w] -
// ring have been used; of a slot, the newest stage is the one whose phase its
// barrier is in.
OP2B_HD constexpr int newest_in_flight(int slot, int ring, const int *last, int turns) {
  int newest = -1;
#pragma unroll 1
  for (int w = 0; w < turns; w++)
#pragma unroll 1
    for (int m = last[w]; m >= 0 && m > last[w] - ring; m -= turns)
      if (m % ring == slot && m > newest) newest = m;
  return newest;
}

}  // namespace op2b
