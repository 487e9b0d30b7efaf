// Limits and arithmetic of the row runs (rowrun.cu) that host code can compile
// and test as well.
#pragma once

#ifdef __CUDACC__
#define NSPB_HD __host__ __device__ __forceinline__
#else
#define NSPB_HD inline
#endif

namespace nspb {

constexpr int kRunMaxA = 128;   // A entries of a row in a run
constexpr int kRunMaxIp = 1536; // products of a row in a run

// A B row's length as the sums over a row's A entries take it: any that is too
// long for a run by itself counts as just too long, so that the sum over
// kRunMaxA entries stays far below 2^31 (a row of A may repeat a column, and 32
// B rows of 2^27 entries add up to zero in 32 bits).
NSPB_HD int run_len(int len) { return len < kRunMaxIp + 1 ? len : kRunMaxIp + 1; }

// Whether rows whose B rows lie `step` entries apart may share a tile of `rows`
// rows. Longer distances fit neither the 110 KB of a tile (32768 values of 4
// bytes are 128 KB) nor the 15 bits of a program word, and products of distance
// and rows past 2^31 made tiles that seemed to fit: B rows of one pattern may
// have rows of any length between them (lags 2 and 3).
constexpr int kRunMaxStep = 1 << 15;
NSPB_HD bool run_step_fits(int step, int rows) { return rows == 1 || step < kRunMaxStep; }

// Whether a block of k_num_run stops because a wait has run out. A look-up warp
// or a lane may find that out at any moment, and a warp that stopped alone
// would leave the others at their next barrier for good: the views of the flag
// become one answer at a barrier, `any`, and all act on it.
template <typename Lost, typename Any>
NSPB_HD bool run_gives_up(Lost &&lost, Any &&any) {
  return any(lost());
}

}  // namespace nspb
