// Single-pass prefix sums over the tiles of one launch (chained scan): each
// tile publishes its own sum, adds up its predecessors' until it meets a
// running total, and publishes its own.  Tiles are numbered by a ticket taken
// at the start of the block, so every predecessor has already started; the
// waits are bounded all the same.  One that gives up raises kErrScanTimeout and
// goes on within its arrays; what the launch wrote is then not complete, and
// every later kernel that takes an index from it returns at its start.  (The
// bit is raised by chained scans alone, so it stands still in those kernels.)
#pragma once
#include "device_common.cuh"

namespace mc {

constexpr unsigned long long kTileSum = 1ull << 62;    // the tile's own sum
constexpr unsigned long long kTileTotal = 2ull << 62;  // the sum up to and with the tile
constexpr unsigned long long kTileValue = kTileSum - 1;

// Polls a wait of a chained scan may take: 2^22, or MERCURY_WAIT_POLLS (tests
// run the waits out with 0).
int wait_polls();

// Sum of the tiles before `tile`, on every lane of the calling warp; status:
// one word per tile, zero before the launch; max_polls: wait_polls().
__device__ __forceinline__ unsigned long long tile_prefix(volatile unsigned long long *status,
                                                          int64_t tile, unsigned long long sum,
                                                          int lane, int max_polls, unsigned *err,
                                                          bool *gave_up) {
  if (lane == 0) status[tile] = (tile == 0 ? kTileTotal : kTileSum) | sum;
  unsigned long long prefix = 0;
  for (int64_t t = tile - 1; t >= 0; t -= kWarp) {
    const int64_t at = t - lane;
    unsigned long long s = 0;
    bool ready = false;
    for (int polls = 0; polls < max_polls && !ready; ++polls) {
      s = kTileTotal;
      if (at >= 0) s = status[at];
      // Nothing beyond the nearest running total matters.
      const unsigned done = __ballot_sync(kFull, (s & ~kTileValue) != 0);
      const unsigned total = __ballot_sync(kFull, (s & ~kTileValue) == kTileTotal);
      const unsigned needed = total ? kFull >> (kWarp - __ffs(total)) : kFull;
      ready = (done & needed) == needed;
    }
    if (!ready) {
      if (lane == 0) atomicOr(err, (unsigned)kErrScanTimeout);
      *gave_up = true;
      break;
    }
    const unsigned total = __ballot_sync(kFull, (s & ~kTileValue) == kTileTotal);
    const unsigned needed = total ? kFull >> (kWarp - __ffs(total)) : kFull;
    unsigned long long v = (needed >> lane) & 1u ? s & kTileValue : 0ull;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
    prefix += v;
    if (total) break;
  }
  if (lane == 0 && tile > 0) status[tile] = kTileTotal | (prefix + sum);
  return prefix;
}

}  // namespace mc
