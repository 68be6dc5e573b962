// Stable LSD radix sort of 64-bit keys, one kernel per digit.
//
// One kernel reads the keys once for the histograms of all digits.  Each pass
// then reads and writes the keys once: a CTA counts its tile's digits,
// publishes the counts, ranks the keys stably and stages them in shared memory
// in digit order, and meanwhile its predecessors publish theirs, so that the
// sums over the tiles before it (a chained scan per digit; tiles are numbered
// by a ticket) are there when it stores each digit's run.
//
// What bounds it: issue (75% of the slots), in the ballots of the ranking and
// the walk over the predecessors' counts, which takes a window of eight tiles
// at a time; HBM traffic is 16 B per key and pass.  33.5 M keys of 41 bits (the
// CSR build at RMAT scale 20): six passes of 8 bits with a counting kernel, a
// scan and a scattering kernel took 1.81 ms; the histograms (103 us) and five
// passes of 9 bits (280 us each) take 1.50.  Measured and left out: counting
// the digits ahead with shared-memory atomics, to publish them before the
// ranking (312 us a pass), and finding a digit's lanes by atomicOr masks in
// shared memory (310 us: 82% of its bandwidth).
#include <algorithm>
#include <cstdlib>

#include "lookback.cuh"
#include "radix.cuh"

namespace mc {
namespace {

using u64 = unsigned long long;

// Digit widths: 8 bits, or 9 where that saves a pass.
constexpr int kRadixBitsMax = 9;
constexpr int kRadixBinsMax = 1 << kRadixBitsMax;
constexpr int kRadixPassesMax = 8;
// All passes' tile counts are cleared at once up to this many bytes.
constexpr size_t kStatusAtOnce = size_t(32) << 20;

template <int kBits>
__device__ __forceinline__ unsigned digit_of(u64 key, int shift) {
  return (unsigned)(key >> shift) & ((1u << kBits) - 1u);
}

// Lanes of the warp holding a real key with the same digit as this lane: the
// intersection over the digit's bits of each bit's ballot (or its
// complement), restricted to the lanes with a key.
template <int kBits>
__device__ __forceinline__ unsigned digit_peers(unsigned d, bool ok) {
  unsigned peers = __ballot_sync(kFull, ok);
#pragma unroll
  for (int b = 0; b < kBits; ++b) {
    const bool bit = (d >> b) & 1u;
    const unsigned m = __ballot_sync(kFull, bit);
    peers &= bit ? m : ~m;
  }
  return peers;
}

// hist[p * kRadixBinsMax + d] += keys whose digit p is d.
template <int kBits>
__global__ void __launch_bounds__(kSortThreads) radix_hist_kernel(const u64 *__restrict__ keys,
                                                                  int64_t count, int begin_bit,
                                                                  int passes, u64 *hist) {
  extern __shared__ int s_hist[];  // passes x bins
  constexpr int kBins = 1 << kBits;
  for (int i = threadIdx.x; i < passes * kBins; i += kSortThreads) s_hist[i] = 0;
  __syncthreads();
  const int64_t stride = (int64_t)gridDim.x * kSortThreads;
  int64_t i = (int64_t)blockIdx.x * kSortThreads + threadIdx.x;
  constexpr int kU = 4;
  for (; i < count; i += kU * stride) {
    u64 k[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) k[u] = i + u * stride < count ? __ldg(keys + i + u * stride) : 0;
#pragma unroll
    for (int u = 0; u < kU; ++u)
      if (i + u * stride < count)
        for (int p = 0; p < passes; ++p)
          atomicAdd(s_hist + p * kBins + digit_of<kBits>(k[u], begin_bit + p * kBits), 1);
  }
  __syncthreads();
  for (int j = threadIdx.x; j < passes * kBins; j += kSortThreads)
    if (s_hist[j]) atomicAdd(hist + (j >> kBits) * kRadixBinsMax + (j & (kBins - 1)), (u64)s_hist[j]);
}

// A tile's count of a digit: its own sum or the running total, in the low bits.
template <class S>
struct TileWord {
  static constexpr S kSum = S(1) << (sizeof(S) * 8 - 2);
  static constexpr S kTotal = S(2) << (sizeof(S) * 8 - 2);
  static constexpr S kValue = kSum - 1;
};

template <int kBits>
constexpr size_t pass_smem() {
  return sizeof(u64) * kSortTile + (sizeof(long long) + sizeof(int) * kSortWarps) * (1 << kBits);
}

// Exclusive prefix over the CTA's threads.
__device__ __forceinline__ int block_exclusive(int v, int *s_warp, int lane, int w) {
  const int incl = warp_inclusive_scan(v, lane);
  if (lane == kWarp - 1) s_warp[w] = incl;
  __syncthreads();
  int base = 0;
  for (int x = 0; x < w; ++x) base += s_warp[x];
  __syncthreads();
  return base + incl - v;
}

// S: word of a tile's count (32 bits hold 30-bit totals, else 64).
template <int kBits, class S>
__global__ void __launch_bounds__(kSortThreads, 4) radix_pass_kernel(
    const u64 *__restrict__ keys_in, u64 *__restrict__ keys_out, int64_t count, int shift,
    const u64 *__restrict__ hist, volatile S *status, unsigned *ticket, int max_polls,
    unsigned *err) {
  constexpr int kBins = 1 << kBits, kPer = (kBins + kSortThreads - 1) / kSortThreads;
  using W = TileWord<S>;
  extern __shared__ __align__(16) unsigned char smem[];
  u64 *stage = reinterpret_cast<u64 *>(smem);
  long long *bin_dest = reinterpret_cast<long long *>(stage + kSortTile);
  int(*cnt)[kBins] = reinterpret_cast<int(*)[kBins]>(bin_dest + kBins);  // per warp
  __shared__ int s_warp[kSortWarps];
  __shared__ long long s_long[kSortWarps];
  __shared__ unsigned s_tile;
  if (threadIdx.x == 0) s_tile = atomicAdd(ticket, 1u);
  for (int i = threadIdx.x; i < kSortWarps * kBins; i += kSortThreads) (&cnt[0][0])[i] = 0;
  __syncthreads();
  const int64_t tile = s_tile;
  const int lane = threadIdx.x & (kWarp - 1), w = threadIdx.x / kWarp;
  const int64_t tile_first = tile * kSortTile;
  const int64_t first = tile_first + (int64_t)w * kWarpSpan + lane;
  u64 k[kSortRounds];
  load_warp_keys(keys_in, count, first, k);
  // Stable ranks among the warp's keys of the same digit (round, then lane =
  // input order), two to a register.
  const unsigned lt = lanemask_lt();
  unsigned rank[kSortRounds / 2];
#pragma unroll
  for (int r = 0; r < kSortRounds; ++r) {
    const bool ok = first + r * kWarp < count;
    const unsigned d = digit_of<kBits>(k[r], shift);
    const unsigned peers = digit_peers<kBits>(d, ok);
    const int before = cnt[w][d];
    __syncwarp();
    if (ok && (peers & lt) == 0) cnt[w][d] = before + __popc(peers);
    __syncwarp();
    const unsigned mine = (unsigned)(before + __popc(peers & lt));
    rank[r / 2] = r % 2 ? rank[r / 2] | mine << 16 : mine;
  }
  __syncthreads();
  // Thread t owns digits t kPer ... : publish the tile's counts, and turn the
  // per-warp counts into first slots within the tile.
  const int d0 = threadIdx.x * kPer;
  int tot[kPer], mine = 0;
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    tot[i] = 0;
    if (d0 + i < kBins) {
#pragma unroll
      for (int x = 0; x < kSortWarps; ++x) tot[i] += cnt[x][d0 + i];
      status[tile * kBins + d0 + i] = (tile == 0 ? W::kTotal : W::kSum) | (S)tot[i];
    }
    mine += tot[i];
  }
  int start = block_exclusive(mine, s_warp, lane, w);
  int starts[kPer];
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    starts[i] = start;
    if (d0 + i < kBins) {
      int at = start;
#pragma unroll
      for (int x = 0; x < kSortWarps; ++x) {
        const int c = cnt[x][d0 + i];
        cnt[x][d0 + i] = at;
        at += c;
      }
    }
    start += tot[i];
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kSortRounds; ++r)
    if (first + r * kWarp < count)
      stage[cnt[w][digit_of<kBits>(k[r], shift)] + (int)(rank[r / 2] >> (r % 2 * 16) & 0xffffu)] = k[r];
  // Keys of smaller digits, then those of this digit in earlier tiles.
  long long below[kPer], sum = 0;
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    below[i] = sum;
    if (d0 + i < kBins) sum += (long long)hist[d0 + i];
  }
  long long incl = sum;
#pragma unroll
  for (int o = 1; o < kWarp; o <<= 1) {
    const long long v = __shfl_up_sync(kFull, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == kWarp - 1) s_long[w] = incl;
  __syncthreads();
  long long base = incl - sum;
  for (int x = 0; x < w; ++x) base += s_long[x];
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    if (d0 + i >= kBins) continue;
    S before = 0;
    int polls = 0;
    bool done = tile == 0;
    for (int64_t t = tile - 1; !done;) {
      if (polls == max_polls) {  // the output of this sort is then not used
        atomicOr(err, (unsigned)kErrScanTimeout);
        break;
      }
      // A window of predecessors at once: their loads overlap.
      constexpr int kWindow = 8;
      S v[kWindow];
#pragma unroll
      for (int u = 0; u < kWindow; ++u)
        v[u] = t - u >= 0 ? (S)status[(t - u) * kBins + d0 + i] : W::kTotal;
      int used = 0;
#pragma unroll
      for (int u = 0; u < kWindow; ++u) {
        if (done || used < u || (v[u] & ~W::kValue) == 0) continue;  // stops at the first gap
        before += v[u] & W::kValue;
        done = (v[u] & ~W::kValue) == W::kTotal;
        ++used;
      }
      t -= used;
      polls += used == 0;
    }
    if (tile > 0) status[tile * kBins + d0 + i] = W::kTotal | (before + (S)tot[i]);
    bin_dest[d0 + i] = base + below[i] + (long long)before - starts[i];
  }
  __syncthreads();
  const int in_tile = (int)min((int64_t)kSortTile, count - tile_first);
  for (int j = threadIdx.x; j < in_tile; j += kSortThreads) {
    const u64 key = stage[j];
    const int64_t to = bin_dest[digit_of<kBits>(key, shift)] + j;
    // (After a wait that gave up the slot may be wrong, never out of range.)
    if (to >= 0 && to < count) keys_out[to] = key;
  }
}

int passes_of(int bits) { return std::max(1, (bits + kRadixBitsMax - 1) / kRadixBitsMax); }
int width_of(int bits) { return passes_of(bits) * 8 >= bits ? 8 : 9; }

size_t word_bytes(int64_t count) { return count < (int64_t(1) << 30) ? 4 : 8; }

size_t head_bytes() { return sizeof(u64) * kRadixBinsMax * kRadixPassesMax + 256; }

template <int kBits, class S>
cudaError_t sort_passes(u64 *keys, u64 *alt, int64_t count, int begin_bit, int passes, void *work,
                        unsigned *err, cudaStream_t s, u64 **sorted, int64_t *launches) {
  // work: the histograms, a ticket per pass, the tile counts.
  u64 *hist = static_cast<u64 *>(work);
  unsigned *tickets = reinterpret_cast<unsigned *>(hist + kRadixBinsMax * kRadixPassesMax);
  S *status = reinterpret_cast<S *>(static_cast<char *>(work) + head_bytes());
  const int64_t tiles = sort_tiles(count);
  const size_t one = sizeof(S) * ((size_t)tiles << kBits);
  const bool at_once = one * passes <= kStatusAtOnce;
  cudaError_t e = cudaMemsetAsync(work, 0, head_bytes() + (at_once ? one * passes : 0), s);
  if (e != cudaSuccess) return e;
  const size_t hist_smem = sizeof(int) * ((size_t)passes << kBits);
  int device = 0, num_sms = 0;
  e = cudaGetDevice(&device);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, device);
  if (e != cudaSuccess) return e;
  const int64_t blocks = std::max<int64_t>(1, std::min<int64_t>(tiles, 8 * num_sms));
  radix_hist_kernel<kBits><<<(unsigned)blocks, kSortThreads, hist_smem, s>>>(keys, count, begin_bit,
                                                                           passes, hist);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  auto kern = radix_pass_kernel<kBits, S>;
  e = allow_smem((const void *)kern, pass_smem<kBits>());
  if (e != cudaSuccess) return e;
  const int polls = wait_polls();
  u64 *buf[2] = {keys, alt};
  int cur = 0;
  for (int p = 0; p < passes; ++p) {
    S *st = status + (at_once ? (size_t)p * ((size_t)tiles << kBits) : 0);
    if (!at_once) {
      e = cudaMemsetAsync(st, 0, one, s);
      if (e != cudaSuccess) return e;
    }
    kern<<<(unsigned)tiles, kSortThreads, pass_smem<kBits>(), s>>>(
        buf[cur], buf[cur ^ 1], count, begin_bit + p * kBits, hist + p * kRadixBinsMax, st,
        tickets + p, polls, err);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    cur ^= 1;
  }
  *launches += 1 + passes;
  *sorted = buf[cur];
  return cudaSuccess;
}

}  // namespace

int wait_polls() {
  const char *env = std::getenv("MERCURY_WAIT_POLLS");
  return env ? std::max(0, std::atoi(env)) : 1 << 22;
}

size_t radix_work_bytes(int64_t count, int bits) {
  const size_t one = word_bytes(count) * (size_t)sort_tiles(count) << kRadixBitsMax;
  const size_t all = one * passes_of(bits);
  return head_bytes() + (all <= kStatusAtOnce ? all : std::max(one, kStatusAtOnce));
}

cudaError_t radix_sort_u64(u64 *keys, u64 *alt, int64_t count, int begin_bit, int end_bit,
                           void *work, unsigned *err, cudaStream_t s, u64 **sorted,
                           int64_t *launches) {
  *sorted = keys;
  if (count <= 0 || end_bit <= begin_bit) return cudaSuccess;
  const int bits = end_bit - begin_bit, passes = passes_of(bits);
  const bool narrow = word_bytes(count) == 4;
  if (width_of(bits) == 8)
    return narrow ? sort_passes<8, unsigned>(keys, alt, count, begin_bit, passes, work, err, s, sorted, launches)
                  : sort_passes<8, u64>(keys, alt, count, begin_bit, passes, work, err, s, sorted, launches);
  return narrow ? sort_passes<9, unsigned>(keys, alt, count, begin_bit, passes, work, err, s, sorted, launches)
                : sort_passes<9, u64>(keys, alt, count, begin_bit, passes, work, err, s, sorted, launches);
}

}  // namespace mc
