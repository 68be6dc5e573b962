// Scratch blocks shared by the counts of a device.
//
// A count takes a block, waits for its stream and gives the block back, and
// the next count, of any handle on any stream, gets the same block as it is.
// The stream-ordered pool alone does not give that: each handle has a stream
// of its own, and a block freed on one stream and asked for on another, or
// asked for in another size, is mapped anew.  Measured over 1,024 resident
// graphs of mixed sizes counted in turn: 3.0 ms per P4 count of 26 us on the
// device from the pool, 0.06 ms from here.
//
// Bounded: blocks above kBlockMax are not kept, and no more than kKeepMax per
// device in all (the ones given back longest ago go first).  Everything goes
// back to the pool when the device's last graph handle is released, and before
// any allocation fails (dev_alloc).
#include <algorithm>
#include <mutex>
#include <vector>

#include "device_common.cuh"

namespace mc {
namespace {

constexpr size_t kBlockMin = size_t(8) << 20;
constexpr size_t kBlockMax = size_t(1) << 30;
constexpr size_t kKeepMax = size_t(2) << 30;
constexpr int kMaxDevices = 64;  // further devices keep no blocks

struct Block {
  void *p;
  size_t bytes;
};

struct Keep {
  std::mutex mu;
  std::vector<Block> blocks;  // oldest first
  size_t bytes = 0;
  int64_t handles = 0;
};

// Never destroyed: a handle may be released while the process exits.
Keep *keep_of(int device) {
  static Keep *all = new Keep[kMaxDevices];
  return device >= 0 && device < kMaxDevices ? all + device : nullptr;
}

// Eight block sizes per power of two, so that counts of similar graphs ask
// for the same ones.
size_t block_bytes(size_t bytes) {
  size_t step = size_t(1) << 20;
  while (step * 16 < bytes) step *= 2;
  return std::max(kBlockMin, (bytes + step - 1) / step * step);
}

}  // namespace

cudaError_t scratch_take(void **p, size_t bytes, size_t *got, int device, cudaStream_t s) {
  if (Keep *k = keep_of(device)) {
    std::lock_guard<std::mutex> lock(k->mu);
    size_t best = k->blocks.size();
    for (size_t i = 0; i < k->blocks.size(); ++i)
      if (k->blocks[i].bytes >= bytes &&
          (best == k->blocks.size() || k->blocks[i].bytes < k->blocks[best].bytes))
        best = i;
    if (best < k->blocks.size()) {
      *p = k->blocks[best].p;
      *got = k->blocks[best].bytes;
      k->bytes -= *got;
      k->blocks.erase(k->blocks.begin() + (std::ptrdiff_t)best);
      return cudaSuccess;
    }
  }
  *got = block_bytes(bytes);
  return dev_alloc(p, *got, s);
}

void scratch_give(void *p, size_t bytes, int device, cudaStream_t s) {
  if (!p) return;
  Keep *k = keep_of(device);
  if (!k || bytes > kBlockMax) {
    dev_free(p, s);
    return;
  }
  std::lock_guard<std::mutex> lock(k->mu);
  if (k->handles == 0) {
    dev_free(p, s);
    return;
  }
  k->blocks.push_back({p, bytes});
  k->bytes += bytes;
  size_t drop = 0;
  while (k->bytes > kKeepMax) {
    dev_free(k->blocks[drop].p, s);
    k->bytes -= k->blocks[drop++].bytes;
  }
  k->blocks.erase(k->blocks.begin(), k->blocks.begin() + (std::ptrdiff_t)drop);
}

bool scratch_flush(int device, cudaStream_t s) {
  Keep *k = keep_of(device);
  if (!k) return false;
  std::lock_guard<std::mutex> lock(k->mu);
  const bool any = !k->blocks.empty();
  for (const Block &b : k->blocks) dev_free(b.p, s);
  k->blocks.clear();
  k->bytes = 0;
  return any;
}

size_t scratch_kept(int device) {
  Keep *k = keep_of(device);
  if (!k) return 0;
  std::lock_guard<std::mutex> lock(k->mu);
  return k->bytes;
}

void scratch_attach(int device) {
  if (Keep *k = keep_of(device)) {
    std::lock_guard<std::mutex> lock(k->mu);
    k->handles += 1;
  }
}

void scratch_detach(int device, cudaStream_t s) {
  Keep *k = keep_of(device);
  if (!k) return;
  bool last = false;
  {
    std::lock_guard<std::mutex> lock(k->mu);
    last = --k->handles == 0;
  }
  if (last) scratch_flush(device, s);
}

cudaError_t dev_alloc(void **p, size_t bytes, cudaStream_t s) {
  cudaError_t e = cudaMallocAsync(p, bytes < 8 ? 8 : bytes, s);
  if (e != cudaErrorMemoryAllocation) return e;
  int device = -1;
  if (cudaGetDevice(&device) != cudaSuccess || !scratch_flush(device, s)) return e;
  cudaGetLastError();
  return cudaMallocAsync(p, bytes < 8 ? 8 : bytes, s);
}

}  // namespace mc
