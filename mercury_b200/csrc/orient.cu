// Device preprocessing of the triangle-count path: contract validation and
// the degree-ordered DAG, built by two streaming row-aware passes over the
// symmetric CSR, plus the counting task queues.
//
// Reference behaviour restated here: Graph::orientation_with_division
// (graph.cc:196-321) runs on the host with OpenMP in five passes.  The DAG
// rule is the same (u->v iff deg v > deg u, or equal and v > u:
// graph.cc:207-214).  The reference then splits edges into a "small" CSR
// (DAG direction, both out-degrees <= 128) and a "large" CSR (REVERSE_DAG:
// from the endpoint with the larger DAG out-degree, ties to the larger id,
// graph.cc:238-263), skipping edges with an endpoint of out-degree 0
// (graph.cc:246).  Here every DAG edge with both out-degrees >= 1 belongs to
// its larger-out-degree end (the reference's "large" rule for all edges);
// the counting kernels find an owner's partners by filtering the owner's own
// symmetric row, so no partner CSR is written.  Routing is per owner
// (d+ <= kLeafMaxOut: warp task, else CTA task).
//
// Passes (each CTA owns a tile of kTileEdges consecutive CSR entries, each warp
// 512 of them in rounds of 32, one entry per lane):
//   A  DAG keep masks, per-tile DAG counts, d+ of every row by atomics
//   B  DAG entries and row offsets written from the keep masks
// Each vertex's (degree, d+) pair is one 8-byte word (key[]).
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <cstdio>
#include <cstdlib>

#include "dgraph.cuh"
#include "device_common.cuh"
#include "lookback.cuh"
#include "radix.cuh"
#include "scan.cuh"

namespace mc {
namespace {

constexpr int kTileWarps = kTileThreads / kWarp;
constexpr int kTileRounds = kEdgesPerThread;                // 32-entry rounds per warp
constexpr int kTileWords = (int)(kTileEdges / kWarp);       // keep words per tile

// The rows of a tile's entries.  Every non-empty row that starts inside the
// tile marks its first entry with its number from the tile's first row on; an
// entry's row is the nearest mark at or before it, which a ballot finds within
// a round, and a carry across rounds.  No lane ever walks rows (sixteen
// consecutive entries per lane, each lane stepping over its rows' offsets,
// diverged on every row boundary and empty row: 322 us for the checks at RMAT
// scale 20, against 157; at scale 22, 1.08 ms for pass A and 1.13 for pass B,
// against 0.79 and 0.36).
struct TileMarks {
  int64_t lo;      // row of the tile's first entry
  bool at_start;   // that row starts at the tile
  int carry;       // this warp's row before its first round
  int m[kTileRounds];
};

// rows (optional): {first row, last row} of this tile, precomputed by
// tile_rows_kernel; without it two threads binary-search rowptr.
__device__ __forceinline__ TileMarks tile_marks(const int64_t *__restrict__ rowptr, int64_t n,
                                                int64_t t0, int64_t t1,
                                                const int64_t *__restrict__ rows) {
  __shared__ __align__(16) int s_mark[kTileEdges];
  __shared__ int64_t s_rows[2];
  __shared__ int s_max[kTileWarps];
  const int lane = threadIdx.x & (kWarp - 1), warp = threadIdx.x / kWarp;
  if (rows) {
    if (threadIdx.x < 2) s_rows[threadIdx.x] = __ldg(rows + threadIdx.x);
  } else {
    if (threadIdx.x == 0) s_rows[0] = upper_row(rowptr, 0, n - 1, t0);
    if (threadIdx.x == kTileThreads - 1) s_rows[1] = upper_row(rowptr, 0, n - 1, t1 - 1);
  }
  int4 *m4 = reinterpret_cast<int4 *>(s_mark);
  for (int i = threadIdx.x; i < kTileEdges / 4; i += kTileThreads) m4[i] = make_int4(0, 0, 0, 0);
  __syncthreads();
  TileMarks t;
  t.lo = s_rows[0];
  const int64_t hi = s_rows[1];
  t.at_start = __ldg(rowptr + t.lo) == t0;
  for (int64_t r = t.lo + 1 + threadIdx.x; r <= hi; r += kTileThreads) {
    const int64_t b = __ldg(rowptr + r);
    if (b < __ldg(rowptr + r + 1)) s_mark[b - t0] = (int)(r - t.lo);
  }
  __syncthreads();
  int mx = 0;
#pragma unroll
  for (int k = 0; k < kTileRounds; ++k) {
    t.m[k] = s_mark[(warp * kTileRounds + k) * kWarp + lane];
    mx = max(mx, t.m[k]);
  }
  mx = __reduce_max_sync(kFull, mx);
  if (lane == 0) s_max[warp] = mx;
  __syncthreads();
  t.carry = 0;
  for (int w = 0; w < warp; ++w) t.carry = max(t.carry, s_max[w]);
  return t;
}

// Where a pass finds its tiles' column entries: the whole array (col_base
// 0, tile_base 0), or a staged chunk of it holding entries from col_base on
// for the tiles from tile_base on (chunks start on tile boundaries).
struct ColumnChunk {
  const int32_t *col;
  int64_t col_base;
  int64_t tile_base;
};

// x in N(u) (binary search; rows are checked sorted, and the probe never
// leaves the column array where their offsets are not).
__device__ bool in_row(const int64_t *__restrict__ rowptr, const int32_t *__restrict__ col,
                       int64_t nnz, int32_t u, int32_t x) {
  int64_t lo = __ldg(rowptr + u), hi = __ldg(rowptr + u + 1) - 1;
  while (lo <= hi && lo >= 0 && hi < nnz) {
    const int64_t mid = lo + ((hi - lo) >> 1);
    const int32_t m = __ldg(col + mid);
    if (m == x) return true;
    if (m < x) lo = mid + 1;
    else hi = mid - 1;
  }
  return false;
}

// Pass A (kKeep): the DAG entries as one bit per entry in keep[] (kTileWords
// words per tile), per-tile counts, and d+ of every row by one atomic per row
// and round on key[].y (which starts at 0).  kCheck: the entries against the
// CSR contract (ids in range, strictly ascending rows, no self-loops and, with
// check_sym, symmetry), what breaks it into *err; an id out of range is then
// never gathered with.  With stop given, nothing runs once a contract bit is
// set there.
template <bool kKeep, bool kCheck>
__global__ void __launch_bounds__(kTileThreads)
    dag_keep_kernel(const int64_t *__restrict__ rowptr, ColumnChunk cc,
                    const int32_t *__restrict__ deg, int64_t n, int64_t nnz, int2 *key,
                    unsigned *keep, int32_t *counts_out, const unsigned *stop, int check_sym,
                    unsigned *err, const int64_t *__restrict__ tile_rows) {
  // One word, the same for the whole CTA: the checks of an earlier chunk found
  // a bad entry.
  if (stop && (*(volatile const unsigned *)stop & kErrContract)) return;
  __shared__ int s_count[kTileWarps];
  const int lane = threadIdx.x & (kWarp - 1), warp = threadIdx.x / kWarp;
  const int64_t tile = cc.tile_base + blockIdx.x;
  const int64_t t0 = tile * kTileEdges;
  const int64_t t1 = min(t0 + kTileEdges, nnz);
  const int64_t e0 = t0 + (int64_t)warp * kTileRounds * kWarp + lane;  // round 0
  int u[kTileRounds], du[kTileRounds];
#pragma unroll
  for (int k = 0; k < kTileRounds; ++k) {
    const int64_t e = e0 + k * kWarp;
    u[k] = e < t1 ? __ldg(cc.col + (e - cc.col_base)) : 0;
  }
  if (kKeep) {
    // All sixteen degree gathers in flight before the rows are known.
#pragma unroll
    for (int k = 0; k < kTileRounds; ++k)
      du[k] = !kCheck || (u[k] >= 0 && u[k] < n) ? __ldg(deg + u[k]) : 0;
  }
  const TileMarks tm = tile_marks(rowptr, n, t0, t1, tile_rows ? tile_rows + 2 * tile : nullptr);
  int carry = tm.carry, count = 0;
  unsigned bad = 0, mine = 0;
  const unsigned upto = kFull >> (kWarp - 1 - lane);
  // The entry before this warp's first (checks of a row that goes on).
  int last = 0;
  if (kCheck && lane == 0 && e0 > 0 && e0 < t1) last = __ldg(cc.col + (e0 - 1 - cc.col_base));
  last = kCheck ? __shfl_sync(kFull, last, 0) : 0;
#pragma unroll
  for (int k = 0; k < kTileRounds; ++k) {
    const int64_t e = e0 + k * kWarp;
    const bool in = e < t1;
    const unsigned starts = __ballot_sync(kFull, tm.m[k] > 0);
    const unsigned before = starts & upto;
    int row = __shfl_sync(kFull, tm.m[k], before ? kWarp - 1 - __clz(before) : 0);
    if (!before) row = carry;
    if (starts) carry = __shfl_sync(kFull, tm.m[k], kWarp - 1 - __clz(starts));
    const int64_t v = tm.lo + row;
    if (kCheck) {
      int prev = __shfl_up_sync(kFull, u[k], 1);
      if (lane == 0) prev = last;
      last = __shfl_sync(kFull, u[k], kWarp - 1);
      if (in) {
        if (u[k] < 0 || (int64_t)u[k] >= n) {
          bad |= kErrIdRange;
        } else {
          const bool first = tm.m[k] > 0 || (e == t0 && tm.at_start);
          if ((int64_t)u[k] == v) bad |= kErrSelfLoop;
          if (!first && prev >= u[k]) bad |= kErrUnsorted;
          if (check_sym && !in_row(rowptr, cc.col - cc.col_base, nnz, u[k], (int32_t)v))
            bad |= kErrAsymmetric;
        }
      }
    }
    if (kKeep) {
      const int dv = __ldg(deg + v);
      const bool up = in && (du[k] > dv || (du[k] == dv && u[k] > (int)v));
      const unsigned word = __ballot_sync(kFull, up);
      if (lane == k) mine = word;
      count += __popc(word);
      // The row's entries of this round, at its first lane.
      if ((lane == 0 || tm.m[k] > 0) && word) {
        const unsigned later = starts & ~upto;
        const unsigned seg = (later ? (1u << (__ffs(later) - 1)) - 1u : kFull) & (kFull << lane);
        const int c = __popc(word & seg);
        if (c) atomicAdd(&key[v].y, c);
      }
    }
  }
  if (kCheck && bad) atomicOr(err, bad);
  if (kKeep) {
    if (lane < kTileRounds) keep[tile * kTileWords + warp * kTileRounds + lane] = mine;
    if (lane == 0) s_count[warp] = count;
    __syncthreads();
    if (threadIdx.x == 0) {
      int t = 0;
      for (int w = 0; w < kTileWarps; ++w) t += s_count[w];
      counts_out[tile] = t;
    }
  }
}

// Pass B: the kept entries compacted into out_col (and, when rank is given,
// their ranks into out_rank), and out_rowptr[r] = kept entries before
// rowptr[r] for the rows that start in the tile, empty ones included.  With
// chunk_end given, nothing is written when *chunk_end (the DAG entries up to
// the end of this chunk) exceeds cap; stop as in pass A.
__global__ void __launch_bounds__(kTileThreads)
    dag_write_kernel(const int64_t *__restrict__ rowptr, ColumnChunk cc, int64_t n, int64_t nnz,
                     const unsigned *__restrict__ keep, const int64_t *__restrict__ offs_in,
                     int64_t *out_rowptr, int32_t *out_col, const int32_t *__restrict__ rank,
                     int32_t *out_rank, const int64_t *chunk_end, int64_t cap,
                     const unsigned *stop, const int64_t *__restrict__ tile_rows) {
  if (stop && (*(volatile const unsigned *)stop & kErrContract)) return;
  if (chunk_end && *chunk_end > cap) return;
  static_assert(kTileWords <= kTileThreads, "one thread per keep word");
  __shared__ unsigned s_word[kTileWords];
  __shared__ int s_pre[kTileWords], s_sum[kTileWarps];
  const int lane = threadIdx.x & (kWarp - 1), warp = threadIdx.x / kWarp;
  const int64_t tile = cc.tile_base + blockIdx.x;
  const int64_t t0 = tile * kTileEdges;
  const int64_t t1 = min(t0 + kTileEdges, nnz);
  const unsigned word = threadIdx.x < kTileWords ? keep[tile * kTileWords + threadIdx.x] : 0u;
  const int incl = warp_inclusive_scan(__popc(word), lane);
  if (lane == kWarp - 1) s_sum[warp] = incl;
  __syncthreads();
  int pre = incl - __popc(word);
  for (int w = 0; w < warp; ++w) pre += s_sum[w];
  if (threadIdx.x < kTileWords) {
    s_word[threadIdx.x] = word;
    s_pre[threadIdx.x] = pre;
  }
  __syncthreads();
  const int64_t base = offs_in[tile];
  const unsigned lt = (1u << lane) - 1u;
  const int64_t e0 = t0 + (int64_t)warp * kTileRounds * kWarp + lane;
  constexpr int kU = 8;
#pragma unroll
  for (int k0 = 0; k0 < kTileRounds; k0 += kU) {
    int u[kU], rk[kU];
    unsigned wd[kU];
#pragma unroll
    for (int i = 0; i < kU; ++i) {
      wd[i] = s_word[warp * kTileRounds + k0 + i];
      const bool kept = (wd[i] >> lane) & 1u;
      u[i] = kept ? __ldg(cc.col + (e0 + (k0 + i) * kWarp - cc.col_base)) : 0;
    }
#pragma unroll
    for (int i = 0; i < kU; ++i)
      rk[i] = out_rank && ((wd[i] >> lane) & 1u) ? __ldg(rank + u[i]) : 0;
#pragma unroll
    for (int i = 0; i < kU; ++i) {
      if (!((wd[i] >> lane) & 1u)) continue;
      const int64_t to = base + s_pre[warp * kTileRounds + k0 + i] + __popc(wd[i] & lt);
      out_col[to] = u[i];
      if (out_rank) out_rank[to] = rk[i];
    }
  }
  // Rows that start here: those after the previous tile's last row.  Rows
  // after the last entry (trailing empty rows and row n) start at nnz.
  const int64_t first = tile > 0 ? __ldg(tile_rows + 2 * tile - 1) + 1 : 0;
  const int64_t last = t1 == nnz ? n : __ldg(tile_rows + 2 * tile + 1);
  const int end_pre = s_pre[kTileWords - 1] + __popc(s_word[kTileWords - 1]);
  for (int64_t r = first + threadIdx.x; r <= last; r += kTileThreads) {
    const int64_t at = __ldg(rowptr + r) - t0;
    const int w = (int)(at / kWarp);
    out_rowptr[r] =
        base + (w < kTileWords ? s_pre[w] + __popc(s_word[w] & ((1u << (at & (kWarp - 1))) - 1u))
                               : end_pre);
  }
}

// rows[2t] / rows[2t + 1] = the rows holding the first and the last entry of
// tile t: each non-empty row marks the tiles whose first or last entry it
// holds (rowptr validated: monotone, ends at nnz).
__global__ void tile_rows_kernel(const int64_t *__restrict__ rowptr, int64_t n, int64_t nnz,
                                 int64_t tiles, int64_t *rows) {
  const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= n) return;
  const int64_t b = rowptr[v], e = rowptr[v + 1];
  if (b >= e) return;
  for (int64_t t = b / kTileEdges; t <= (e - 1) / kTileEdges && t < tiles; ++t) {
    const int64_t first = t * kTileEdges;
    const int64_t last = min(first + kTileEdges, nnz) - 1;
    if (first >= b && first < e) rows[2 * t] = v;
    if (last >= b && last < e) rows[2 * t + 1] = v;
  }
}

// Tile offsets of one staged chunk: offs[0] holds the DAG entries of the
// earlier chunks; offs[i] = offs[0] + local[i] for i in [0, count] (local is
// the chunk's exclusive scan, local[0] = 0, so offs[0] is rewritten with its
// own value). The chunk's end above cap raises kErrDagCapacity.
__global__ void chunk_offsets_kernel(const int64_t *__restrict__ local, int64_t count,
                                     int64_t *offs, int64_t cap, unsigned *err) {
  const int64_t base = offs[0];
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i > count) return;
  const int64_t v = base + local[i];
  offs[i] = v;
  if (i == count && v > cap) atomicOr(err, (unsigned)kErrDagCapacity);
}

// Offsets monotone with the right ends; *max_deg receives the largest row.
__global__ void validate_rowptr_kernel(const int64_t *rowptr, int64_t n, int64_t nnz,
                                       unsigned *err, unsigned long long *max_deg) {
  const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  long long d = 0;
  if (v <= n) {
    const int64_t a = rowptr[v];
    bool bad = (v == 0 && a != 0) || (v == n && a != nnz) || a < 0 || a > nnz;
    if (v < n) {
      d = rowptr[v + 1] - a;
      if (d < 0) bad = true;
    }
    if (bad) atomicOr(err, (unsigned)kErrRowptr);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) d = max(d, __shfl_down_sync(kFull, d, o));
  if ((threadIdx.x & 31) == 0 && d > 0) atomicMax(max_deg, (unsigned long long)d);
}

// Degree-rank sort keys: position i holds vertex n-1-i, keyed by
// (max_degree - degree) in the high word. A stable sort of the high word
// keeps equal degrees in descending id order, so the sorted position is the
// rank in (degree desc, id desc) order.
__global__ void rank_keys_kernel(const int2 *__restrict__ key, int64_t n, int max_degree,
                                 unsigned long long *__restrict__ keys) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n)
    keys[i] = ((unsigned long long)(unsigned)(max_degree - key[n - 1 - i].x) << 32) |
              (unsigned long long)i;
}

__global__ void rank_scatter_kernel(const unsigned long long *__restrict__ sorted, int64_t n,
                                    int32_t *__restrict__ rank) {
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  // (A sort whose wait gave up leaves positions unwritten.)
  if (p < n && (int64_t)(uint32_t)sorted[p] < n)
    rank[n - 1 - (int64_t)(uint32_t)sorted[p]] = (int32_t)p;
}

// Core bitmaps: warp per rank p < core_ranks; its vertex is the one whose
// sort key sits at position p. Every entry z of N+(v) ranks below p, so it
// sets bit z of the words from core_offset(p) (which start
// cleared; the row's last quad pads to a multiple of 128 bits with zeros).
// Nothing runs when an exact-size DAG was overrun: its rows were
// then never written.
__global__ void core_bits_kernel(const unsigned long long *__restrict__ sorted, int64_t n,
                                 int core_ranks, const int64_t *__restrict__ dag_rowptr,
                                 const int32_t *__restrict__ dag_rank, unsigned *core,
                                 unsigned *err) {
  const int64_t p = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / kWarp;
  const int lane = threadIdx.x & (kWarp - 1);
  if (p >= core_ranks || (*(volatile unsigned *)err & (kErrDagCapacity | kErrContract | kErrScanTimeout)))
    return;
  const int64_t v = n - 1 - (int64_t)(uint32_t)sorted[p];
  if (v < 0) return;
  unsigned *row = core + core_offset(p);
  for (int64_t e = dag_rowptr[v] + lane; e < dag_rowptr[v + 1]; e += kWarp) {
    const int z = __ldg(dag_rank + e);
    if (z >= 0 && z < p) atomicOr(row + (z >> 5), 1u << (z & 31));
    else atomicOr(err, (unsigned)kErrRank);
  }
}

// key[v] = {degree, 0}; deg[v] = degree alone (4 bytes per gather in pass A).
// The first `words` words of status are cleared (words <= n + 4), and so are
// the waits that gave up in an earlier orientation or count.
__global__ void init_key_kernel(const int64_t *rowptr, int64_t n, int2 *key, int32_t *deg,
                                unsigned long long *status, int64_t words, int64_t *lists_bad,
                                unsigned *err) {
  const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (v == 0) {
    atomicAnd(err, ~(unsigned)(kErrScanTimeout | kErrWaitTimeout));
    *lists_bad = 0;
  }
  if (v < words) status[v] = 0;
  if (v < n) {
    const int d = (int)(rowptr[v + 1] - rowptr[v]);
    key[v] = make_int2(d, 0);
    deg[v] = d;
  }
}

struct TaskLists {
  int64_t *hub_end, *leaf_end, *mega_end;  // receive the lists' lengths
  int64_t *bad;                            // set: the ranks or the lists are not complete
  uint64_t *hub, *leaf, *mega;
  // One running sum per list and block (kTaskThreads x kTaskItems vertices), a
  // ticket; cleared by init_key_kernel.
  unsigned long long *status;
  int64_t blocks;
};
constexpr int kTaskThreads = 256, kTaskItems = 4;  // vertices per thread

// pinfo[v] = {d+(v), rank(v) (INT_MAX without ranks), dag_rowptr[v]}; the
// largest d+; and the tasks of each owner (chunks of its symmetric row; a task
// word is the owner in the high half, the chunk in the low half), appended to
// the hub, leaf and large-table hub lists in vertex order: shards name tasks
// by position, and the leaf kernel took 849 instead of 632 us on a Chung-Lu
// graph of 2 M vertices with the blocks' tasks in order of arrival.  One launch
// with a chained scan per list; a counting kernel, three scans and a filling
// kernel took 188 us there and 64 us at RMAT scale 16.
__global__ void __launch_bounds__(kTaskThreads) partner_tasks_kernel(
    const int2 *__restrict__ key, const int32_t *__restrict__ rank,
    const int64_t *__restrict__ dag_rowptr, int64_t n, int4 *__restrict__ pinfo, TaskLists t,
    unsigned long long *max_out, BatchView bv, int max_polls, unsigned *err) {
  constexpr int kW = kTaskThreads / kWarp;
  __shared__ int s_warp[3][kW];
  __shared__ int s_max[kW];
  __shared__ int64_t s_base[3], s_block;
  if (threadIdx.x == 0) s_block = (int64_t)atomicAdd(t.status + 3 * t.blocks, 1ull);
  __syncthreads();
  const int64_t block = s_block;
  const int64_t v0 = (block * kTaskThreads + threadIdx.x) * kTaskItems;
  const int lane = threadIdx.x & (kWarp - 1), warp = threadIdx.x / kWarp;
  int dmax = 0, c[3] = {0, 0, 0};  // hub, leaf, mega
  int own[kTaskItems], chunks[kTaskItems];  // each vertex's list (-1: none) and tasks
#pragma unroll
  for (int i = 0; i < kTaskItems; ++i) {
    const int64_t v = v0 + i;
    own[i] = -1;
    chunks[i] = 0;
    if (v >= n) continue;
    const int2 kv = key[v];
    const int d = kv.y;
    dmax = max(dmax, d);
    const long long st = dag_rowptr[v];
    pinfo[v] = make_int4(d, rank ? rank[v] : INT_MAX, (int)(unsigned)(st & 0xffffffffll),
                         (int)(st >> 32));
    int leaf_max = kLeafMaxOut;
    bool counted = true;
    if (bv.gid) {  // batch: only triangle jobs get tasks, with their graph's threshold
      const int g = bv.gid[v];
      counted = bv.job[g] == 0;
      if (bv.param) leaf_max = bv.param[g].x;
    }
    // Owners need d+ >= 1; every neighbour of the row may be a partner.
    if (counted && d >= 1) {
      own[i] = d <= leaf_max ? 1 : d <= kHubSmallMaxOut ? 0 : 2;
      const int per = own[i] == 1 ? kLeafChunk : kHubChunk;
      chunks[i] = (kv.x + per - 1) / per;
#pragma unroll
      for (int k = 0; k < 3; ++k) c[k] += own[i] == k ? chunks[i] : 0;
    }
  }
  int incl[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) incl[k] = warp_inclusive_scan(c[k], lane);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) dmax = max(dmax, __shfl_xor_sync(kFull, dmax, o));
  if (lane == kWarp - 1) {
#pragma unroll
    for (int k = 0; k < 3; ++k) s_warp[k][warp] = incl[k];
    s_max[warp] = dmax;
  }
  __syncthreads();
  if (warp < 3) {  // warp k: list k
    unsigned long long sum = 0;
    for (int w = 0; w < kW; ++w) sum += (unsigned)s_warp[warp][w];
    bool gave_up = false;
    const unsigned long long before =
        tile_prefix(t.status + warp * t.blocks, block, sum, lane, max_polls, err, &gave_up);
    // (The rank sort's waits are over before this launch.)
    if (lane == 0 && block == 0 && warp == 0) gave_up = (*err & kErrScanTimeout) != 0;
    if (lane == 0) {
      if (gave_up) *t.bad = 1;
      s_base[warp] = (int64_t)before;
      if (block == t.blocks - 1)
        *(warp == 0 ? t.hub_end : warp == 1 ? t.leaf_end : t.mega_end) = (int64_t)(before + sum);
    }
  } else if (warp == 3 && lane == 0) {
    int m = 0;
    for (int w = 0; w < kW; ++w) m = max(m, s_max[w]);
    if (m > 0) atomicMax(max_out, (unsigned long long)m);
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    if (c[k] == 0) continue;
    uint64_t *out = k == 0 ? t.hub : k == 1 ? t.leaf : t.mega;
    int64_t at = s_base[k] + incl[k] - c[k];
    for (int w = 0; w < warp; ++w) at += s_warp[k][w];
#pragma unroll
    for (int i = 0; i < kTaskItems; ++i) {
      if (own[i] != k) continue;
      const uint64_t hi = (uint64_t)(v0 + i) << 32;
      for (int j = 0; j < chunks[i]; ++j) out[at++] = hi | (uint32_t)j;
    }
  }
}

// Partner edges (owner rule) and their streamed-list work, for statistics:
// one warp per row, lanes over its entries.
__global__ void partner_stats_kernel(const int64_t *rowptr, const int32_t *col, const int2 *key,
                                     int64_t n, unsigned long long *out) {
  unsigned long long pe = 0, work = 0;
  const int lane = threadIdx.x & (kWarp - 1);
  const int64_t warps = (int64_t)gridDim.x * blockDim.x / kWarp;
  for (int64_t x = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / kWarp; x < n; x += warps) {
    const int px = key[x].y;
    if (px < 1) continue;
    for (int64_t e = rowptr[x] + lane; e < rowptr[x + 1]; e += kWarp) {
      const int y = col[e];
      const int py = key[y].y;
      if (py >= 1 && (px > py || (px == py && (int)x > y))) {
        ++pe;
        work += (unsigned long long)py;
      }
    }
  }
  pe = warp_sum_u64(pe);
  work = warp_sum_u64(work);
  if ((threadIdx.x & 31) == 0) {
    if (pe) atomicAdd(out, pe);
    if (work) atomicAdd(out + 1, work);
  }
}

unsigned grid_for(int64_t items, int threads) {
  return (unsigned)std::max<int64_t>(1, (items + threads - 1) / threads);
}

}  // namespace

int validate_graph(mc_dgraph *g, unsigned flags) {
  NvtxRange range("validate_graph");
  MC_CUDA_TRY(cudaMemsetAsync(g->err, 0, sizeof(unsigned), g->stream));
  MC_CUDA_TRY(cudaMemsetAsync(g->counters + 7, 0, sizeof(unsigned long long), g->stream));
  validate_rowptr_kernel<<<grid_for(g->n + 1, 256), 256, 0, g->stream>>>(
      g->rowptr, g->n, g->nnz, g->err, g->counters + 7);
  MC_CUDA_TRY(cudaGetLastError());
  MC_CUDA_TRY(cudaMemcpyAsync(g->h_err, g->err, sizeof(unsigned), cudaMemcpyDeviceToHost, g->stream));
  MC_CUDA_TRY(cudaMemcpyAsync(g->h_counters + 7, g->counters + 7, sizeof(unsigned long long),
                              cudaMemcpyDeviceToHost, g->stream));
  MC_CUDA_TRY(cudaStreamSynchronize(g->stream));
  if (*g->h_err) return MC_ERR_FORMAT;  // the entry walk needs monotone offsets
  g->max_degree = (int64_t)g->h_counters[7];
  const int64_t tiles = (g->nnz + kTileEdges - 1) / kTileEdges;
  g->launches += 1 + (tiles > 0 ? 1 : 0);
  if (tiles > 0) {
    dag_keep_kernel<false, true><<<(unsigned)tiles, kTileThreads, 0, g->stream>>>(
        g->rowptr, ColumnChunk{g->col, 0, 0}, nullptr, g->n, g->nnz, nullptr, nullptr, nullptr,
        nullptr, (flags & MC_VALIDATE_SYMMETRY) ? 1 : 0, g->err, nullptr);
    MC_CUDA_TRY(cudaGetLastError());
  }
  MC_CUDA_TRY(cudaMemcpyAsync(g->h_err, g->err, sizeof(unsigned), cudaMemcpyDeviceToHost, g->stream));
  MC_CUDA_TRY(cudaStreamSynchronize(g->stream));
  return *g->h_err ? MC_ERR_FORMAT : MC_OK;
}

int validate_rowptr(mc_dgraph *g) {
  MC_CUDA_TRY(cudaMemsetAsync(g->err, 0, sizeof(unsigned), g->stream));
  MC_CUDA_TRY(cudaMemsetAsync(g->counters + 7, 0, sizeof(unsigned long long), g->stream));
  validate_rowptr_kernel<<<grid_for(g->n + 1, 256), 256, 0, g->stream>>>(
      g->rowptr, g->n, g->nnz, g->err, g->counters + 7);
  MC_CUDA_TRY(cudaGetLastError());
  g->launches += 1;
  MC_CUDA_TRY(cudaMemcpyAsync(g->h_err, g->err, sizeof(unsigned), cudaMemcpyDeviceToHost, g->stream));
  MC_CUDA_TRY(cudaMemcpyAsync(g->h_counters + 7, g->counters + 7, sizeof(unsigned long long),
                              cudaMemcpyDeviceToHost, g->stream));
  MC_CUDA_TRY(cudaStreamSynchronize(g->stream));
  if (*g->h_err) return MC_ERR_FORMAT;
  g->max_degree = (int64_t)g->h_counters[7];
  return MC_OK;
}

int validate_csr_words(const int64_t *rowptr, const int32_t *col, int64_t n, int64_t nnz,
                       unsigned *d_err, unsigned long long *d_max_deg, cudaStream_t s,
                       int64_t *max_degree) {
  unsigned h_err = 0;
  unsigned long long h_max = 0;
  MC_CUDA_TRY(cudaMemsetAsync(d_err, 0, sizeof(unsigned), s));
  MC_CUDA_TRY(cudaMemsetAsync(d_max_deg, 0, sizeof(unsigned long long), s));
  validate_rowptr_kernel<<<grid_for(n + 1, 256), 256, 0, s>>>(rowptr, n, nnz, d_err, d_max_deg);
  MC_CUDA_TRY(cudaGetLastError());
  MC_CUDA_TRY(cudaMemcpyAsync(&h_err, d_err, sizeof(h_err), cudaMemcpyDeviceToHost, s));
  MC_CUDA_TRY(cudaMemcpyAsync(&h_max, d_max_deg, sizeof(h_max), cudaMemcpyDeviceToHost, s));
  MC_CUDA_TRY(cudaStreamSynchronize(s));
  if (h_err) return MC_ERR_FORMAT;  // the entry walk needs monotone offsets
  const int64_t tiles = (nnz + kTileEdges - 1) / kTileEdges;
  if (tiles > 0) {
    dag_keep_kernel<false, true><<<(unsigned)tiles, kTileThreads, 0, s>>>(
        rowptr, ColumnChunk{col, 0, 0}, nullptr, n, nnz, nullptr, nullptr, nullptr, nullptr, 0, d_err,
        nullptr);
    MC_CUDA_TRY(cudaGetLastError());
    MC_CUDA_TRY(cudaMemcpyAsync(&h_err, d_err, sizeof(h_err), cudaMemcpyDeviceToHost, s));
    MC_CUDA_TRY(cudaStreamSynchronize(s));
  }
  *max_degree = (int64_t)h_max;
  return h_err ? MC_ERR_FORMAT : MC_OK;
}

namespace {
// DAG capacity: every entry in device memory; with host columns the exact
// m+ = nnz / 2 of a symmetric simple graph (tc_orient refuses more).
int64_t dag_capacity(int64_t nnz, bool col_host) {
  return col_host ? nnz / 2 + 1 : std::max<int64_t>(nnz, 1);
}
}  // namespace

// Column entries per chunk: with host columns (two staging buffers) 64 MB; of
// a streamed upload 16 MB, so that the copy starts early and the passes over
// the last chunk, which nothing overlaps, are short (pageable arrays at RMAT
// scale 20, 126 MB: 7.08, 6.20, 5.95, 6.03 and 7.17 ms per call with 64, 32, 16,
// 8 and 4 MB).  Or MERCURY_STAGE_EDGES rounded down to whole tiles (tests use it to run
// many chunks on small graphs).
int64_t stage_capacity(int64_t nnz, bool col_host) {
  int64_t stage = col_host ? 1ll << 24 : 1ll << 22;
  if (const char *env = std::getenv("MERCURY_STAGE_EDGES")) {
    const long long v = std::atoll(env);
    if (v > 0) stage = std::max<int64_t>(kTileEdges, v / kTileEdges * kTileEdges);
  }
  return std::min(stage, std::max<int64_t>((nnz + kTileEdges - 1) / kTileEdges, 1) * kTileEdges);
}

// Ranks with core bitmaps: kCoreRanks, on small graphs a sixteenth of the
// vertices (clearing 67 MB of bitmaps and filling them cost more than the hub
// kernel gained there: 521 -> 499 us per count at RMAT scale 16, 0.944 -> 0.933
// ms at 18), and one per 512 entries where those are more: dense graphs live on
// them (hub kernel, n / 16 ranks against this, ms: complete graph of 2,500 vertices
// 1.57 / 0.42; random ones of 5,000 with 30%, of 8,000 with 10% and of 20,000 with
// 7.7% of all edges 1.44 / 0.45, 0.75 / 0.37 and, with 8,192 ranks, 3.9 / 2.3).  Or
// MERCURY_TC_CORE_RANKS (0 turns them off; tests move the boundary with it), at
// most n.
int core_rank_count(int64_t n, int64_t nnz) {
  int64_t k = std::min<int64_t>(kCoreRanks, std::max<int64_t>(n / 16, nnz / 512));
  if (const char *env = std::getenv("MERCURY_TC_CORE_RANKS")) {
    const long long v = std::atoll(env);
    if (v >= 0) k = std::min<long long>(v, 1 << 18);
  }
  return (int)std::min<int64_t>(k, n);
}

int64_t tc_device_bytes(int64_t n, int64_t nnz, bool col_host, bool dag_host) {
  const int64_t cap = std::max<int64_t>(nnz, 1);
  const int64_t tiles = std::max<int64_t>((nnz + kTileEdges - 1) / kTileEdges, 1);
  const int64_t tasks = n + cap / std::min(kHubChunk, kLeafChunk) + 1;
  const int64_t scan = (int64_t)scan_temp_bytes(tiles + 1);
  const int64_t staging =
      col_host ? 2 * 4 * stage_capacity(nnz, true) + 8 * (stage_capacity(nnz, true) / kTileEdges + 1) : 0;
  return (n + 1) * (8 + 16 + 8 + 4 + 4 + 16) + n / 8 + 3 * 8 * tasks +
         (dag_host ? 0 : 2 * 4 * (dag_capacity(nnz, col_host) + 4)) +
         tiles * (2 * kTileThreads + 28) +
         (int64_t)radix_work_bytes(n, 32) + scan + staging + 4 * core_offset(core_rank_count(n, nnz));
}

int tc_alloc(mc_dgraph *g) {
  if (g->tc_ready) return MC_OK;
  const int64_t n = g->n, cap = std::max<int64_t>(g->nnz, 1);
  const int64_t tiles = std::max<int64_t>((g->nnz + kTileEdges - 1) / kTileEdges, 1);
  g->dag_cap = dag_capacity(g->nnz, g->col_host);
  // Each owner contributes ceil(deg / chunk) <= 1 + deg / chunk tasks.
  g->task_capacity = n + cap / std::min(kHubChunk, kLeafChunk) + 1;
  g->scan_temp_size = scan_temp_bytes(tiles + 1);
  const bool ranked = g->batch.gid == nullptr;
#define MC_ALLOC(ptr, count) \
  MC_CUDA_TRY(dev_alloc((void **)&(ptr), sizeof(*(ptr)) * (size_t)(count), g->stream))
  MC_ALLOC(g->key, n + 1);
  MC_ALLOC(g->pinfo, n + 1);
  MC_ALLOC(g->dag_rowptr, n + 1);
  // 4 entries of padding: the staged hub kernel copies whole 16-byte groups.
  // With the DAG on the host, its entries and ranks live in pinned memory
  // that the kernels reach through the device's mapping.
  auto dag_alloc = [&](int32_t **dev, int32_t **host) -> cudaError_t {
    if (!g->dag_host) return dev_alloc((void **)dev, sizeof(int32_t) * (size_t)(g->dag_cap + 4), g->stream);
    cudaError_t e = cudaHostAlloc((void **)host, sizeof(int32_t) * (size_t)(g->dag_cap + 4),
                                  cudaHostAllocMapped);
    if (e != cudaSuccess) return e;
    return cudaHostGetDevicePointer((void **)dev, *host, 0);
  };
  MC_CUDA_TRY(dag_alloc(&g->dag_col, &g->dag_col_h));
  MC_ALLOC(g->keep, tiles * kTileWords);
  MC_ALLOC(g->tile_counts, tiles);
  MC_ALLOC(g->tile_offsets, tiles + 1);
  MC_ALLOC(g->tile_rows, 2 * tiles);
  MC_ALLOC(g->deg, n + 1);
  MC_ALLOC(g->list_len, 4);
  MC_ALLOC(g->task_status, n / kTaskThreads + 4);  // at least 3 per block of 1,024, and a ticket
  MC_ALLOC(g->hub_tasks, g->task_capacity);
  MC_ALLOC(g->leaf_tasks, g->task_capacity);
  MC_ALLOC(g->mega_tasks, g->task_capacity);
  if (ranked) {
    MC_ALLOC(g->rank, n + 1);
    MC_CUDA_TRY(dag_alloc(&g->dag_rank, &g->dag_rank_h));
    MC_ALLOC(g->rank_keys, 2 * n + 2);
    MC_CUDA_TRY(dev_alloc(&g->rank_work, radix_work_bytes(n, 32), g->stream));
    g->core_ranks = core_rank_count(n, g->nnz);
    if (g->core_ranks > 0) MC_ALLOC(g->core_bits, core_offset(g->core_ranks));
  }
  // Chunked column passes (host columns, or a streamed upload of a single
  // graph): the copy stream, its events and one chunk's tile offsets.
  if (ranked) {
    g->chunk_edges = stage_capacity(g->nnz, g->col_host);
    MC_ALLOC(g->chunk_offsets, g->chunk_edges / kTileEdges + 1);
    MC_CUDA_TRY(cudaStreamCreateWithFlags(&g->copy_stream, cudaStreamNonBlocking));
    for (cudaEvent_t &e : g->stage_ev)
      MC_CUDA_TRY(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  }
  if (g->col_host && ranked) {
    g->stage_edges = g->chunk_edges;
    MC_ALLOC(g->stage, 2 * g->stage_edges);
  }
  MC_CUDA_TRY(dev_alloc(&g->scan_temp, g->scan_temp_size, g->stream));
#undef MC_ALLOC
  g->tc_ready = true;
  return MC_OK;
}

// Host copy of count entries by all host threads, in 1 MB pieces.
static void parallel_copy(int32_t *dst, const int32_t *src, int64_t count) {
  constexpr int64_t kPiece = 1 << 18;
  const int64_t pieces = (count + kPiece - 1) / kPiece;
#pragma omp parallel for schedule(static)
  for (int64_t p = 0; p < pieces; ++p) {
    const int64_t a = p * kPiece, b = std::min(count, a + kPiece);
    std::memcpy(dst + a, src + a, sizeof(int32_t) * (size_t)(b - a));
  }
}

// Passes A and B over a column array that crosses from host memory in
// chunks of whole tiles, copied by DMA on a copy stream while the passes run
// on the previous chunk.  Each chunk runs A, the scan of its tile counts on
// top of the earlier chunks' total, and B, so no pass waits for the whole
// array.  Two forms:
//  * host columns (in_place false): chunks go to two staging buffers; the
//    columns were validated when the handle was made;
//  * streamed upload (in_place true): chunks land in the handle's own device
//    column array, and pass A checks each chunk against the contract on the
//    way (no gather with an id out of range); once a check has failed, the
//    later passes do nothing.
// The DAG holds dag_cap entries; a chunk that would end past it raises
// kErrDagCapacity and writes nothing.  The caller reads the flags before
// counting.
static int staged_dag_passes(mc_dgraph *g, const int32_t *deg, const int32_t *src, bool in_place) {
  const int64_t n = g->n, nnz = g->nnz;
  cudaStream_t s = g->stream, cs = g->copy_stream;
  cudaEvent_t *copied = g->stage_ev, *drained = g->stage_ev + 2;
  const int64_t chunk = in_place ? g->chunk_edges : g->stage_edges;
  const unsigned *stop = in_place ? g->err : nullptr;
  // A streamed upload from pageable memory goes through the pinned slots when
  // the caller provided them (the driver's own pageable copies are slower).
  bool pageable = false;
  if (in_place && g->pin_slot[0] && g->pin_slot[1] && g->pin_entries >= chunk) {
    cudaPointerAttributes attr{};
    if (cudaPointerGetAttributes(&attr, src) == cudaSuccess)
      pageable = attr.type == cudaMemoryTypeUnregistered;
    else
      cudaGetLastError();  // an unknown pointer: plain copies
  }
  MC_CUDA_TRY(cudaMemsetAsync(g->tile_offsets, 0, sizeof(int64_t), s));
  // Copies start after the work already queued on the handle's stream.
  MC_CUDA_TRY(cudaEventRecord(drained[0], s));
  MC_CUDA_TRY(cudaStreamWaitEvent(cs, drained[0], 0));
  const int64_t chunks = (nnz + chunk - 1) / chunk;
  for (int64_t c = 0; c < chunks; ++c) {
    const int slot = (int)(c & 1);
    const int64_t e0 = c * chunk, e1 = std::min(nnz, e0 + chunk);
    const int64_t tb = e0 / kTileEdges, ct = (e1 - e0 + kTileEdges - 1) / kTileEdges;
    int32_t *buf = in_place ? g->col + e0 : g->stage + (int64_t)slot * g->stage_edges;
    if (!in_place && c >= 2) MC_CUDA_TRY(cudaStreamWaitEvent(cs, drained[slot], 0));
    if (pageable) {
      // The host threads copy the chunk into a pinned slot (free once its
      // previous copy to the device is done), then the DMA engine takes it,
      // while the threads fill the other slot.
      if (c >= 2) MC_CUDA_TRY(cudaEventSynchronize(g->pin_done[slot]));
      parallel_copy(g->pin_slot[slot], src + e0, e1 - e0);
      MC_CUDA_TRY(cudaMemcpyAsync(buf, g->pin_slot[slot], sizeof(int32_t) * (size_t)(e1 - e0),
                                  cudaMemcpyHostToDevice, cs));
      MC_CUDA_TRY(cudaEventRecord(g->pin_done[slot], cs));
    } else {
      MC_CUDA_TRY(cudaMemcpyAsync(buf, src + e0, sizeof(int32_t) * (size_t)(e1 - e0),
                                  cudaMemcpyHostToDevice, cs));
    }
    MC_CUDA_TRY(cudaEventRecord(copied[slot], cs));
    MC_CUDA_TRY(cudaStreamWaitEvent(s, copied[slot], 0));
    const ColumnChunk cc = in_place ? ColumnChunk{g->col, 0, tb} : ColumnChunk{buf, e0, tb};
    (in_place ? dag_keep_kernel<true, true> : dag_keep_kernel<true, false>)
        <<<(unsigned)ct, kTileThreads, 0, s>>>(g->rowptr, cc, deg, n, nnz, g->key, g->keep,
                                               g->tile_counts, stop, 0, g->err, g->tile_rows);
    MC_CUDA_TRY(cudaGetLastError());
    MC_CUDA_TRY(exclusive_scan(g->tile_counts + tb, g->chunk_offsets, ct, g->scan_temp, s));
    chunk_offsets_kernel<<<grid_for(ct + 1, 256), 256, 0, s>>>(g->chunk_offsets, ct,
                                                               g->tile_offsets + tb, g->dag_cap,
                                                               g->err);
    MC_CUDA_TRY(cudaGetLastError());
    dag_write_kernel<<<(unsigned)ct, kTileThreads, 0, s>>>(
        g->rowptr, cc, n, nnz, g->keep, g->tile_offsets, g->dag_rowptr, g->dag_col,
        g->ranked ? g->rank : nullptr, g->ranked ? g->dag_rank : nullptr, g->tile_offsets + tb + ct,
        g->dag_cap, stop, g->tile_rows);
    MC_CUDA_TRY(cudaGetLastError());
    MC_CUDA_TRY(cudaEventRecord(drained[slot], s));
    g->launches += 3 + scan_launches(ct);
  }
  return MC_OK;
}

int tc_orient(mc_dgraph *g, const int32_t *upload) {
  NvtxRange range("tc_orient");
  const int64_t n = g->n, nnz = g->nnz;
  cudaStream_t s = g->stream;
  MC_CUDA_TRY(cudaMemsetAsync(g->counters, 0, sizeof(unsigned long long) * 7, s));
  g->core_used = 0;
  g->dag_built = false;
  if (n == 0) return MC_OK;
  const int64_t tiles = (nnz + kTileEdges - 1) / kTileEdges;
  // The degrees alone, for pass A's gathers.
  int32_t *deg = g->deg;
  // d+(v)^2 <= nnz (v's out-neighbours have at least its degree), so without
  // room for a hub owner nothing reads the ranks.
  g->max_out_bound = std::min<int64_t>(g->max_degree, (int64_t)std::sqrt((double)nnz) + 1);
  const bool ranked = g->rank && !g->batch.gid && g->max_out_bound > kLeafMaxOut;
  g->ranked = ranked;
  const int64_t task_blocks = (n + kTaskThreads * kTaskItems - 1) / (kTaskThreads * kTaskItems);
  init_key_kernel<<<grid_for(n + 4, 256), 256, 0, s>>>(g->rowptr, n, g->key, deg, g->task_status,
                                                       3 * task_blocks + 1, g->list_len + 3, g->err);
  MC_CUDA_TRY(cudaGetLastError());
  g->launches += 1;
  if (ranked) {
    // Degree ranks (the hub kernel's bitmaps are indexed by them).
    rank_keys_kernel<<<grid_for(n, 256), 256, 0, s>>>(g->key, n, (int)g->max_degree, g->rank_keys);
    MC_CUDA_TRY(cudaGetLastError());
    unsigned long long *sorted = nullptr;
    MC_CUDA_TRY(radix_sort_u64(g->rank_keys, g->rank_keys + n, n, 32,
                               32 + bit_width((uint64_t)g->max_degree), g->rank_work, g->err, s,
                               &sorted, &g->launches));
    rank_scatter_kernel<<<grid_for(n, 256), 256, 0, s>>>(sorted, n, g->rank);
    MC_CUDA_TRY(cudaGetLastError());
    g->rank_sorted = sorted;
    g->launches += 2;
  }
  if (tiles > 0) {
    tile_rows_kernel<<<grid_for(n, 256), 256, 0, s>>>(g->rowptr, n, nnz, tiles, g->tile_rows);
    MC_CUDA_TRY(cudaGetLastError());
    g->launches += 1;
  }
  if (tiles == 0) {
    MC_CUDA_TRY(cudaMemsetAsync(g->dag_rowptr, 0, sizeof(int64_t) * (n + 1), s));
  } else if (upload) {
    // A streamed upload needs the chunk machinery of a single-graph handle.
    if (!g->copy_stream || !g->chunk_offsets || g->chunk_edges <= 0) return MC_ERR_ARG;
    const int rc = staged_dag_passes(g, deg, upload, true);
    if (rc != MC_OK) return rc;
  } else if (g->col_host) {
    if (!g->copy_stream || !g->stage || g->stage_edges <= 0) return MC_ERR_ARG;
    const int rc = staged_dag_passes(g, deg, g->col_h, false);
    if (rc != MC_OK) return rc;
  } else {
    const unsigned grid = (unsigned)tiles;
    const ColumnChunk all{g->col, 0, 0};
    dag_keep_kernel<true, false><<<grid, kTileThreads, 0, s>>>(
        g->rowptr, all, deg, n, nnz, g->key, g->keep, g->tile_counts, nullptr, 0, g->err,
        g->tile_rows);
    MC_CUDA_TRY(cudaGetLastError());
    MC_CUDA_TRY(exclusive_scan(g->tile_counts, g->tile_offsets, tiles, g->scan_temp, s));
    dag_write_kernel<<<grid, kTileThreads, 0, s>>>(
        g->rowptr, all, n, nnz, g->keep, g->tile_offsets, g->dag_rowptr, g->dag_col,
        ranked ? g->rank : nullptr, ranked ? g->dag_rank : nullptr, nullptr, 0, nullptr,
        g->tile_rows);
    MC_CUDA_TRY(cudaGetLastError());
    g->launches += 2 + scan_launches(tiles);
  }
  // A handle reused for a smaller graph keeps its capacity: only the ranks
  // of this graph get core bitmaps.
  if (g->core_bits && ranked) {
    g->core_used = std::min(g->core_ranks, core_rank_count(n, nnz));
    MC_CUDA_TRY(cudaMemsetAsync(g->core_bits, 0, sizeof(unsigned) * core_offset(g->core_used), s));
    core_bits_kernel<<<grid_for((int64_t)g->core_used * kWarp, 256), 256, 0, s>>>(
        g->rank_sorted, n, g->core_used, g->dag_rowptr, g->dag_rank, g->core_bits, g->err);
    MC_CUDA_TRY(cudaGetLastError());
    g->launches += 1;
  }
  partner_tasks_kernel<<<(unsigned)task_blocks, kTaskThreads, 0, s>>>(
      g->key, ranked ? g->rank : nullptr, g->dag_rowptr, n, g->pinfo,
      TaskLists{g->list_len, g->list_len + 1, g->list_len + 2, g->list_len + 3, g->hub_tasks, g->leaf_tasks,
                g->mega_tasks, g->task_status, task_blocks},
      g->counters + 3, g->batch, wait_polls(), g->err);
  MC_CUDA_TRY(cudaGetLastError());
  g->launches += 1;
  return MC_OK;
}

int tc_partner_stats(mc_dgraph *g, unsigned long long *partner_edges, unsigned long long *work) {
  *partner_edges = *work = 0;
  if (!g->tc_ready || g->n == 0) return MC_OK;
  MC_CUDA_TRY(cudaMemsetAsync(g->counters + 4, 0, sizeof(unsigned long long) * 2, g->stream));
  partner_stats_kernel<<<g->num_sms * 8, 256, 0, g->stream>>>(g->rowptr, g->col, g->key, g->n,
                                                              g->counters + 4);
  MC_CUDA_TRY(cudaGetLastError());
  unsigned long long c[2];
  MC_CUDA_TRY(cudaMemcpyAsync(c, g->counters + 4, sizeof(c), cudaMemcpyDeviceToHost, g->stream));
  MC_CUDA_TRY(cudaStreamSynchronize(g->stream));
  *partner_edges = c[0];
  *work = c[1];
  return MC_OK;
}

}  // namespace mc
