// P1..P8 from non-induced motif sums: the default route of whole counts.
//
// Reference: subgraph_matching/pattern_kernels.cuh (P1..P8) and the combine of
// subgraph_matching/sm_multigpu.cu:206-232.  While no 32-bit product of those
// formulas can wrap (maximum degree at most 46,340), each is a fixed multiple
// of induced subgraph counts (claws, forks, K1,4, 4-paths, bulls, paws, darts,
// K1,1,3, tailed K4).  An induced count is a signed sum of non-induced ones
// over the graphs that contain the pattern on the same vertices, and every
// non-induced count needed is a sum over vertices, edges, triangles, or pairs
// at distance two of small polynomials in
//   d   degrees,
//   a   triangles on an edge,
//   k   common neighbours of a triangle's three vertices,
//   c   common neighbours of a vertex pair,
// plus the numbers of K4, K5, 4-cycles (C4), 4-wheels (W4) and of K2,3 with
// one edge in its side of three (X7).  So nothing is enumerated beyond
// triangles and two-paths, where the per-edge formulas test every pair of an
// edge's neighbours.
//
// What bounds it: latency of dependent gathers (row offsets, then columns,
// then per-edge words) and, on small graphs, the launches.  On the Chung-Lu
// graph of 100,000 vertices (mean 10, cap 200: m = 498,340, 84 k triangles,
// 429 k triangle pairs on an edge, 81 M two-paths) the per-edge formulas
// took P1..P8 1.9, 28.0, 9.7, 4.8, 11.1, 3.6, 0.95 and 3.6 ms per call on a
// B200, and these sums take 0.28, 1.37, 0.39, 0.76, 1.25, 0.38, 0.31 and 0.31.
// On the one of 60,000 (mean 20, cap 50,000, a hub of degree 17,215) P1, P4,
// P7 and P8 took 74.7, 276, 25.9 and 26.1 ms, and take 0.82, 1.66, 1.3 and 1.3.
// There the pairs of P2 and P5 take 0.24 s (544 M two-paths).
//
// Stages (each vertex pair ordered by (degree, id), written u < v below; an
// "up" entry of the CSR is one with u < v):
//   rows    entry -> row, degrees
//   up      N+(u): the up entries of each row, compacted in place; the
//           reverse entry of each edge; room for the edge's two lists below
//   tri     every pair (x, y) of N+(u) tested once in the row of the lower of
//           the two (sum of C(d+, 2) searches): a of each entry, and per entry
//           (u -> v) a list of the entries (u -> w) of its common neighbours
//           w, slot j of (u -> v) and slot j of (v -> u) holding the same w
//   tau     edge sums; per u, bit rows of its up neighbours over N(u) and over N+(u):
//           k is a popcount of two rows, K4 and K5 of two and three
//   pairs   common neighbours c of pairs (s, t), counted per s in a table
//           over t: C4, K2,3, X7
//   wheel   4-cycles inside N(v), counted per (v, x) in a table over N(v)
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>

#include "device_common.cuh"
#include "dgraph.cuh"
#include "motifs.cuh"
#include "slices.cuh"

namespace mc {
namespace {

// Words of MotifArgs::counts: list lengths, then queue positions.
enum Count : int {
  kTauN, kMidN, kHashN, kHugeN, kBigN, kSplitN, kTauQueue, kMidQueue, kHashQueue, kUnused,
  kBigQueue,                   // 64 bits each: run_slices clears them
  kWheelQueue = kBigQueue + 2,
  kCounts = kWheelQueue + 2
};

struct MotifArgs {
  const int64_t *__restrict__ rp;
  const int32_t *__restrict__ ci;
  int n, nnz;
  int pattern;
  unsigned need;
  int32_t *deg;    // n
  int32_t *dp;     // n: |N+(v)|
  int32_t *tv2;    // n: twice the triangles of v
  u64 *d2;         // n: sum of (d - 1) over N(v)
  u64 *walk;       // n: table entries the pairs stage visits for s = v
  int32_t *src;    // nnz: row of an entry
  int32_t *upe;    // nnz: rp[u] + i -> i-th up entry of u
  int32_t *pos1;   // nnz: 1 + position in N+(row) of an up entry, else 0
  int32_t *rev1;   // nnz: 1 + reverse entry, 0 if there is none
  int32_t *a;      // nnz: triangles on the entry's edge = length of its list
  int32_t *cnt;    // nnz: the same at the up entry, counted ahead (null: not)
  int64_t *off;    // nnz: list offsets
  int32_t *list;   // common-neighbour lists
  int64_t list_cap;
  u64 *pool;       // list entries handed out (above list_cap: all later stages stop)
  u64 *probe;      // two-paths sampled, and the closed ones among them
  int probe_percent;  // closed from here on: every stage stops (0: no samples)
  bool early;      // motif_outweighs is asked before the tau stage
  u64 *acc;        // kSums
  // Vertices too large for one warp.  pair_mid: the two hash classes, from the
  // front and from the back of its n entries; pair_big: tables over all
  // vertices, the longest walks from the front, so that they start first.
  int32_t *tau_big, *pair_mid, *pair_big;
  unsigned *counts;  // see Count
  // Parts of the longest walks (ordered), or those walks themselves (all pairs):
  // split_cap entries (s, part, parts) at most (0:
  // none); num_sms and the sum of walk place the line.
  int4 *split;
  int split_cap, num_sms;
  u64 *walk_total;
  u64 warp_walk, mid_walk;  // where the warp class and pair_mid's front class end
  unsigned *slices;  // bit rows of the tau stage that exceed shared memory
  int64_t slice_words;
};

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / kWarp;
constexpr int kTauOut = 32;       // warp form of the tau stage: d+ and d at most
constexpr int kTauDeg = 512;
constexpr int kTauSmem = 96 << 10;  // bit rows of a CTA, two CTAs per SM
constexpr int kTauBoth = 8 << 10;   // up to here the two forms share a launch
// Classes of the pairs stage by table entries visited (a vertex's walk bounds
// the keys of its table, which has at least twice as many slots): a warp, a
// CTA of 128 and of 512 threads with a hash table, and a CTA of 1,024 with a
// counter for every vertex.  With warps and 1,024-thread CTAs alone the stage
// took 6.2 ms in P2 on the graph of 100,000 (one CTA per SM, three barriers
// per vertex of some 1,000 entries); with the four classes it takes 1.1 ms.
constexpr u64 kWarpWalk = 512, kMidWalk = 2048, kHashWalk = 8192;
constexpr u64 kHugeWalk = 1 << 15;
// Ordered walks above this, and above an SM's share of all of them, go in parts
// of the table's range, a CTA each: a CTA alone with the largest (677 k entries
// of 27.7 M on the Chung-Lu graph of 60,000 vertices, cap 50,000) lasted 1.5 ms
// of P4's 2.6 ms, which takes 1.66 so; 100,000 vertices of mean 60: 17.7 -> 14.5
// ms.  Counters in L2 that all warps share were slower there (25.3 ms: atomics
// on one address), and the sum of the walks by an atomic per warp of the up
// stage cost 0.04 ms at 1 M entries.
constexpr u64 kSplitWalk = 1 << 16;
constexpr int kSplitMax = 1024;
// Of all pairs, the walks of vertices above this degree (whose X7 outlasts any walk)
// stand in front and run in the first slice, beside one another: in the order of
// their arrival, slices of 250 ms waited for one hub each (P5 at n = 500,000, cap
// 50,000: 6.5 to 7.1 s against 6.0 in one launch).
constexpr int kGiantDegree = 1024;
constexpr u64 kFewWalk = 64;
constexpr int kFewVertices = 16384;
constexpr int kHashSlots = 1024;  // of a warp
constexpr int kWheelDeg = 512;    // warp form of the wheel stage
constexpr int kWheelClaim = 32;   // entries a CTA claims at once in the other
constexpr int kProbeBlocks = 4;   // samples: a thread each
constexpr int kEarlyOut = 400;    // bound on d+ above which a^2 is summed before tau (7 us at 1 M entries)

// (degree, id) order.
__device__ __forceinline__ bool lower(int du, int u, int dv, int v) {
  return du < dv || (du == dv && u < v);
}

// Index of x in the ascending ci[b, e), or -1.
__device__ __forceinline__ int find_entry(const int32_t *__restrict__ ci, int b, int e, int x) {
  while (b < e) {
    const int mid = (b + e) >> 1;
    const int y = __ldg(ci + mid);
    if (y == x) return mid;
    if (y < x) b = mid + 1;
    else e = mid;
  }
  return -1;
}

// The warp's 32 lists laid end to end: flat position f belongs to list l (the
// first whose inclusive end exceeds f) at offset f - excl(l).
struct FlatLists {
  int incl, total;
  __device__ __forceinline__ FlatLists(int len, int lane) {  // every lane calls it
    incl = warp_inclusive_scan(len, lane);
    total = __shfl_sync(kFull, incl, kWarp - 1);
  }
  // Every lane calls it; positions past the end give list 31.
  __device__ __forceinline__ int owner(int f) const {
    int l = 0;
#pragma unroll
    for (int step = 16; step > 0; step >>= 1)
      if (__shfl_sync(kFull, incl, l + step - 1) <= f) l += step;
    return min(l, kWarp - 1);
  }
};

// Calls f(entry, owner lane, place) for the entries of this warp's 32 lists
// [lo, lo + len) of a.list, flat.
template <class F>
__device__ __forceinline__ void walk_lists(const MotifArgs &a, int64_t lo, int len, int lane, F f) {
  const FlatLists fl(len, lane);
  const int64_t start = lo - (fl.incl - len);
  for (int base = 0; base < fl.total; base += kWarp) {
    const int g = base + lane;
    const int l = fl.owner(g);
    const int64_t at = __shfl_sync(kFull, start, l) + g;
    if (g < fl.total) f(a.list[at], l, at);
  }
}

// The lanes of a warp that hold entries of the same row u (rows in order): from
// the last row head at or below this lane to the one before the next head.
struct RowLanes {
  int first;
  unsigned mask;
  __device__ __forceinline__ RowLanes(int u, int lane) {  // every lane calls it
    const int prev = __shfl_up_sync(kFull, u, 1);
    const unsigned heads = __ballot_sync(kFull, lane == 0 || u != prev);
    const unsigned upto = kFull >> (kWarp - 1 - lane);
    const unsigned later = heads & ~upto;
    first = kWarp - 1 - __clz(heads & upto);
    mask = (later ? (1u << (__ffs(later) - 1)) - 1u : kFull) & (kFull << first);
  }
};

__device__ __forceinline__ bool lists_overrun(const MotifArgs &a) {
  return *a.pool > (u64)a.list_cap;
}
constexpr u64 kClosed = ~0ull;  // in *pool: the samples sent the count elsewhere

// The stages that a^2 drives: not for lists that overran, nor where the formulas
// are the shorter way.
__device__ __forceinline__ bool stops_here(const MotifArgs &a) {
  return lists_overrun(a) || ((a.need & kNeedWork) && motif_outweighs(a.pattern, a.acc));
}

// Offsets of the lists of this lane's up entry e and its reverse, `len` entries
// each (0: none); one atomic per warp.
__device__ __forceinline__ void take_lists(const MotifArgs &a, int e, int r, int len, int lane) {
  u64 incl = 2 * (u64)len;
#pragma unroll
  for (int o = 1; o < kWarp; o <<= 1) {
    const u64 x = __shfl_up_sync(kFull, incl, o);
    if (lane >= o) incl += x;
  }
  u64 base = 0;
  if (lane == kWarp - 1 && incl) base = atomicAdd(a.pool, incl);
  base = __shfl_sync(kFull, base, kWarp - 1);
  if (len > 0) {
    a.off[e] = (int64_t)(base + incl - 2 * (u64)len);
    a.off[r] = (int64_t)(base + incl - (u64)len);
  }
}

// ---- rows, up ---------------------------------------------------------------
// A sample of two-paths u - v - w per thread (from a random entry u -> v on),
// counted, and the closed ones among them.
__device__ void sample_two_paths(const MotifArgs &a, unsigned sample, int lane) {
  u64 r = (u64)(sample + 1) * 0x9e3779b97f4a7c15ull;
  r = (r ^ (r >> 30)) * 0xbf58476d1ce4e5b9ull;
  r ^= r >> 31;
  const int e = (int)((r & 0xffffffffu) % (unsigned)a.nnz);
  const int u = (int)upper_row(a.rp, 0, a.n - 1, e), v = __ldg(a.ci + e);
  const int b = (int)__ldg(a.rp + v), d = (int)__ldg(a.rp + v + 1) - b;
  const int w = d > 0 ? __ldg(a.ci + b + (int)((unsigned)(r >> 32) % (unsigned)d)) : u;
  const bool path = w != u;
  const bool closed =
      path && find_entry(a.ci, (int)__ldg(a.rp + u), (int)__ldg(a.rp + u + 1), w) >= 0;
  const unsigned paths = __ballot_sync(kFull, path), hits = __ballot_sync(kFull, closed);
  if (lane == 0) {
    if (paths) atomicAdd(a.probe, (u64)__popc(paths));
    if (hits) atomicAdd(a.probe + 1, (u64)__popc(hits));
  }
}

// Warp per row: src, deg, and the sums of degrees alone.  The blocks from
// row_blocks on take the samples beside them.
__global__ void __launch_bounds__(kThreads) motif_rows_kernel(MotifArgs a, int row_blocks) {
  __shared__ u64 sm[kSums];
  const BlockSums bs{sm};
  bs.init();
  const int lane = threadIdx.x & (kWarp - 1);
  if ((int)blockIdx.x >= row_blocks) {
    sample_two_paths(a, (blockIdx.x - row_blocks) * kThreads + threadIdx.x, lane);
    return;
  }
  u64 d3 = 0, d4 = 0;
  const int stride = row_blocks * kWarps;
  for (int v = blockIdx.x * kWarps + threadIdx.x / kWarp; v < a.n; v += stride) {
    const int b = (int)__ldg(a.rp + v), e = (int)__ldg(a.rp + v + 1);
    for (int i = b + lane; i < e; i += kWarp) a.src[i] = v;
    if (lane == 0) {
      a.deg[v] = e - b;
      d3 += c3(e - b);
      d4 += c4(e - b);
    }
  }
  bs.add(kVd3, d3);
  bs.add(kVd4, d4);
  bs.flush(a.acc);
}

// Thread per entry.  Up entries are compacted per row with one atomic per
// (row, warp) piece (their order within a row does not matter), and find
// their reverse entry in the longer row.
__global__ void __launch_bounds__(kThreads) motif_up_kernel(MotifArgs a) {
  const int lane = threadIdx.x & (kWarp - 1);
  const int64_t e64 = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  if (a.probe_percent > 0 && a.probe[0] > 0 &&
      100 * a.probe[1] >= (u64)a.probe_percent * a.probe[0]) {
    if (e64 == 0) *a.pool = kClosed;
    return;
  }
  const bool in = e64 < a.nnz;
  const int e = in ? (int)e64 : a.nnz - 1;
  const int u = a.src[e], v = __ldg(a.ci + e);
  const int64_t bu = __ldg(a.rp + u);
  const int du = a.deg[u], dv = a.deg[v];
  int r = -1;
  int bv = 0;
  if (in && lower(du, u, dv, v)) {
    bv = (int)__ldg(a.rp + v);
    r = find_entry(a.ci, bv, bv + dv, u);
  }
  const bool up = r >= 0;
  const unsigned ups = __ballot_sync(kFull, up);
  const RowLanes rl(u, lane);
  const int first = rl.first;
  const unsigned row = rl.mask;
  int base = 0;
  if (lane == first && (ups & row)) base = atomicAdd(a.dp + u, __popc(ups & row));
  base = __shfl_sync(kFull, base, first);
  if (up) {
    const int k = base + __popc(ups & row & ((1u << lane) - 1u));
    a.upe[bu + k] = e;
    a.pos1[e] = k + 1;
    a.rev1[e] = r + 1;
    a.rev1[r] = e + 1;
    if (a.need & kNeedC4) {
      atomicAdd(a.walk + v, (u64)du);  // s = v visits N(u)
    } else if (a.need & kNeedPairs) {
      atomicAdd(a.walk + u, (u64)(r - bv));
      atomicAdd(a.walk + v, (u64)(e - (int)bu));
    }
    if (a.need & kNeedD2) {
      atomicAdd(a.d2 + u, (u64)(dv - 1));
      atomicAdd(a.d2 + v, (u64)(du - 1));
    }
  } else if (in) {
    a.pos1[e] = 0;  // a down entry, or one with no reverse, which the up lists leave out
  }
  // Without counts: u's other neighbours bound the list.
  if (!a.cnt) take_lists(a, e, r, up ? du - 1 : 0, lane);
}

// With counts: exactly sized lists.
__global__ void __launch_bounds__(kThreads) motif_lists_kernel(MotifArgs a) {
  if (*a.pool == kClosed) return;
  const int64_t e64 = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  const int e = (int)(e64 < a.nnz ? e64 : 0);
  const bool up = e64 < a.nnz && a.pos1[e];
  take_lists(a, e, up ? a.rev1[e] - 1 : 0, up ? a.cnt[e] : 0, threadIdx.x & (kWarp - 1));
}

// ---- triangles --------------------------------------------------------------
// A warp takes `per` consecutive slots of the compacted up lists (32, fewer
// on graphs that would leave warps idle: see spread()); slot i of N+(u) pairs
// with the later slots, and the pairs of all of them are walked flat.
// kCount: the list lengths alone.  Otherwise the lists, and the vertices of
// the later stages' classes.
template <bool kCount>
__global__ void __launch_bounds__(kThreads) motif_tri_kernel(MotifArgs a, int per) {
  __shared__ u64 sm[kSums];
  const BlockSums bs{sm};
  bs.init();
  const int lane = threadIdx.x & (kWarp - 1);
  if (!kCount && lists_overrun(a)) return;  // the host makes room and starts over
  const int64_t s64 = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  if (!kCount && a.split_cap > 0 && (a.need & kNeedC4) && s64 - lane < a.n) {
    const u64 w = warp_sum_u64(s64 < a.n ? a.walk[s64] : 0);
    if (lane == 0 && w) atomicAdd(a.walk_total, w);
  }
  if (!kCount && s64 < a.n) {
    const int v = (int)s64;
    const int d = a.deg[v], p = a.dp[v];
    if (p > kTauOut || (p >= 2 && d > kTauDeg)) a.tau_big[atomicAdd(a.counts + kTauN, 1u)] = v;
    if (a.need & (kNeedC4 | kNeedPairs)) {
      const u64 w = a.walk[v];
      unsigned front = kSplitMax;
      if (w > kHashWalk && d > kGiantDegree && a.split_cap > 0 && !(a.need & kNeedC4))
        front = atomicAdd(a.counts + kSplitN, 1u);
      if (front < (unsigned)kSplitMax) a.split[front] = make_int4(v, 0, 1, 0);
      else if (w > kHugeWalk) a.pair_big[atomicAdd(a.counts + kHugeN, 1u)] = v;
      else if (w > kHashWalk) a.pair_big[a.n - 1 - atomicAdd(a.counts + kBigN, 1u)] = v;
      else if (w > a.mid_walk) a.pair_mid[a.n - 1 - atomicAdd(a.counts + kHashN, 1u)] = v;
      else if (w > a.warp_walk) a.pair_mid[atomicAdd(a.counts + kMidN, 1u)] = v;
    }
  }
  int slot = 0, len = 0, e_ux = 0, x = 0, dx = 0, du = 0;
  const int64_t mine = s64 / kWarp * per + lane;
  if (lane < per && mine < a.nnz) {
    slot = (int)mine;
    const int u = a.src[slot];
    const int i = slot - (int)__ldg(a.rp + u), p = a.dp[u];
    if (i < p - 1) {
      len = p - 1 - i;
      e_ux = a.upe[slot];
      x = __ldg(a.ci + e_ux);
      dx = a.deg[x];
      du = a.deg[u];
    }
  }
  const FlatLists fl(len, lane);
  u64 tri = 0, vtd = 0;
  for (int base = 0; base < fl.total; base += kWarp) {
    const int f = base + lane;
    const int l = fl.owner(f);
    const int ys = f + __shfl_sync(kFull, slot + 1 - (fl.incl - len), l);
    const int ex = __shfl_sync(kFull, e_ux, l);
    const int vx = __shfl_sync(kFull, x, l), dvx = __shfl_sync(kFull, dx, l);
    const int dvu = __shfl_sync(kFull, du, l);
    if (f >= fl.total) continue;
    const int ey = a.upe[ys];
    const int y = __ldg(a.ci + ey);
    const int dy = a.deg[y];
    const bool x_low = lower(dvx, vx, dy, y);
    const int lo = x_low ? vx : y, hi = x_low ? y : vx;
    const int b = (int)__ldg(a.rp + lo);
    const int exy = find_entry(a.ci, b, b + (x_low ? dvx : dy), hi);
    if (exy < 0 || a.rev1[exy] == 0) continue;
    if (kCount) {
      atomicAdd(a.cnt + ex, 1);
      atomicAdd(a.cnt + ey, 1);
      atomicAdd(a.cnt + exy, 1);
    } else {
      const int rx = a.rev1[ex] - 1, ry = a.rev1[ey] - 1, rxy = a.rev1[exy] - 1;
      const int jx = atomicAdd(a.a + ex, 1), jy = atomicAdd(a.a + ey, 1),
                jxy = atomicAdd(a.a + exy, 1);
      atomicAdd(a.a + rx, 1);
      atomicAdd(a.a + ry, 1);
      atomicAdd(a.a + rxy, 1);
      a.list[a.off[ex] + jx] = ey;
      a.list[a.off[rx] + jx] = x_low ? exy : rxy;  // x -> y
      a.list[a.off[ey] + jy] = ex;
      a.list[a.off[ry] + jy] = x_low ? rxy : exy;  // y -> x
      a.list[a.off[exy] + jxy] = x_low ? rx : ry;  // lo -> u
      a.list[a.off[rxy] + jxy] = x_low ? ry : rx;  // hi -> u
      vtd += (u64)(dvu + dvx) + (u64)dy;
      ++tri;
    }
  }
  __syncwarp();
  if (!kCount) {
    bs.add(kT, tri);
    bs.add(kVtd, vtd);
    bs.flush(a.acc);
  }
}

// Triangles alone, in three launches (rows, up, pairs) where the DAG's
// orientation takes a dozen: the up neighbours of each row compacted in place
// (upe holds vertices here), then the pairs of motif_tri_kernel, counted.
__global__ void __launch_bounds__(kThreads) tri_up_kernel(MotifArgs a) {
  const int lane = threadIdx.x & (kWarp - 1);
  const int64_t e64 = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  const bool in = e64 < a.nnz;
  const int e = in ? (int)e64 : a.nnz - 1;
  const int u = a.src[e], v = __ldg(a.ci + e);
  const bool up = in && lower(a.deg[u], u, a.deg[v], v);
  const unsigned ups = __ballot_sync(kFull, up);
  const RowLanes rl(u, lane);
  int base = 0;
  if (lane == rl.first && (ups & rl.mask)) base = atomicAdd(a.dp + u, __popc(ups & rl.mask));
  base = __shfl_sync(kFull, base, rl.first);
  if (up) a.upe[__ldg(a.rp + u) + base + __popc(ups & rl.mask & ((1u << lane) - 1u))] = v;
}

__global__ void __launch_bounds__(kThreads) tri_pairs_kernel(MotifArgs a, int per) {
  __shared__ u64 s_total;
  if (threadIdx.x == 0) s_total = 0;
  __syncthreads();
  const int lane = threadIdx.x & (kWarp - 1);
  const int64_t s64 = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  const int64_t mine = s64 / kWarp * per + lane;
  int slot = 0, len = 0, x = 0, dx = 0;
  if (lane < per && mine < a.nnz) {
    slot = (int)mine;
    const int u = a.src[slot];
    const int i = slot - (int)__ldg(a.rp + u), p = a.dp[u];
    if (i < p - 1) {
      len = p - 1 - i;
      x = a.upe[slot];
      dx = a.deg[x];
    }
  }
  const FlatLists fl(len, lane);
  u64 hits = 0;
  for (int base = 0; base < fl.total; base += kWarp) {
    const int f = base + lane;
    const int l = fl.owner(f);
    const int ys = f + __shfl_sync(kFull, slot + 1 - (fl.incl - len), l);
    const int vx = __shfl_sync(kFull, x, l), dvx = __shfl_sync(kFull, dx, l);
    if (f >= fl.total) continue;
    const int y = a.upe[ys];
    const int dy = a.deg[y];
    const bool x_low = lower(dvx, vx, dy, y);
    const int b = (int)__ldg(a.rp + (x_low ? vx : y));
    hits += find_entry(a.ci, b, b + (x_low ? dvx : dy), x_low ? y : vx) >= 0;
  }
  __syncwarp();
  hits = warp_sum_u64(hits);
  if (lane == 0 && hits) atomicAdd(&s_total, hits);
  __syncthreads();
  if (threadIdx.x == 0 && s_total) atomicAdd(a.acc + kT, s_total);
}

// ---- triangles with their common neighbours -----------------------------------
// The sum of a^2 ahead of the tau stage, thread per entry, where a graph's up lists
// may be long: K5 can then take that stage as long as the wheels and X7 take later
// (a complete graph of 512 vertices beside a path, P3: 75 ms of 450 in tau).
__global__ void __launch_bounds__(kThreads) motif_squares_kernel(MotifArgs a) {
  __shared__ u64 sm[kSums];
  const BlockSums bs{sm};
  bs.init();
  if (lists_overrun(a)) return;
  u64 a2 = 0;
  for (int64_t e = (int64_t)blockIdx.x * kThreads + threadIdx.x; e < a.nnz;
       e += (int64_t)gridDim.x * kThreads)
    if (a.pos1[e]) a2 += (u64)a.a[e] * (u64)a.a[e];  // an edge once, at its up entry
  __syncwarp();
  bs.add(kA2, a2);
  bs.flush(a.acc);
}

struct TauSums {
  u64 D = 0, C3 = 0, p4 = 0, fork = 0, dart = 0, vt2 = 0;
  u64 cricket = 0, bull = 0, lolli = 0, kite = 0, gem = 0, kd = 0, ka = 0, kk = 0, K4 = 0, K5 = 0;
  // Up edge (u, v) with t triangles.
  __device__ __forceinline__ void edge(u64 du, u64 dv, u64 t) {
    D += c2(t);
    C3 += c3((long long)t);
    p4 += (du - 1 - t) * (dv - 1 - t);
    fork += c2(du - 1) * (dv - 1) + c2(dv - 1) * (du - 1) - t * (du + dv - 4);
    dart += c2(t) * (du + dv - 6);
  }
  __device__ __forceinline__ void flush(const BlockSums &bs, bool tau) const {
    bs.add(kD, D);
    bs.add(kC3, C3);
    bs.add(kEp4, p4);
    bs.add(kEfork, fork);
    bs.add(kEdart, dart);
    bs.add(kVt2, vt2);
    if (tau) {
      bs.add(kCricket, cricket);
      bs.add(kBull, bull);
      bs.add(kLolli, lolli);
      bs.add(kKite, kite);
      bs.add(kGem, gem);
      bs.add(kKd, kd);
      bs.add(kKa, ka);
      bs.add(kKk, kk);
    }
    bs.add(kK4, K4);
    bs.add(kK5, K5);
  }
};

// Triangle (u, x, y): degrees, triangles on its edges, k common neighbours.
__device__ __forceinline__ void tau_terms(const MotifArgs &a, TauSums &t, int u, int x, int y,
                                          long long du, long long aux, long long auy,
                                          long long axy, long long k) {
  const long long dx = a.deg[x], dy = a.deg[y];
  const long long sd = du + dx + dy, sa = aux + auy + axy;
  t.cricket += c2((u64)(du - 2)) + c2((u64)(dx - 2)) + c2((u64)(dy - 2));
  t.bull += (u64)((du - 2) * (dx - 2) + (du - 2) * (dy - 2) + (dx - 2) * (dy - 2) - sa + 3);
  if (a.need & kNeedD2)
    t.lolli += a.d2[u] + a.d2[x] + a.d2[y] - (u64)(2 * (sd - 3) + 2 * (sa - 3));
  t.kite += (u64)((aux - 1) * (dy - 2) + (auy - 1) * (dx - 2) + (axy - 1) * (du - 2));
  t.gem += (u64)((aux - 1) * (auy - 1) + (aux - 1) * (axy - 1) + (auy - 1) * (axy - 1));
  t.kd += (u64)(k * sd);
  t.ka += (u64)(k * sa);
  t.kk += c2((u64)k);
}

// Element idx of the list of up entry i of u (entry e), the same slot of its
// reverse list being at rev_at: when its neighbour is an up neighbour j > i,
// the triangle (u, i, j).  R: rows over N(u) (wd words), M: rows over N+(u)
// (wp words).
__device__ __forceinline__ void tau_element(const MotifArgs &a, TauSums &t, int u, int du, int i,
                                            int e, int64_t rev_at, int idx, const unsigned *R,
                                            int wd, const unsigned *M, int wp) {
  const int j = a.pos1[idx] - 1;
  if (j <= i) return;
  if (a.need & kNeedTau) {
    int k = 0;
    for (int w = 0; w < wd; ++w) k += __popc(R[i * wd + w] & R[j * wd + w]);
    tau_terms(a, t, u, __ldg(a.ci + e), __ldg(a.ci + idx), du, a.a[e], a.a[idx],
              a.a[a.list[rev_at]], k);
  }
  for (int w = (j + 1) >> 5; w < wp; ++w) {
    unsigned m = M[i * wp + w] & M[j * wp + w] & above(j, w);
    t.K4 += __popc(m);
    if (!(a.need & kNeedTau)) continue;
    while (m) {
      const int l = 32 * w + __ffs(m) - 1;
      m &= m - 1;
      for (int w2 = (l + 1) >> 5; w2 < wp; ++w2)
        t.K5 += __popc(M[i * wp + w2] & M[j * wp + w2] & M[l * wp + w2] & above(l, w2));
    }
  }
}

// Warps over all u: vertex and edge sums, and the bit rows of u with d+ <= 32
// and d <= 512, lane i owning row i.  R: kTauOut x kTauDeg bits, M: kTauOut.
__device__ void tau_small(const MotifArgs &a, TauSums &t, unsigned *R, unsigned *M, int lane) {
  const int stride = gridDim.x * kWarps;
  for (int u = blockIdx.x * kWarps + threadIdx.x / kWarp; u < a.n; u += stride) {
    const int p = a.dp[u], d = a.deg[u];
    const int b = (int)__ldg(a.rp + u);
    if (a.need & kNeedT) {
      int t2 = 0;
      for (int i = b + lane; i < b + d; i += kWarp) t2 += a.a[i];
      const u64 sum = warp_sum_u64((u64)t2);
      if (lane == 0) t.vt2 += c2(sum >> 1);
    }
    if (p == 0 || p > kTauOut) continue;
    int e = 0, na = 0;
    int64_t off = 0, roff = 0;
    if (lane < p) {
      e = a.upe[b + lane];
      na = a.a[e];
      t.edge((u64)d, (u64)a.deg[__ldg(a.ci + e)], (u64)na);
    }
    if (p < 2 || d > kTauDeg || !__any_sync(kFull, na > 0)) continue;
    const int wd = (a.need & kNeedTau) ? (d + 31) >> 5 : 0;
    for (int w = lane; w < p * wd; w += kWarp) R[w] = 0;
    M[lane] = 0;
    if (na > 0) {
      off = a.off[e];
      roff = a.off[a.rev1[e] - 1];
    }
    __syncwarp();
    walk_lists(a, off, na, lane, [&](int idx, int i, int64_t) {
      const int ps = idx - b, j1 = a.pos1[idx];
      if (wd) atomicOr(R + i * wd + (ps >> 5), 1u << (ps & 31));
      if (j1) atomicOr(M + i, 1u << (j1 - 1));
    });
    __syncwarp();
    // The up entry of the list's row, and where its reverse list starts
    // against its own, by lane.
    const int64_t shift = roff - off;
    const FlatLists fl(na, lane);
    const int64_t start = off - (fl.incl - na);
    for (int base = 0; base < fl.total; base += kWarp) {
      const int g = base + lane;
      const int i = fl.owner(g);
      const int64_t q = __shfl_sync(kFull, start, i) + g;
      const int64_t sh = __shfl_sync(kFull, shift, i);
      const int ei = __shfl_sync(kFull, e, i);
      if (g < fl.total) tau_element(a, t, u, d, i, ei, q + sh, a.list[q], R, wd, M, 1);
    }
    __syncwarp();
  }
}

// CTA per larger u (queue over tau_big): warp per row, lanes over its list.
// The rows take p (wd + wp) words: p d <= nnz and p^2 <= nnz, since u's p up
// neighbours have at least u's degree, so slice_words bounds them.
__device__ void tau_large(const MotifArgs &a, TauSums &t, unsigned *s_rows, int smem_words,
                          int *s_u, int lane, int warp) {
  for (;;) {
    if (threadIdx.x == 0) {
      const unsigned i = atomicAdd(a.counts + kTauQueue, 1u);
      *s_u = i < a.counts[kTauN] ? a.tau_big[i] : -1;
    }
    __syncthreads();
    const int u = *s_u;
    __syncthreads();
    if (u < 0) break;
    const int p = a.dp[u], d = a.deg[u], b = (int)__ldg(a.rp + u);
    const int wd = (a.need & kNeedTau) ? (d + 31) >> 5 : 0, wp = (p + 31) >> 5;
    const int64_t words = (int64_t)p * (wd + wp);
    unsigned *R = words <= smem_words ? s_rows : a.slices + blockIdx.x * a.slice_words;
    unsigned *M = R + (int64_t)p * wd;
    for (int64_t i = threadIdx.x; i < words; i += kThreads) R[i] = 0;
    __syncthreads();
    for (int i = warp; i < p; i += kWarps) {
      const int e = a.upe[b + i], na = a.a[e];
      if (p > kTauOut && lane == 0) t.edge((u64)d, (u64)a.deg[__ldg(a.ci + e)], (u64)na);
      if (na == 0) continue;
      const int64_t off = a.off[e];
      for (int q = lane; q < na; q += kWarp) {
        const int idx = a.list[off + q];
        const int ps = idx - b, j1 = a.pos1[idx];
        if (wd) atomicOr(R + (int64_t)i * wd + (ps >> 5), 1u << (ps & 31));
        if (j1) atomicOr(M + (int64_t)i * wp + ((j1 - 1) >> 5), 1u << ((j1 - 1) & 31));
      }
    }
    __syncthreads();
    for (int i = warp; i < p; i += kWarps) {
      const int e = a.upe[b + i], na = a.a[e];
      if (na == 0) continue;
      const int64_t off = a.off[e], roff = a.off[a.rev1[e] - 1];
      for (int q = lane; q < na; q += kWarp)
        tau_element(a, t, u, d, i, e, roff + q, a.list[off + q], R, wd, M, wp);
    }
    __syncthreads();
  }
}

// Between the sum of all walks and the pairs stage: the walks to take in parts
// leave the list of the huge ones (-1).
__device__ __forceinline__ void split_walks(const MotifArgs &a) {
  const int huge = (int)a.counts[kHugeN];
  const u64 share = *a.walk_total / (u64)a.num_sms;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < huge; i += gridDim.x * blockDim.x) {
    const int s = a.pair_big[i];
    const u64 w = a.walk[s];
    if (w <= kSplitWalk || w <= share) continue;
    const int parts = (int)min(min(w >> 15, (u64)8), 2 * (w / (share + 1) + 1));
    const int at = (int)atomicAdd(a.counts + kSplitN, (unsigned)parts);
    const bool fits = at + parts <= a.split_cap;
    for (int k = 0; k < parts && at + k < a.split_cap; ++k)
      a.split[at + k] = make_int4(fits ? s : -1, k, parts, 0);
    if (fits) a.pair_big[i] = -1;
  }
}

// Both forms in one launch while the large form's rows leave the SM full of
// CTAs, else one launch each.
template <bool kLarge, bool kSmall>
__global__ void __launch_bounds__(kThreads) motif_tau_kernel(MotifArgs a, int smem_words) {
  extern __shared__ unsigned s_rows[];
  __shared__ u64 sm[kSums];
  __shared__ unsigned s_r[kSmall ? kWarps : 1][kSmall ? kTauOut * (kTauDeg / 32) : 1];
  __shared__ unsigned s_m[kSmall ? kWarps : 1][kTauOut];
  __shared__ int s_u;
  const BlockSums bs{sm};
  bs.init();
  if (a.early ? stops_here(a) : lists_overrun(a)) return;
  const int lane = threadIdx.x & (kWarp - 1), warp = threadIdx.x / kWarp;
  TauSums t;
  if (kLarge && a.split_cap > 0 && (a.need & kNeedC4)) split_walks(a);
  if (kLarge) tau_large(a, t, s_rows, smem_words, &s_u, lane, warp);
  if (kSmall) tau_small(a, t, s_r[kSmall ? warp : 0], s_m[kSmall ? warp : 0], lane);
  t.flush(bs, a.need & kNeedTau);
  bs.flush(a.acc);
}

// ---- pairs at distance two -----------------------------------------------------
// Per s, a table over t counts the two-paths s - v - t.  kOrdered: v and t
// below s in (degree, id), so that a 4-cycle is counted once, at its highest
// vertex (sum over edges of the smaller degree in entries).  Otherwise every
// pair t < s by id: entries of N(v) before s, which the reverse entry ends
// (half the two-paths).  An increment from c to c + 1 adds c to sum C(c, 2)
// and C(c, 2) to sum C(c, 3).
struct PairSums {
  u64 c4 = 0, c4d = 0, c4a = 0, x7 = 0, k23 = 0;
};

// This warp's share of a row's 32-entry pieces among nwarps warps: whole
// pieces when there are enough of them, else a part of one piece each.
struct Share {
  int first, step, part, parts;
  __device__ __forceinline__ Share(int d, int warp, int nwarps) {
    const int pieces = (d + kWarp - 1) / kWarp;
    parts = pieces >= nwarps || pieces == 0 ? 1 : nwarps / pieces;
    first = warp / parts;
    step = max(pieces, nwarps / parts);  // parts > 1: one piece
    if (parts == 1) step = nwarps;
    part = warp % parts;
  }
};

// First entry of the ascending ci[b, e) that is at least x, or e.
__device__ __forceinline__ int first_entry(const int32_t *__restrict__ ci, int b, int e, int x) {
  while (b < e) {
    const int mid = (b + e) >> 1;
    if (__ldg(ci + mid) < x) b = mid + 1;
    else e = mid;
  }
  return b;
}

// Calls f(t, entry of v -> t, entry of s -> v, v) for this warp's share of the
// two-paths from s (kRanged: of those with t in [t0, t1)).
template <bool kOrdered, bool kRanged = false, class F>
__device__ __forceinline__ void walk_pairs(const MotifArgs &a, int s, int b, int d, const Share &sh,
                                           int lane, F f, int t0 = 0, int t1 = 0) {
  for (int c = sh.first; c * kWarp < d; c += sh.step) {
    const int k = c * kWarp + lane;
    int e = 0, v = 0, st = 0, len = 0;
    if (k < d) {
      e = b + k;
      v = __ldg(a.ci + e);
      const int r1 = a.rev1[e];
      if (r1) {
        st = (int)__ldg(a.rp + v);
        if (kOrdered) {
          const int dv = a.deg[v];
          len = lower(dv, v, d, s) ? dv : 0;
          if (kRanged && len > 0) {
            const int end = st + dv;
            st = first_entry(a.ci, st, end, t0);
            len = first_entry(a.ci, st, end, t1) - st;
          }
        } else {
          len = r1 - 1 - st;
        }
      }
    }
    const FlatLists fl(len, lane);
    constexpr int kU = 4;
    for (int base = sh.part * kU * kWarp; base < fl.total; base += sh.parts * kU * kWarp) {
      int q[kU], t[kU], l[kU];
#pragma unroll
      for (int i = 0; i < kU; ++i) {
        const int g = base + i * kWarp + lane;
        l[i] = fl.owner(g);
        const int start = __shfl_sync(kFull, st - (fl.incl - len), l[i]);
        q[i] = g < fl.total ? start + g : -1;
        t[i] = q[i] >= 0 ? __ldg(a.ci + q[i]) : 0;
      }
      bool ok[kU];
#pragma unroll
      for (int i = 0; i < kU; ++i)
        ok[i] = q[i] >= 0 && (!kOrdered || lower(a.deg[t[i]], t[i], d, s));
#pragma unroll
      for (int i = 0; i < kU; ++i) {
        const int le = __shfl_sync(kFull, e, l[i]), lv = __shfl_sync(kFull, v, l[i]);
        if (ok[i]) f(t[i], q[i], le, lv);
      }
    }
  }
}

// All terms of one s with the table's operations: count(t) returns the count
// before an increment, get(t) the count; sync() orders the phases among the
// threads that share the table, which the caller clears afterwards.
template <bool kOrdered, class Count, class Get, class Sync>
__device__ __forceinline__ void pair_terms(const MotifArgs &a, PairSums &ps, int s, int b, int d,
                                           const Share &sh, int lane, Count count, Get get,
                                           Sync sync) {
  const bool k23 = a.need & kNeedK23;
  walk_pairs<kOrdered>(a, s, b, d, sh, lane, [&](int t, int, int, int) {
    const u64 c = count(t);
    ps.c4 += c;
    if (!kOrdered && k23 && c) {
      ps.c4d += c * (u64)(d + a.deg[t]);
      ps.k23 += c2(c);
    }
  });
  sync();
  if (kOrdered) return;
  walk_pairs<kOrdered>(a, s, b, d, sh, lane, [&](int t, int q, int e, int v) {
    const u64 c = get(t);
    if (c < 2) return;
    ps.c4a += (c - 1) * (u64)(a.a[e] + a.a[q]);
    if (k23) ps.c4d += (c - 1) * (u64)a.deg[v];
  });
  // X7: for each edge (p, r) inside N(s), the pairs (s, t) with t adjacent to
  // p and r: the lists of 32 p's are walked flat for 32 r's at a time, and
  // those edges' lists flat again.
  for (int c = sh.first; c * kWarp < d; c += sh.step) {
    const int k = c * kWarp + lane;
    const int e = b + k;
    const int na = k < d ? a.a[e] : 0;
    int64_t off = 0, shift = 0;
    if (na > 0) {
      off = a.off[e];
      shift = a.off[a.rev1[e] - 1] - off;
    }
    const FlatLists fl(na, lane);
    const int64_t start = off - (fl.incl - na);
    for (int base = sh.part * kWarp; base < fl.total; base += sh.parts * kWarp) {
      const int g = base + lane;
      const int l = fl.owner(g);
      const int64_t at = __shfl_sync(kFull, start, l) + g, sft = __shfl_sync(kFull, shift, l);
      const int ep = __shfl_sync(kFull, e, l);
      int len = 0;
      int64_t lo = 0;
      if (g < fl.total && a.list[at] > ep) {  // each edge from one end
        const int pr = a.list[at + sft];
        lo = a.off[pr];
        len = a.a[pr];
      }
      walk_lists(a, lo, len, lane, [&](int idx, int, int64_t) {
        const int t = __ldg(a.ci + idx);
        if (t < s) ps.x7 += get(t) - 2;
      });
    }
  }
  sync();
}

__device__ __forceinline__ void flush_pairs(const BlockSums &bs, const PairSums &ps, u64 *acc) {
  bs.add(kC4, ps.c4);
  bs.add(kC4d, ps.c4d);
  bs.add(kC4a, ps.c4a);
  bs.add(kX7, ps.x7);
  bs.add(kK23, ps.k23);
  bs.flush(acc);
}

// An open-addressing table of 2^lg slots: keys, and 16-bit counts two to a
// word (a count is at most the maximum degree, 46,340).  Never more than half
// full, so every probe ends.
struct HashTable {
  int *key;
  unsigned *cnt;
  int lg;
  __device__ __forceinline__ void size_for(unsigned walk) {
    lg = 6;
    while ((1u << lg) < 2 * walk) ++lg;
  }
  __device__ __forceinline__ u64 count(int t) const {
    const int mask = (1 << lg) - 1;
    int sl = (int)hash_slot(t, 32 - lg);
    for (;;) {
      const int k = atomicCAS(key + sl, -1, t);
      if (k == -1 || k == t) break;
      sl = (sl + 1) & mask;
    }
    const int sh = (sl & 1) * 16;
    return (u64)((atomicAdd(cnt + (sl >> 1), 1u << sh) >> sh) & 0xffffu);
  }
  __device__ __forceinline__ u64 get(int t) const {
    const int mask = (1 << lg) - 1;
    int sl = (int)hash_slot(t, 32 - lg);
    for (;;) {
      const int k = key[sl];
      if (k == t) return (u64)((cnt[sl >> 1] >> ((sl & 1) * 16)) & 0xffffu);
      if (k == -1) return 0;
      sl = (sl + 1) & mask;
    }
  }
  __device__ __forceinline__ void clear(int tid, int threads) const {
    int4 *k4 = reinterpret_cast<int4 *>(key);
    uint4 *c4 = reinterpret_cast<uint4 *>(cnt);
    for (int i = tid; i < 1 << (lg - 2); i += threads) k4[i] = make_int4(-1, -1, -1, -1);
    for (int i = tid; i < 1 << (lg - 3); i += threads) c4[i] = make_uint4(0, 0, 0, 0);
  }
};

constexpr size_t hash_bytes(int slots) { return (sizeof(int) + 2) * (size_t)slots; }

// Warp per s of at most kWarpWalk table entries.
template <bool kOrdered>
__global__ void __launch_bounds__(kThreads) motif_pairs_kernel(MotifArgs a) {
  extern __shared__ __align__(16) int s_tab[];
  __shared__ u64 sm[kSums];
  const BlockSums bs{sm};
  bs.init();
  if (stops_here(a)) return;
  const int lane = threadIdx.x & (kWarp - 1), warp = threadIdx.x / kWarp;
  int *mine = s_tab + warp * (kHashSlots + kHashSlots / 2);
  HashTable tab{mine, reinterpret_cast<unsigned *>(mine + kHashSlots), 10};
  tab.clear(lane, kWarp);
  __syncwarp();
  PairSums ps;
  const int stride = gridDim.x * kWarps;
  for (int s = blockIdx.x * kWarps + warp; s < a.n; s += stride) {
    const u64 w = a.walk[s];
    if (w < 2 || w > a.warp_walk) continue;
    tab.size_for((unsigned)w);
    const int b = (int)__ldg(a.rp + s), d = a.deg[s];
    pair_terms<kOrdered>(
        a, ps, s, b, d, Share(d, 0, 1), lane, [&](int t) { return tab.count(t); },
        [&](int t) { return tab.get(t); }, [&]() { __syncwarp(); });
    tab.clear(lane, kWarp);
    __syncwarp();
  }
  flush_pairs(bs, ps, a.acc);
}

// CTA per s of the hash classes: kFront the front list of pair_mid, else the
// back one; 2^kLg slots.
template <bool kOrdered, bool kFront, int kT, int kLg>
__global__ void __launch_bounds__(kT) motif_pairs_hash_kernel(MotifArgs a) {
  extern __shared__ __align__(16) int s_tab[];
  __shared__ u64 sm[kSums];
  __shared__ int s_s;
  const BlockSums bs{sm};
  bs.init();
  if (stops_here(a)) return;
  const int lane = threadIdx.x & (kWarp - 1), warp = threadIdx.x / kWarp;
  HashTable tab{s_tab, reinterpret_cast<unsigned *>(s_tab + (1 << kLg)), kLg};
  PairSums ps;
  for (bool first = true;; first = false) {
    if (threadIdx.x == 0) {
      const unsigned i = atomicAdd(a.counts + (kFront ? kMidQueue : kHashQueue), 1u);
      s_s = i < a.counts[kFront ? kMidN : kHashN] ? a.pair_mid[kFront ? i : a.n - 1 - i] : -1;
    }
    __syncthreads();
    const int s = s_s;
    if (s < 0) break;
    if (first) {
      tab.clear(threadIdx.x, kT);
      __syncthreads();
    }
    tab.size_for((unsigned)a.walk[s]);
    const int b = (int)__ldg(a.rp + s), d = a.deg[s];
    pair_terms<kOrdered>(
        a, ps, s, b, d, Share(d, warp, kT / kWarp), lane, [&](int t) { return tab.count(t); },
        [&](int t) { return tab.get(t); }, [&]() { __syncthreads(); });
    tab.clear(threadIdx.x, kT);  // as far as this walk's table went
  }
  flush_pairs(bs, ps, a.acc);
}

constexpr int kPairThreads = 1024;

// First row that starts at or after entry e; n if none does.
__device__ int row_at(const int64_t *__restrict__ rp, int n, int64_t e) {
  int lo = 0, hi = n;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (__ldg(rp + mid) < e) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// CTA per larger s (longest walks first): 16-bit counters over all vertices,
// two to a word, in shared memory when n of them fit, else one slice of
// `counters` per CTA.  Items [begin, end) of the list (ordered walks, with their
// parts in front: all).
template <bool kOrdered, bool kShared>
__global__ void __launch_bounds__(kPairThreads) motif_pairs_big_kernel(MotifArgs a, unsigned *counters,
                                                                       unsigned begin, unsigned end) {
  extern __shared__ __align__(16) int s_tab[];
  __shared__ u64 sm[kSums];
  __shared__ int2 s_item;
  __shared__ int s_range[2];
  const BlockSums bs{sm};
  bs.init();
  if (stops_here(a)) return;
  const int words = (a.n + 1) >> 1;
  unsigned *cnt = kShared ? reinterpret_cast<unsigned *>(s_tab)
                          : counters + (int64_t)blockIdx.x * words;
  const int lane = threadIdx.x & (kWarp - 1), warp = threadIdx.x / kWarp;
  constexpr int kEnd = -2;
  bool clean = false;  // the counters are zero
  PairSums ps;
  const int splits = (int)min(a.counts[kSplitN], (unsigned)a.split_cap);
  for (;;) {
    if (threadIdx.x == 0) {
      unsigned i = begin + atomicAdd(a.counts + kBigQueue, 1u);
      const unsigned huge = a.counts[kHugeN], big = a.counts[kBigN];
      int4 item = make_int4(kEnd, 0, 1, 0);
      if (i < end && (int)i < splits) {
        item = a.split[i];
        // Parts of about the same number of entries: t's place in the CSR.
        for (int k = 0; k < 2; ++k)
          s_range[k] = row_at(a.rp, a.n, (int64_t)a.nnz * (item.y + k) / item.z);
      } else if (i < end && i - (unsigned)splits < huge + big) {
        i -= (unsigned)splits;
        item.x = i < huge ? a.pair_big[i] : a.pair_big[a.n - 1 - (i - huge)];
      }
      s_item = make_int2(item.x, item.z);
    }
    __syncthreads();
    const int s = s_item.x, parts = s_item.y;
    const int t0 = s_range[0], t1 = s_range[1];
    if (s == kEnd) break;
    if (s < 0) {  // a walk taken in parts, or room that no walk's parts fitted
      __syncthreads();
      continue;
    }
    if (!clean) {
      for (int i = threadIdx.x; i < words; i += kPairThreads) cnt[i] = 0;
      __syncthreads();
    }
    const int b = (int)__ldg(a.rp + s), d = a.deg[s];
    const Share sh(d, warp, kPairThreads / kWarp);
    if (kOrdered && parts > 1) {
      walk_pairs<kOrdered, true>(
          a, s, b, d, sh, lane,
          [&](int t, int, int, int) {
            const int bit = (t & 1) * 16;
            ps.c4 += (u64)((atomicAdd(cnt + (t >> 1), 1u << bit) >> bit) & 0xffffu);
          },
          t0, t1);
      clean = false;
      __syncthreads();
      continue;
    }
    pair_terms<kOrdered>(
        a, ps, s, b, d, sh, lane,
        [&](int t) {
          const int bit = (t & 1) * 16;
          return (u64)((atomicAdd(cnt + (t >> 1), 1u << bit) >> bit) & 0xffffu);
        },
        [&](int t) { return (u64)((cnt[t >> 1] >> ((t & 1) * 16)) & 0xffffu); },
        [&]() { __syncthreads(); });
    // A walk much shorter than the table clears its words one by one (both
    // counters of a word in this phase), a longer one leaves it to the sweep.
    clean = a.walk[s] * 4 < (u64)words;
    if (clean)
      walk_pairs<kOrdered>(a, s, b, d, sh, lane, [&](int t, int, int, int) { cnt[t >> 1] = 0; });
    __syncthreads();
  }
  flush_pairs(bs, ps, a.acc);
}

// ---- 4-wheels ---------------------------------------------------------------
// Per entry (v -> x), the two-paths x - y - z inside N(v) with y and z before
// x in v's row, counted in a table over N(v): a 4-cycle of N(v) is counted
// once, at its last vertex.  Warp per entry of a row of at most kWheelDeg, a
// warp taking `per` consecutive entries.
__global__ void __launch_bounds__(kThreads) motif_wheel_kernel(MotifArgs a, int per) {
  __shared__ u64 sm[kSums];
  __shared__ unsigned s_cnt[kWarps][kWheelDeg];
  const BlockSums bs{sm};
  bs.init();
  if (stops_here(a)) return;
  const int lane = threadIdx.x & (kWarp - 1), warp = threadIdx.x / kWarp;
  unsigned *cnt = s_cnt[warp];
  for (int i = lane; i < kWheelDeg; i += kWarp) cnt[i] = 0;
  __syncwarp();
  u64 w4 = 0;
  const int64_t stride = (int64_t)gridDim.x * kWarps * per;
  for (int64_t base = ((int64_t)blockIdx.x * kWarps + warp) * per; base < a.nnz; base += stride) {
    const int64_t e64 = base + lane;
    unsigned todo = __ballot_sync(
        kFull, lane < per && e64 < a.nnz && a.a[e64] >= 2 && a.deg[a.src[e64]] <= kWheelDeg);
    while (todo) {
      const int e = (int)base + __ffs(todo) - 1;
      todo &= todo - 1;
      const int b = (int)__ldg(a.rp + a.src[e]);
      const int na = a.a[e];
      const int64_t off = a.off[e];
      for (int pass = 0; pass < 2; ++pass) {
        for (int j0 = 0; j0 < na; j0 += kWarp) {
          const int y = j0 + lane < na ? a.list[off + j0 + lane] : e;
          const bool before = y < e;
          walk_lists(a, before ? a.off[y] : 0, before ? a.a[y] : 0, lane,
                     [&](int z, int, int64_t) {
            if (z >= e) return;
            if (pass == 0) w4 += atomicAdd(cnt + (z - b), 1u);
            else cnt[z - b] = 0;
          });
        }
        __syncwarp();
      }
    }
  }
  bs.add(kW4, w4);
  bs.flush(a.acc);
}

// CTA per entry of a longer row: warp per y, lanes over y's list; entries [begin,
// end), claimed `per` at a time: the hubs' entries lie together, and with fixed
// shares the slices of the Chung-Lu graph of 10^6 vertices (cap 50,000) took 13.7 s
// in P3 where one launch took 5.6.
__global__ void __launch_bounds__(kThreads) motif_wheel_big_kernel(MotifArgs a, int table, int64_t begin,
                                                                   int64_t end, int per) {
  extern __shared__ unsigned s_cnt[];
  __shared__ u64 sm[kSums];
  __shared__ int s_e[kThreads], s_n;
  __shared__ int64_t s_base;
  const BlockSums bs{sm};
  bs.init();
  if (stops_here(a)) return;
  const int lane = threadIdx.x & (kWarp - 1), warp = threadIdx.x / kWarp;
  for (int i = threadIdx.x; i < table; i += kThreads) s_cnt[i] = 0;
  u64 *queue = reinterpret_cast<u64 *>(a.counts + kWheelQueue);
  u64 w4 = 0;
  for (;;) {
    if (threadIdx.x == 0) {
      s_n = 0;
      s_base = begin + (int64_t)(atomicAdd(queue, 1ull) * (u64)per);
    }
    __syncthreads();
    const int64_t base = s_base;
    if (base >= end) break;
    const int64_t e64 = base + threadIdx.x;
    if ((int)threadIdx.x < per && e64 < end && a.a[e64] >= 2 && a.deg[a.src[e64]] > kWheelDeg)
      s_e[atomicAdd(&s_n, 1)] = (int)e64;
    __syncthreads();
    for (int i = 0; i < s_n; ++i) {
      const int e = s_e[i];
      const int b = (int)__ldg(a.rp + a.src[e]);
      const int na = a.a[e];
      const int64_t off = a.off[e];
      for (int pass = 0; pass < 2; ++pass) {
        for (int j = warp; j < na; j += kWarps) {
          const int y = a.list[off + j];
          if (y >= e) continue;
          const int64_t lo = a.off[y], hi = lo + a.a[y];
          for (int64_t q = lo + lane; q < hi; q += kWarp) {
            const int z = a.list[q];
            if (z >= e) continue;
            if (pass == 0) w4 += atomicAdd(s_cnt + (z - b), 1u);
            else s_cnt[z - b] = 0;
          }
        }
        __syncthreads();
      }
    }
    __syncthreads();
  }
  bs.add(kW4, w4);
  bs.flush(a.acc);
}

// ---- host -------------------------------------------------------------------
unsigned blocks(int64_t items, int per_block) {
  return (unsigned)std::max<int64_t>(1, (items + per_block - 1) / per_block);
}

// Entries a warp takes at once, so that some 64 warps per SM have work.
int spread(int64_t entries, int num_sms) {
  return (int)std::max<int64_t>(1, std::min<int64_t>(kWarp, entries / (64 * (int64_t)num_sms)));
}

int resident(const void *kernel, int threads, size_t smem) {
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem) != cudaSuccess)
    per_sm = 1;
  return std::max(per_sm, 1);
}

// Carves aligned arrays out of one allocation.
struct Carver {
  char *base = nullptr;
  size_t used = 0;
  template <typename T>
  T *take(int64_t count) {
    T *p = reinterpret_cast<T *>(base + used);
    used += (sizeof(T) * (size_t)std::max<int64_t>(count, 1) + 255) & ~size_t(255);
    return p;
  }
};

// The pairs stage's classes that walks up to `longest` reach.
template <bool kOrdered>
int launch_pairs(mc_dgraph *g, const MotifArgs &a, int64_t longest, int big_grid, bool shared,
                 size_t table_b, unsigned *counters, Slicer &sl) {
  cudaStream_t s = g->stream;
  auto launch = [&](auto kern, int threads, size_t smem, int64_t items) -> int {
    MC_CUDA_TRY(allow_smem((const void *)kern, smem));
    const int64_t fit = items <= g->num_sms
                            ? items
                            : (int64_t)g->num_sms * resident((const void *)kern, threads, smem);
    kern<<<(unsigned)std::max<int64_t>(1, std::min(items, fit)), threads, smem, s>>>(a);
    MC_CUDA_TRY(cudaGetLastError());
    g->launches += 1;
    return MC_OK;
  };
  int rc = launch(motif_pairs_kernel<kOrdered>, kThreads, kWarps * hash_bytes(kHashSlots),
                  blocks(a.n, kWarps));
  if (rc == MC_OK && longest > (int64_t)a.warp_walk)
    rc = launch(motif_pairs_hash_kernel<kOrdered, true, 128, 12>, 128, hash_bytes(1 << 12), a.n);
  if (rc == MC_OK && longest > (int64_t)a.mid_walk)
    rc = launch(motif_pairs_hash_kernel<kOrdered, false, 512, 14>, 512, hash_bytes(1 << 14), a.n);
  if (rc != MC_OK || longest <= (int64_t)kHashWalk) return rc;
  auto big = shared ? motif_pairs_big_kernel<kOrdered, true> : motif_pairs_big_kernel<kOrdered, false>;
  const size_t smem = shared ? table_b : 0;
  MC_CUDA_TRY(allow_smem((const void *)big, smem));
  // In slices the walks of all pairs, of hubs seconds in all (ordered ones are
  // bounded by the edges' smaller degrees).
  unsigned n_items[kCounts] = {};
  if (sl.on && !kOrdered) {
    MC_CUDA_TRY(cudaMemcpyAsync(n_items, a.counts, sizeof(n_items), cudaMemcpyDeviceToHost, s));
    MC_CUDA_TRY(cudaStreamSynchronize(s));
  }
  auto run = [&](int64_t b, int64_t e) -> int {
    big<<<big_grid, kPairThreads, smem, s>>>(a, counters, (unsigned)b, e < 0 ? ~0u : (unsigned)e);
    MC_CUDA_TRY(cudaGetLastError());
    g->launches += 1;
    return MC_OK;
  };
  if (kOrdered) return run(0, -1);
  const int64_t giants = std::min<unsigned>(n_items[kSplitN], (unsigned)a.split_cap);
  return run_slices(g, sl, "pairs", giants + n_items[kHugeN] + n_items[kBigN], giants + big_grid,
                    reinterpret_cast<u64 *>(a.counts + kBigQueue), run);
}

}  // namespace

// The route of a whole count: by sizes (routes.h), unless the environment asks
// for another route or its forms; never the motif sums with columns in host
// memory (the pairs stage reads rows once per two-path).
PatternRoute pattern_route(const mc_dgraph *g, int pattern) {
  if (!motif_sums_apply(g->n, g->nnz, g->max_degree) || g->batch.gid || g->col_host)
    return PatternRoute::kFormula;
  for (const char *name : {"MERCURY_PATTERN_KERNEL", "MERCURY_CLIQUE_ROUTE", "MERCURY_PATTERN_SETS",
                           "MERCURY_PATTERN_SLICE", "MERCURY_HUB_P1", "MERCURY_HOP_ROWS"})
    if (std::getenv(name)) return PatternRoute::kFormula;
  // MERCURY_MOTIF_ROUTE=formula|dense|sparse (tests and timing comparisons).
  if (const char *env = std::getenv("MERCURY_MOTIF_ROUTE")) {
    if (std::strcmp(env, "formula") == 0) return PatternRoute::kFormula;
    if (std::strcmp(env, "dense") == 0)
      return g->n <= kDenseMax ? PatternRoute::kDense : PatternRoute::kSparse;
    if (std::strcmp(env, "sparse") == 0) return PatternRoute::kSparse;
  }
  return pattern_route_by_size(g->n, g->nnz, g->max_degree, pattern);
}

int motif_triangles(mc_dgraph *g, uint64_t *out) {
  NvtxRange range("motif_triangles");
  cudaStream_t s = g->stream;
  const int n = (int)g->n, nnz = (int)g->nnz;
  MotifArgs a{};
  a.rp = g->rowptr;
  a.ci = g->col;
  a.n = n;
  a.nnz = nnz;
  size_t zeroed = 0;
  auto lay_out = [&](Carver &c) {
    a.acc = c.take<u64>(kSums);
    a.dp = c.take<int32_t>(n);
    zeroed = c.used;
    a.deg = c.take<int32_t>(n);
    a.src = c.take<int32_t>(nnz);
    a.upe = c.take<int32_t>(nnz);
  };
  Carver size, c;
  lay_out(size);
  size_t got = 0;
  MC_CUDA_TRY(scratch_take(reinterpret_cast<void **>(&c.base), size.used, &got, g->device, s));
  lay_out(c);
  u64 total = 0;
  auto run = [&]() -> int {
    MC_CUDA_TRY(cudaMemsetAsync(c.base, 0, zeroed, s));
    const unsigned row_blocks = std::min(blocks(n, kWarps), 4096u);
    motif_rows_kernel<<<row_blocks, kThreads, 0, s>>>(a, (int)row_blocks);
    MC_CUDA_TRY(cudaGetLastError());
    tri_up_kernel<<<blocks(nnz, kThreads), kThreads, 0, s>>>(a);
    MC_CUDA_TRY(cudaGetLastError());
    const int per = spread(nnz, g->num_sms);
    tri_pairs_kernel<<<blocks(((int64_t)nnz + per - 1) / per * kWarp, kThreads), kThreads, 0, s>>>(a, per);
    MC_CUDA_TRY(cudaGetLastError());
    g->launches += 3;
    MC_CUDA_TRY(cudaEventRecord(g->ev[3], s));
    MC_CUDA_TRY(cudaMemcpyAsync(&total, a.acc + kT, sizeof(total), cudaMemcpyDeviceToHost, s));
    MC_CUDA_TRY(cudaStreamSynchronize(s));
    return MC_OK;
  };
  const int rc = run();
  if (rc == MC_OK) scratch_give(c.base, got, g->device, s);
  else dev_free(c.base, s);
  if (rc == MC_OK) *out = total;
  return rc;
}

int motif_count(mc_dgraph *g, int pattern, bool estimates, uint64_t *out, bool *elsewhere) {
  NvtxRange range("motif_count");
  cudaStream_t s = g->stream;
  const int n = (int)g->n, nnz = (int)g->nnz;
  const bool asked_for = estimates && n > kEstimateAbove;
  const unsigned need = motif_needs(pattern) & (asked_for ? ~0u : ~(unsigned)kNeedWork);
  *elsewhere = false;
  const bool pairs = need & (kNeedC4 | kNeedPairs), ordered = need & kNeedC4;
  const bool wheel = need & kNeedW4;
  // Shared-memory tables of the pairs stage: 16 bits per vertex.
  const size_t table_b = sizeof(unsigned) * (size_t)((n + 1) / 2);
  const bool table_shared = table_b <= (size_t(200) << 10);
  const int pair_grid = table_shared ? g->num_sms
                                     : (int)std::max<int64_t>(
                                           1, std::min<int64_t>(2 * g->num_sms,
                                                                (int64_t(2) << 30) / (int64_t)table_b));
  // A vertex's walk is at most the entries of its neighbours' rows.
  const int64_t longest = std::min<int64_t>(nnz, g->max_degree * g->max_degree);
  const int64_t root = (int64_t)std::sqrt((double)nnz) + 1;
  const int64_t slice_words = (2 * (int64_t)nnz + 64 * root) / 32 + 64;
  const bool slices = slice_words * 4 > kTauSmem;
  const int tau_grid = (int)std::max<int64_t>(
      1, std::min<int64_t>(2 * g->num_sms, slices ? (int64_t(1) << 30) / (4 * slice_words) : 1 << 20));
  // Room for the lists: nnz x max_degree bounds what the up stage hands out.
  // Where that exceeds the first guess, the count starts over with the room it
  // asked for, or, above 2 GiB, with lists sized by a counting pass.
  int64_t list_cap = std::min<int64_t>((int64_t)nnz * g->max_degree,
                                       std::max<int64_t>(int64_t(16) << 20, 64 * (int64_t)nnz));
  bool counted = false;
  for (;;) {
    MotifArgs a{};
    a.rp = g->rowptr;
    a.ci = g->col;
    a.n = n;
    a.nnz = nnz;
    a.pattern = pattern;
    a.need = need;
    a.probe_percent = estimates ? probe_percent(n, nnz, g->max_degree, pattern) : 0;
    a.early = (need & kNeedWork) && std::min(g->max_degree, root) > kEarlyOut;
    a.list_cap = list_cap;
    a.slice_words = slice_words;
    // Few vertices: a CTA for all but the shortest walks.
    a.warp_walk = n <= kFewVertices ? kFewWalk : kWarpWalk;
    a.mid_walk = kMidWalk;
    a.num_sms = g->num_sms;
    a.split_cap = (ordered && longest > (int64_t)kSplitWalk) ||
                          (pairs && !ordered && g->max_degree > kGiantDegree)
                      ? kSplitMax
                      : 0;
    size_t zeroed = 0;
    // The same layout for every pattern (so that each finds the last one's block).
    auto lay_out = [&](Carver &c) {
      // Zeroed before the first kernel.
      a.acc = c.take<u64>(kSums + 4);
      a.pool = a.acc + kSums;
      a.walk_total = a.pool + 1;
      a.probe = a.walk_total + 1;
      a.counts = c.take<unsigned>(kCounts);
      a.dp = c.take<int32_t>(n);
      a.d2 = c.take<u64>(n);
      a.walk = c.take<u64>(n);
      a.rev1 = c.take<int32_t>(nnz);
      a.a = c.take<int32_t>(nnz);
      if (counted) a.cnt = c.take<int32_t>(nnz);
      zeroed = c.used;
      a.split = c.take<int4>(kSplitMax);
      a.deg = c.take<int32_t>(n);
      a.src = c.take<int32_t>(nnz);
      a.upe = c.take<int32_t>(nnz);
      a.pos1 = c.take<int32_t>(nnz);
      a.off = c.take<int64_t>(nnz);
      a.tau_big = c.take<int32_t>(n);
      a.pair_mid = c.take<int32_t>(n);
      a.pair_big = c.take<int32_t>(n);
      a.slices = c.take<unsigned>(slices ? tau_grid * slice_words : 0);
      a.list = c.take<int32_t>(list_cap);
    };
    Carver size;
    lay_out(size);
    Carver c;
    // Large scratch leaves half of the free memory alone: first with lists
    // sized by a counting pass, then the caller takes a formula route, as it
    // does when the allocation fails.
    const size_t counters_b = pairs && !table_shared ? pair_grid * table_b : 0;
    if (size.used + counters_b > size_t(1) << 30) {
      const int64_t wanted = (int64_t)(size.used + counters_b);
      bool fits = false;
      const int arc = device_bytes_hold(g->device, 2 * wanted, &fits);
      if (arc != MC_OK) return arc;
      if (!fits) {
        if (counted) return MC_ERR_OOM;
        counted = true;
        list_cap = std::min<int64_t>(list_cap, 4 * (int64_t)nnz);
        continue;
      }
    }
    size_t got = 0, got_counters = 0;
    MC_CUDA_TRY(scratch_take(reinterpret_cast<void **>(&c.base), size.used, &got, g->device, s));
    lay_out(c);
    unsigned *counters = nullptr;
    if (counters_b) {
      const cudaError_t e = scratch_take(reinterpret_cast<void **>(&counters), counters_b,
                                         &got_counters, g->device, s);
      if (e != cudaSuccess) dev_free(c.base, s);
      MC_CUDA_TRY(e);
    }
    u64 h[kSums + 1];
    Slicer sl(g, -1.0);
    auto run = [&]() -> int {
      const int per = spread(nnz, g->num_sms);
      const unsigned tri_grid = blocks(std::max<int64_t>(n, ((int64_t)nnz + per - 1) / per * kWarp),
                                       kThreads);
      MC_CUDA_TRY(cudaMemsetAsync(c.base, 0, zeroed, s));
      const unsigned row_blocks = std::min(blocks(n, kWarps), 4096u);
      motif_rows_kernel<<<row_blocks + (a.probe_percent > 0 ? kProbeBlocks : 0), kThreads, 0, s>>>(
          a, (int)row_blocks);
      MC_CUDA_TRY(cudaGetLastError());
      motif_up_kernel<<<blocks(nnz, kThreads), kThreads, 0, s>>>(a);
      MC_CUDA_TRY(cudaGetLastError());
      if (counted) {
        motif_tri_kernel<true><<<tri_grid, kThreads, 0, s>>>(a, per);
        MC_CUDA_TRY(cudaGetLastError());
        motif_lists_kernel<<<blocks(nnz, kThreads), kThreads, 0, s>>>(a);
        MC_CUDA_TRY(cudaGetLastError());
        g->launches += 2;
      }
      motif_tri_kernel<false><<<tri_grid, kThreads, 0, s>>>(a, per);
      MC_CUDA_TRY(cudaGetLastError());
      if (a.early) {
        motif_squares_kernel<<<std::min(blocks(nnz, kThreads), (unsigned)(8 * g->num_sms)), kThreads,
                               0, s>>>(a);
        MC_CUDA_TRY(cudaGetLastError());
        g->launches += 1;
      }
      const unsigned tau_small_grid = std::min(blocks(n, kWarps), (unsigned)(8 * g->num_sms));
      if (slice_words * 4 <= kTauBoth) {
        motif_tau_kernel<true, true><<<tau_small_grid, kThreads, slice_words * 4, s>>>(
            a, (int)slice_words);
        MC_CUDA_TRY(cudaGetLastError());
        g->launches += 4;
      } else {
        MC_CUDA_TRY(allow_smem((const void *)motif_tau_kernel<true, false>, kTauSmem));
        motif_tau_kernel<true, false><<<tau_grid, kThreads, kTauSmem, s>>>(a, kTauSmem / 4);
        MC_CUDA_TRY(cudaGetLastError());
        motif_tau_kernel<false, true><<<tau_small_grid, kThreads, 0, s>>>(a, 0);
        MC_CUDA_TRY(cudaGetLastError());
        g->launches += 5;
      }
      // Slices are for stages that last: 2^30 of a^2 are some 7 ms of wheels and 30 of
      // X7, 2^32 two-paths some 20 (a star of 5,000, P3: 77 us in one launch, 163 in
      // slices).
      bool long_lists = false, long_walks = false;
      if (sl.on && !ordered && (pairs || wheel)) {
        MC_CUDA_TRY(cudaMemcpyAsync(h, a.acc, sizeof(h), cudaMemcpyDeviceToHost, s));
        MC_CUDA_TRY(cudaStreamSynchronize(s));
        long_lists = 4 * h[kD] + 6 * h[kT] > u64(1) << 30;
        long_walks = long_lists || (int64_t)nnz * g->max_degree > int64_t(1) << 33;
      }
      if (pairs) {
        sl.on = long_walks;
        const int rcp = ordered ? launch_pairs<true>(g, a, longest, pair_grid, table_shared, table_b, counters, sl)
                                : launch_pairs<false>(g, a, longest, pair_grid, table_shared, table_b, counters, sl);
        if (rcp != MC_OK) return rcp;
      }
      sl.on = long_lists;
      if (wheel) {
        motif_wheel_kernel<<<std::min(blocks(nnz, kWarps * per), (unsigned)(8 * g->num_sms)), kThreads,
                             0, s>>>(a, per);
        MC_CUDA_TRY(cudaGetLastError());
        g->launches += 1;
        if (g->max_degree > kWheelDeg) {
          const int table = (int)g->max_degree;
          const size_t smem = sizeof(unsigned) * (size_t)table;
          MC_CUDA_TRY(allow_smem((const void *)motif_wheel_big_kernel, smem));
          const int per_sm = resident((const void *)motif_wheel_big_kernel, kThreads, smem);
          const int64_t ctas = std::min(blocks(nnz, kThreads), (unsigned)(per_sm * g->num_sms));
          u64 *queue = reinterpret_cast<u64 *>(a.counts + kWheelQueue);
          const int rcw = run_slices(g, sl, "wheels", nnz, 4 * ctas, queue, [&](int64_t b, int64_t e) {
            if (e < 0) e = nnz;
            const int each = (int)std::max<int64_t>(1, std::min<int64_t>(kWheelClaim, (e - b) / (4 * ctas)));
            motif_wheel_big_kernel<<<(unsigned)ctas, kThreads, smem, s>>>(a, table, b, e, each);
            MC_CUDA_TRY(cudaGetLastError());
            g->launches += 1;
            return MC_OK;
          });
          if (rcw != MC_OK) return rcw;
        }
      }
      MC_CUDA_TRY(cudaEventRecord(g->ev[3], s));
      MC_CUDA_TRY(cudaMemcpyAsync(h, a.acc, sizeof(h), cudaMemcpyDeviceToHost, s));
      MC_CUDA_TRY(cudaStreamSynchronize(s));
      return MC_OK;
    };
    const int rc = run();
    if (rc != MC_OK) {  // work may be in flight: freed in the stream's order
      dev_free(c.base, s);
      if (counters) dev_free(counters, s);
      return rc;
    }
    scratch_give(c.base, got, g->device, s);
    scratch_give(counters, got_counters, g->device, s);
    if (h[kSums] == kClosed || (h[kSums] <= (u64)list_cap && (need & kNeedWork) &&
                                motif_outweighs(pattern, h))) {
      *elsewhere = true;
      return MC_OK;
    }
    const int64_t asked = (int64_t)h[kSums];
    if (asked <= list_cap) {
      *out = motif_combine(pattern, h);
      return MC_OK;
    }
    if (!counted && asked > int64_t(512) << 20) {
      counted = true;  // six entries per triangle instead of two rows per edge
    } else {
      list_cap = asked;
    }
  }
}

}  // namespace mc
