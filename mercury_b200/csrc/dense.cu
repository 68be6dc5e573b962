// P1..P8 of small graphs (at most kDenseMax vertices) from bit rows: the same
// motif sums as motifs.cu, read off popcounts of the adjacency matrix, which
// a CTA holds in shared memory.
//
// What bounds it: on graphs this small a call is launches and the latency of
// one pass over the CSR, so every CTA builds the whole matrix for itself and
// the sums take one kernel.  A vertex pair's common neighbours are the AND of
// two rows; each common neighbour v adds popcounts of v's row against them,
// so the work is n^2 / 2 row ANDs plus one per two-path.  RMAT scale 8 (256
// vertices, 1,297 edges), all eight patterns: the per-edge kernels took 6.1
// ms (P2 1.39), the sparse motif stages 1.3 (P2 0.41), these 0.7 (P2 0.13).
// In a batch, 455 such graphs took the persistent per-edge kernel some 5 ms,
// and take 0.75 ms, beside the triangle jobs.
#include <algorithm>
#include <cstdlib>

#include "device_common.cuh"
#include "dgraph.cuh"
#include "motifs.cuh"

namespace mc {
namespace {

constexpr int kDenseThreads = 512;
constexpr int kBatchThreads = 256;

// One graph: vertices [v0, v0 + n) of the CSR.
struct DenseGraph {
  const int64_t *__restrict__ rp;
  const int32_t *__restrict__ ci;
  int64_t v0;
  int n;
  int64_t nnz = 0;  // entries the caller gave (checked loads only)
};

// Rows of W words (bit_words: the loops over a row's words are unrolled up to 8)
// at an odd stride, so that lanes reading the same word of consecutive rows hit
// distinct banks; then n + 1 row offsets.
__host__ __device__ constexpr int dense_stride(int n) { return bit_words(n) | 1; }
size_t dense_bytes(int n) { return sizeof(int) * ((size_t)n * dense_stride(n) + n + 1); }

// The last row starting at or before entry e.
__device__ __forceinline__ int row_of(const int *off, int n, int e) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (off[mid] <= e) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// The graph's matrix and row offsets into shared memory, by the whole CTA.
// kCheck: a whole CSR against its contract, what breaks it in *err; false
// (on every thread) when the offsets do, and then no entry is read.  An id
// outside the graph sets nothing.
template <bool kCheck>
__device__ __forceinline__ bool load_matrix(const DenseGraph &g, unsigned *bits, int *off, int P,
                                            unsigned *err) {
  const int n = g.n;
  const int64_t base = kCheck ? 0 : __ldg(g.rp + g.v0);
  int bad_rows = 0;
  for (int i = threadIdx.x; i <= n; i += blockDim.x) {
    const int64_t a = __ldg(g.rp + g.v0 + i);
    if (kCheck)
      bad_rows |= a < 0 || a > g.nnz || (i == 0 && a != 0) || (i == n && a != g.nnz) ||
                  (i < n && __ldg(g.rp + i + 1) < a);
    off[i] = (int)(a - base);
  }
  for (int i = threadIdx.x; i < n * P; i += blockDim.x) bits[i] = 0;
  if (kCheck) {
    if (__syncthreads_or(bad_rows)) {
      if (threadIdx.x == 0) atomicOr(err, (unsigned)kErrRowptr);
      return false;
    }
  } else {
    __syncthreads();
  }
  const int nnz = off[n];
  for (int e = threadIdx.x; e < nnz; e += blockDim.x) {
    const int64_t id = (int64_t)__ldg(g.ci + base + e) - g.v0;
    const int r = row_of(off, n, e), x = (int)id;
    if (kCheck) {
      unsigned bad = 0;
      if (id < 0 || id >= n) bad |= kErrIdRange;
      if (id == r) bad |= kErrSelfLoop;
      if (e > off[r] && __ldg(g.ci + e - 1) >= id) bad |= kErrUnsorted;
      if (bad) atomicOr(err, bad);
      if (bad & kErrIdRange) continue;
    }
    atomicOr(bits + r * P + (x >> 5), 1u << (x & 31));
  }
  __syncthreads();
  return true;
}

// Adds this part's share of the graph's sums: warp tasks of (vertex) and of
// (vertex t, 32 vertices s below it), dealt round-robin over the warps of all
// parts.  need: Need bits; kW: words of a row, 0 above 8; smem: dense_bytes(n).
template <unsigned need, int kW>
__device__ __forceinline__ void dense_sums(const DenseGraph &g, int part, int parts, unsigned *smem,
                                           const BlockSums &bs) {
  const int n = g.n, W = kW > 0 ? kW : bit_words(n), P = W | 1;
  unsigned *bits = smem;
  int *off = reinterpret_cast<int *>(smem + (size_t)n * P);
  const int lane = threadIdx.x & (kWarp - 1), warp = threadIdx.x / kWarp;
  load_matrix<false>(g, bits, off, P, nullptr);
  auto deg = [&](int v) { return (u64)(off[v + 1] - off[v]); };
  const int gw = part * (blockDim.x / kWarp) + warp, step = parts * (blockDim.x / kWarp);
  constexpr bool tau = need & kNeedTau, pairs = need & kNeedPairs, wheel = need & kNeedW4;
  constexpr bool k23 = need & kNeedK23;

  u64 d3 = 0, d4 = 0, vt2 = 0, lolli = 0;
  for (int v = gw; v < n; v += step) {
    if (lane == 0) {
      d3 += c3((long long)deg(v));
      d4 += c4((long long)deg(v));
    }
    if (!(need & (kNeedT | kNeedD2))) continue;
    int t2 = 0;
    u64 dd = 0;
    if (lane < W) {
      unsigned word = bits[v * P + lane];
      while (word) {
        const int x = 32 * lane + __ffs(word) - 1;
        word &= word - 1;
        for (int w = 0; w < W; ++w) t2 += __popc(bits[v * P + w] & bits[x * P + w]);
        dd += deg(x) - 1;
      }
    }
    const u64 t = warp_sum_u64((u64)t2) >> 1;
    dd = warp_sum_u64(dd);
    if (lane == 0) {
      vt2 += c2(t);
      lolli += t * dd;
    }
  }
  bs.add(kVd3, d3);
  bs.add(kVd4, d4);
  bs.add(kVt2, vt2);

  u64 D = 0, C3 = 0, p4 = 0, fork = 0, dart = 0, T = 0, vtd = 0;
  u64 cricket = 0, bull = 0, kite = 0, gem = 0, kd = 0, ka = 0, kk = 0, K4 = 0, K5 = 0;
  u64 C4 = 0, C4d = 0, C4a = 0, X7 = 0, W4 = 0, K23 = 0;
  for (int task = gw; task < n * W; task += step) {
    const int t = task / W, s = 32 * (task - t * W) + lane;
    if (s - lane >= t) continue;  // every s of the warp
    const bool in = s < t;
    const unsigned *rs = bits + (in ? s : 0) * P, *rt = bits + t * P;
    const bool adj = in && ((rs[t >> 5] >> (t & 31)) & 1u);
    int c = 0, below = 0;
    if (adj || (in && (need & (kNeedC4 | kNeedPairs | kNeedW4)))) {
      for (int w = 0; w < W; ++w) {
        const unsigned S = rs[w] & rt[w];
        c += __popc(S);
        below += __popc(S & ~above(t - 1, w));
      }
      const u64 cu = (u64)c, ds = deg(s), dt = deg(t);
      if (need & kNeedC4) C4 += c2((u64)below);  // a 4-cycle once, at its last vertex
      if (pairs) {
        C4 += c2(cu);
        if (k23) {
          K23 += c3(c);
          C4d += c2(cu) * (ds + dt);
        }
      }
      if (adj) {
        D += c2(cu);
        C3 += c3(c);
        p4 += (ds - 1 - cu) * (dt - 1 - cu);
        fork += c2(ds - 1) * (dt - 1) + c2(dt - 1) * (ds - 1) - cu * (ds + dt - 4);
        dart += c2(cu) * (ds + dt - 6);
      }
    }
    // The common neighbours v of the warp's 32 pairs, one lane each.
    const int len = in && c > 0 && (adj || (c > 1 && (pairs || wheel))) ? c : 0;
    const int incl = warp_inclusive_scan(len, lane);
    const int total = __shfl_sync(kFull, incl, kWarp - 1);
    for (int first = 0; first < total; first += kWarp) {
      const int f = first + lane;
      int l = 0;  // the pair of item f
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
        if (__shfl_sync(kFull, incl, l + o - 1) <= f) l += o;
      l = min(l, kWarp - 1);
      const int cl = __shfl_sync(kFull, c, l);
      int j = f - (__shfl_sync(kFull, incl, l) - __shfl_sync(kFull, len, l));
      const bool adjl = __shfl_sync(kFull, (int)adj, l);
      if (f >= total) continue;
      const int sl = 32 * (task - t * W) + l;
      const unsigned *ra = bits + sl * P;
      int v = -1;  // the j-th common neighbour
      for (int w = 0; w < W; ++w) {
        unsigned set = ra[w] & rt[w];
        const int here = __popc(set);
        if (j >= here) {
          j -= here;
          continue;
        }
        while (j-- > 0) set &= set - 1;
        v = 32 * w + __ffs(set) - 1;
        break;
      }
      const unsigned *rv = bits + v * P;
      int k = 0, kb = 0, asv = 0, atv = 0;
      for (int w = 0; w < W; ++w) {
        const unsigned x = ra[w], y = rt[w], z = rv[w];
        const unsigned m = x & y & z;
        k += __popc(m);
        kb += __popc(m & ~above(t - 1, w));
        asv += __popc(x & z);
        atv += __popc(y & z);
      }
      const u64 cu = (u64)cl;
      if (wheel) W4 += c2((u64)kb);  // a wheel once, at its rim's last vertex
      if (pairs) {
        X7 += (u64)k * (cu - 2);  // twice: each edge among the pair's common neighbours
        C4a += (cu - 1) * (u64)(asv + atv);
        if (k23) C4d += (cu - 1) * deg(v);
      }
      if (!adjl || v < t) continue;
      // The triangle s < t < v.
      const long long du = (long long)deg(sl), dx = (long long)deg(t), dy = (long long)deg(v);
      const long long sd = du + dx + dy, sa = (long long)cl + asv + atv;
      ++T;
      vtd += (u64)sd;
      if (tau) {
        cricket += c2((u64)(du - 2)) + c2((u64)(dx - 2)) + c2((u64)(dy - 2));
        bull += (u64)((du - 2) * (dx - 2) + (du - 2) * (dy - 2) + (dx - 2) * (dy - 2) - sa + 3);
        lolli -= (u64)(2 * (sd - 3) + 2 * (sa - 3));
        kite += (u64)((cl - 1) * (dy - 2) + (asv - 1) * (dx - 2) + (atv - 1) * (du - 2));
        gem += (u64)((long long)(cl - 1) * (asv - 1) + (long long)(cl - 1) * (atv - 1) +
                     (long long)(asv - 1) * (atv - 1));
        kd += (u64)(k * sd);
        ka += (u64)(k * sa);
        kk += c2((u64)k);
      }
      if (k == 0) continue;
      for (int w = v >> 5; w < W; ++w) {
        unsigned m = ra[w] & rt[w] & rv[w] & above(v, w);
        K4 += __popc(m);
        while (tau && m) {
          const int q = 32 * w + __ffs(m) - 1;
          m &= m - 1;
          for (int w2 = q >> 5; w2 < W; ++w2)
            K5 += __popc(ra[w2] & rt[w2] & rv[w2] & bits[q * P + w2] & above(q, w2));
        }
      }
    }
  }
  __syncwarp();
  const u64 sums[] = {D, C3, p4, fork, dart, T, vtd, K4};
  const int at[] = {kD, kC3, kEp4, kEfork, kEdart, kT, kVtd, kK4};
#pragma unroll
  for (int i = 0; i < 8; ++i) bs.add(at[i], sums[i]);
  if (tau) {
    const u64 more[] = {cricket, bull, lolli, kite, gem, kd, ka, kk, K5};
    const int to[] = {kCricket, kBull, kLolli, kKite, kGem, kKd, kKa, kKk, kK5};
#pragma unroll
    for (int i = 0; i < 9; ++i) bs.add(to[i], more[i]);
  }
  if (need & (kNeedC4 | kNeedPairs)) bs.add(kC4, C4);
  if (wheel) bs.add(kW4, W4);
  if (pairs) {
    bs.add(kC4a, C4a);
    bs.add(kX7, X7);
    if (k23) {
      bs.add(kC4d, C4d);
      bs.add(kK23, K23);
    }
  }
}

template <unsigned need>
__device__ __forceinline__ void dense_words_of(const DenseGraph &g, int part, int parts,
                                               unsigned *smem, const BlockSums &bs) {
  switch (bit_words(g.n)) {
    case 1: return dense_sums<need, 1>(g, part, parts, smem, bs);
    case 2: return dense_sums<need, 2>(g, part, parts, smem, bs);
    case 4: return dense_sums<need, 4>(g, part, parts, smem, bs);
    case 8: return dense_sums<need, 8>(g, part, parts, smem, bs);
    default: return dense_sums<need, 0>(g, part, parts, smem, bs);
  }
}

__device__ __forceinline__ void dense_pattern(const DenseGraph &g, int pattern, int part, int parts,
                                              unsigned *smem, const BlockSums &bs) {
  switch (pattern) {
    case 1: return dense_words_of<motif_needs(1)>(g, part, parts, smem, bs);
    case 2: return dense_words_of<motif_needs(2)>(g, part, parts, smem, bs);
    case 3: return dense_words_of<motif_needs(3)>(g, part, parts, smem, bs);
    case 4: return dense_words_of<motif_needs(4)>(g, part, parts, smem, bs);
    case 5: return dense_words_of<motif_needs(5)>(g, part, parts, smem, bs);
    case 6: return dense_words_of<motif_needs(6)>(g, part, parts, smem, bs);
    default: return dense_words_of<motif_needs(7)>(g, part, parts, smem, bs);  // 7 and 8 alike
  }
}

__global__ void __launch_bounds__(kDenseThreads) dense_kernel(DenseGraph g, int pattern, u64 *acc) {
  extern __shared__ unsigned smem[];
  __shared__ u64 sm[kSums];
  const BlockSums bs{sm};
  bs.init();
  dense_pattern(g, pattern, blockIdx.x, gridDim.x, smem, bs);
  bs.flush(acc);
}

// A batch's small pattern graphs: one CTA per part (task) of a graph; acc
// holds kSums per batch graph.
__global__ void __launch_bounds__(kBatchThreads) dense_batch_kernel(
    const int64_t *__restrict__ rp, const int32_t *__restrict__ ci,
    const DenseTask *__restrict__ tasks, u64 *acc) {
  extern __shared__ unsigned smem[];
  __shared__ u64 sm[kSums];
  const BlockSums bs{sm};
  bs.init();
  const DenseTask t = tasks[blockIdx.x];
  dense_pattern(DenseGraph{rp, ci, t.v0, t.n}, t.job, t.part, t.parts, smem, bs);
  bs.flush(acc + (int64_t)t.graph * kSums);
}

// Triangles: for each entry (s -> t) with s < t, the common neighbours above t.
template <bool kCheck>
__global__ void __launch_bounds__(kDenseThreads) dense_triangles_kernel(DenseGraph g, u64 *count,
                                                                        unsigned *err) {
  extern __shared__ unsigned smem[];
  __shared__ u64 s_total;
  if (threadIdx.x == 0) s_total = 0;
  const int n = g.n, W = bit_words(n), P = W | 1;
  int *off = reinterpret_cast<int *>(smem + (size_t)n * P);
  if (!load_matrix<kCheck>(g, smem, off, P, err)) return;
  const int nnz = off[n];
  u64 hits = 0;
  for (int e = blockIdx.x * kDenseThreads + threadIdx.x; e < nnz; e += gridDim.x * kDenseThreads) {
    const int t = __ldg(g.ci + __ldg(g.rp + g.v0) + e) - (int)g.v0;
    const int s = row_of(off, n, e);
    if (t <= s || (kCheck && t >= n)) continue;
    const unsigned *rs = smem + s * P, *rt = smem + t * P;
    for (int w = t >> 5; w < W; ++w) hits += __popc(rs[w] & rt[w] & above(t, w));
  }
  hits = warp_sum_u64(hits);
  if ((threadIdx.x & (kWarp - 1)) == 0 && hits) atomicAdd(&s_total, hits);
  __syncthreads();
  if (threadIdx.x == 0 && s_total) atomicAdd(count, s_total);
}

}  // namespace

// Triangles of g (at most kDenseMax vertices) into counters[0]; check: a CSR
// that nothing has looked at yet, its contract errors in the low half of
// counters[1].  Asynchronous.
int dense_triangles(mc_dgraph *g, bool check) {
  cudaStream_t s = g->stream;
  const int n = (int)g->n;
  const size_t smem = dense_bytes(n);
  auto kern = check ? dense_triangles_kernel<true> : dense_triangles_kernel<false>;
  MC_CUDA_TRY(cudaMemsetAsync(g->counters, 0, 2 * sizeof(u64), s));
  if (smem > (size_t(40) << 10))
    MC_CUDA_TRY(allow_smem((const void *)kern, smem));
  // About 2^16 row words per CTA: each builds the matrix for itself.
  const int64_t words = g->nnz * bit_words(n) / 2;
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(g->num_sms, words >> 16));
  kern<<<grid, kDenseThreads, smem, s>>>(DenseGraph{g->rowptr, g->col, 0, n, g->nnz}, g->counters,
                                         reinterpret_cast<unsigned *>(g->counters + 1));
  MC_CUDA_TRY(cudaGetLastError());
  g->launches += 1;
  return MC_OK;
}

int dense_count(mc_dgraph *g, int pattern, uint64_t *out) {
  cudaStream_t s = g->stream;
  const int n = (int)g->n;
  const size_t smem = dense_bytes(n);
  u64 *acc = g->sums;
  u64 h[kSums];
  MC_CUDA_TRY(cudaMemsetAsync(acc, 0, sizeof(u64) * kSums, s));
  MC_CUDA_TRY(allow_smem((const void *)dense_kernel, smem));
  // A CTA per SM at most: each builds the matrix, which costs as much as
  // its share of the tasks.
  const int tasks = n * bit_words(n), warps = kDenseThreads / kWarp;
  dense_kernel<<<std::min(g->num_sms, (tasks + warps - 1) / warps), kDenseThreads, smem, s>>>(
      DenseGraph{g->rowptr, g->col, 0, n}, pattern, acc);
  MC_CUDA_TRY(cudaGetLastError());
  g->launches += 1;
  MC_CUDA_TRY(cudaEventRecord(g->ev[3], s));
  MC_CUDA_TRY(cudaMemcpyAsync(h, acc, sizeof(h), cudaMemcpyDeviceToHost, s));
  MC_CUDA_TRY(cudaStreamSynchronize(s));
  h[kX7] >>= 1;  // counted from both ends of its inner edge
  *out = motif_combine(pattern, h);
  return MC_OK;
}

// Row words of one graph of a batch: pairs, and three rows per two-path, bounded
// through the largest degree.
int64_t dense_work(int64_t n, int64_t nnz, int64_t max_degree) {
  return bit_words((int)n) * (n * n / 2 + 3 * nnz * max_degree / 2);
}

// Its parts: about 1 M words each, so that a batch's largest graphs do not end it
// on one SM, while few CTAs build a matrix again.  512 graphs (57 triangle jobs,
// 455 patterns on RMAT scale 5 to 8), whole batch: 1.50, 1.42, 1.33, 1.28, 1.24 and
// 1.23 ms at 2^15 to 2^20 words, 2.8 ms with one part per graph.  A batch whose
// words (total: of all its graphs) are fewer than that on every SM takes smaller
// parts, down to four times the matrix that each of them builds: a complete graph
// of 100 vertices alone took 5.3 ms in P5 on its one CTA, 1.2 so.  One that fills
// the SMs sixteen times over takes larger ones: 40 random graphs of 1,000
// vertices, 100,000 entries each, took 25 ms in P7 at 2^20, 9.6 in 64 parts.
int dense_parts(int64_t n, int64_t nnz, int64_t max_degree, int64_t total, int num_sms) {
  const int64_t own = 4 * n * bit_words((int)n);
  const int64_t share = std::max({std::min<int64_t>(total / num_sms, 1 << 20),
                                  total / (16 * num_sms), own, int64_t(1)});
  return (int)std::max<int64_t>(
      1, std::min<int64_t>(num_sms, dense_work(n, nnz, max_degree) / share));
}

int dense_batch_launch(const int64_t *rp, const int32_t *ci, const DenseTask *tasks, int num_tasks,
                       int largest, unsigned long long *acc, cudaStream_t s) {
  const size_t smem = dense_bytes(largest);
  MC_CUDA_TRY(allow_smem((const void *)dense_batch_kernel, dense_bytes(kDenseMax)));
  dense_batch_kernel<<<num_tasks, kBatchThreads, smem, s>>>(rp, ci, tasks, acc);
  MC_CUDA_TRY(cudaGetLastError());
  return MC_OK;
}

}  // namespace mc
