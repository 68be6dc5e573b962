// The route of a whole count by its graph's sizes alone.  Plain C++, so that the
// CPU tests compile it; the settings that force a route are read by the callers
// (dgraph.cu, motifs.cu).
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define MC_HOST_DEVICE __host__ __device__
#else
#define MC_HOST_DEVICE
#endif

namespace mc {

constexpr int kDenseMax = 1024;  // vertices of a graph that bit rows take

// The stages of the motif sums and the pairs of up neighbours walk vertices and
// entries in 32-bit loops of up to kMotifStride (4,096 blocks of 8 warps, or
// fewer, larger ones) past the last one.
constexpr int64_t kMotifMax = int64_t(1) << 30;
constexpr int64_t kMotifStride = int64_t(1) << 20;
static_assert(kMotifMax + kMotifStride <= INT32_MAX, "32-bit loops end");
inline bool motif_range(int64_t n, int64_t nnz) {
  return n > 0 && nnz > 0 && n <= kMotifMax && nnz <= kMotifMax;
}

// How a whole triangle count runs: over the DAG's tasks; on small graphs from
// bit rows, or from pairs of up neighbours in three launches.
enum class TriangleRoute { kDag, kBits, kPairs };
// Whole calls on a B200, us, bits / pairs / DAG: RMAT scale 10, edge factor 16:
// 74 / 49 / 144; scale 13, 16 (203,886 entries): - / 144 / 189; scale 13, 32
// (365,688): - / 336 / 195; Chung-Lu of 100,000, mean 5 (499,200): - / 78 / 190;
// mean 20 (1,960,194): - / 323 / 284.  The pairs grow with the square of the
// out-degrees, so beyond 2^18 entries they keep sparse graphs only, and none where
// the entries times the mean degree exceed 2^25 (pairs / DAG: complete graphs of
// 300, 400 and 512 vertices, 27, 64 and 134 million: 147 / 139, 364 / 157 and 798
// / 170; random ones of 1,200, 700 and 1,000 vertices, 29, 42 and 250 million: 171 /
// 137, 253 / 137 and 1,228 / 220; 64 x 2,000 complete bipartite, 32: 109 / 128).
// Bits win while one pass over the CSR is all there is (RMAT 8, edge factors 4,
// 16 and 64: 37 / 46 / 98, 47 / 45 / 135 and 62 / 47 / 137); each of their CTAs
// reads every entry, so dense graphs lose there too (complete graphs of 512 and
// 1,000: 358 and 1,307).
constexpr int64_t kBitVertices = 256, kBitEntries = 4096;
inline bool pairs_pay(int64_t n, int64_t nnz) {
  return motif_range(n, nnz) && nnz <= 1 << 19 && (nnz <= 1 << 18 || nnz <= 16 * n) &&
         nnz * nnz <= (n << 25);
}
inline TriangleRoute triangle_route_by_size(int64_t n, int64_t nnz) {
  if (!motif_range(n, nnz)) return TriangleRoute::kDag;
  if (n <= kBitVertices && nnz <= kBitEntries) return TriangleRoute::kBits;
  return pairs_pay(n, nnz) ? TriangleRoute::kPairs : TriangleRoute::kDag;
}

// P1..P8 from motif sums (over sparse stages, or, for graphs of at most
// kDenseMax vertices, from bit rows), or the per-edge formulas.  No motif sums
// above the degree at which the reference's 32-bit products could wrap (its
// counts are then no subgraph counts).
//
// By size (measured on a B200, whole calls, formula / bit rows / sparse, ms):
//  - bit rows take P2 and P5 up to 512 vertices (RMAT scale 8, edge factor 8:
//    1.39 / 0.14 / 0.41 and 0.32 / 0.14 / 0.41; at 1,024 vertices the two
//    differ by -15% to +50%), and every pattern up to 64, where the sparse
//    stages are launches alone (RMAT 6, P6: 0.068 / 0.055 / 0.079);
//  - the per-edge formulas, one launch against five or more, keep P4 to P8
//    on small graphs of low degree (the limits below), where every set of an
//    edge is a warp or two: Chung-Lu of 10,001 vertices, mean 4, cap 40 (39,942
//    entries, degree 61), P4 to P8: 0.094, 0.093, 0.081, 0.081 and 0.094 against
//    0.122, 0.139, 0.096, 0.091 and 0.091 sparse; of 30,001 (119,934 entries):
//    0.172, 0.167, 0.146, 0.132 and 0.170 against 0.165, 0.165, 0.107, 0.097 and
//    0.097.  Hubs turn it: 3,001 vertices, mean 4, cap 200 (11,186 entries,
//    degree 165), P5 to P8: 0.52, 1.20, 0.33 and 0.71 against 0.37, 0.10, 0.09
//    and 0.09.
//  - the formulas keep near-complete graphs (formula / default without them:
//    complete graphs of 100, 200 and 512 vertices, P1: 0.23 / 0.33, 0.70 / 0.53,
//    1.3 / 5.4; P2: 0.86 / 1.5, 3.8 / 6.3, 5.7 / 74; P3: 0.23 / 1.7, 0.64 / 9.0, 1.07 /
//    431; P4 of 128: 0.07 / 0.45; P5, P6 and P8 of 64: 0.21, 0.25 and 0.17 / 0.52; 90%
//    of all edges, 400 vertices, P1 to P4: 0.77 / 2.1, 17 / 24, 13 / 91, 2.7 / 2.3).
//    Cliques in larger graphs show on the way (probe_percent, motif_outweighs).
enum class PatternRoute { kFormula, kDense, kSparse };
inline bool motif_sums_apply(int64_t n, int64_t nnz, int64_t max_degree) {
  return motif_range(n, nnz) && max_degree <= 46340;
}
inline PatternRoute pattern_route_by_size(int64_t n, int64_t nnz, int64_t max_degree,
                                          int pattern) {
  if (!motif_sums_apply(n, nnz, max_degree)) return PatternRoute::kFormula;
  // In percent of all entries: near-complete graphs, where the ends of an edge share
  // almost every neighbour and the formulas have next to nothing to test.
  const auto filled = [&](int percent) {
    return 100.0 * (double)nnz >= percent * (double)n * (double)(n - 1);
  };
  switch (pattern) {
    case 1:
      if ((n >= 256 && filled(78)) || (n > 64 && n <= 140 && filled(95)))
        return PatternRoute::kFormula;
      break;
    case 2:
      if ((n >= 64 && filled(97)) || (n >= 300 && filled(88))) return PatternRoute::kFormula;
      break;
    case 3:
      if ((n >= 32 && filled(88)) || (n >= 300 && filled(75))) return PatternRoute::kFormula;
      break;
    case 4:
      if (filled(93)) return PatternRoute::kFormula;
      break;
    case 6:
      if (n >= 32 && n <= 128 && filled(93)) return PatternRoute::kFormula;
      break;
    case 7: break;
    default:  // 5, 8
      if (n >= 32 && n <= 140 && filled(97)) return PatternRoute::kFormula;
  }
  if (n <= 64 && pattern != 4) return PatternRoute::kDense;
  if (n <= 512 && (pattern == 2 || pattern == 5)) return PatternRoute::kDense;
  struct Limit {
    int64_t degree, entries;
  };
  constexpr Limit kFormulaUpTo[] = {{100, 65536}, {80, 98304}, {72, 49152}, {80, 65536}, {64, 16384}};
  if (pattern >= 4) {
    const Limit &up = kFormulaUpTo[pattern - 4];
    if (max_degree <= up.degree && nnz <= up.entries) return PatternRoute::kFormula;
    if (pattern == 4 && nnz <= 12288) return PatternRoute::kFormula;
  }
  return PatternRoute::kSparse;
}

// Graphs above 256 vertices that may be unions of cliques, by sizes: P1 to P4 then
// sample two-paths beside the first stage, and go to the formulas when this many
// percent of them are closed; 0: no samples.  Formula / sums, ms: 20 complete
// graphs of 128 vertices, P1 to P4: 0.39 / 1.3, 1.6 / 47, 0.36 / 24, 0.44 / 1.5; 20
// random ones of 150 with 80% of all edges: 0.88 / 1.3, 11 / 29, 7.4 / 14.5, 1.3 /
// 1.5; with 50%: 0.39 / 0.45, 4.5 / 4.8, 2.6 / 2.0, 0.87 / 0.54; one of 800, 80%, P4:
// 31 / 11, 98%: 6.4 / 18; 2,000 complete graphs of 20, P1 to P4: 0.21 / 0.32, 0.74 /
// 1.8, 0.18 / 1.2, 0.60 / 0.36.
inline int probe_percent(int64_t n, int64_t nnz, int64_t max_degree, int pattern) {
  if (pattern > 4 || n <= 256 || max_degree * n > 8 * nnz) return 0;
  return pattern == 4 ? (nnz >= 32 * n ? 88 : 0) : (nnz >= 16 * n ? 78 : 0);
}
constexpr int64_t kEstimateAbove = 512;  // vertices from which motif_outweighs is asked

// A batch's pattern job (P1..P8) by bit rows, or by the persistent per-edge
// kernel: whichever is shorter on a full GPU, in ns per graph.  The bit rows take
// the ANDs of all vertex pairs; the formulas some ns per entry and, by pattern, a
// part of the sum of squared degrees (and, of P1, of the largest one: a hub's star
// is one warp's).  Fitted to 40 copies of one graph, us per graph, formulas / bit
// rows: a path of 1,000 vertices, P4 and P7: 2 / 28 and 1.5 / 10; random graphs of
// 1,000 vertices, 10,034 entries, P2, P4, P7: 82 / 33, 13 / 32, 8 / 17; of 500,
// 12,418 entries: 320 / 14, 23 / 8, 10 / 8; a star of 1,000, P1, P4, P8: 130 / 15,
// 12 / 28, 50 / 15; complete graphs of 100, P2 to P4 (no two neighbours of an edge
// apart, which the sizes do not show otherwise): 25 / 150, 16 / 142, 14 / 21.
MC_HOST_DEVICE constexpr int bit_words(int64_t n) {
  return n <= 32 ? 1 : n <= 64 ? 2 : n <= 128 ? 4 : n <= 256 ? 8 : (int)((n + 31) / 32);
}
inline bool batch_takes_bits(int64_t n, int64_t nnz, int64_t max_degree, int64_t degree_squares,
                             int pattern) {
  if (n > kDenseMax) return false;
  if (pattern >= 2 && pattern <= 4 && n >= 24 && 10 * nnz >= 9 * n * (n - 1)) return false;
  const double pairs = 0.5 * (double)n * (double)n * bit_words(n);
  const double bits = pairs * (pattern == 1 || pattern >= 7 ? 0.0011 : 0.002);
  constexpr double kPerSquare[] = {0.013, 0.75, 0.57, 0.012, 0.06, 0.01, 0.002, 0.04};
  double formula = (pattern == 7 ? 0.8 : 1.1) * (double)nnz +
                   kPerSquare[pattern - 1] * (double)degree_squares;
  if (pattern == 1) formula += 0.13 * (double)max_degree * (double)max_degree;
  return bits <= formula;
}

}  // namespace mc
