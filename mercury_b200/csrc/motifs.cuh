// Motif sums and their combination into P1..P8: shared by the sparse route
// (motifs.cu, which derives them) and the bit-row route of small graphs
// (dense.cu).
#pragma once
#include "device_common.cuh"

namespace mc {

using u64 = unsigned long long;

// Sums over the graph, modulo 2^64.
enum Sum : int {
  kVd3, kVd4, kVt2, kVtd,                  // vertices: C(d,3), C(d,4), C(t,2), t d
  kD, kC3, kEp4, kEfork, kEdart,           // edges
  kT, kCricket, kBull, kLolli, kKite, kGem,  // triangles
  kKd, kKa, kKk, kK4, kK5,                 // with common neighbours; cliques
  kC4, kC4d, kC4a, kX7, kW4, kK23,         // 4-cycles and beyond
  kA2,                                     // edges: a^2, where it is taken ahead of kD
  kSums
};

// What a pattern needs beyond a and the vertex and edge sums.
enum Need : unsigned {
  kNeedTau = 1u,    // triangle sums with k (else K4 alone)
  kNeedD2 = 2u,     // sum of (d - 1) over each neighbourhood
  kNeedT = 4u,      // C(t, 2) over the triangles per vertex
  kNeedC4 = 8u,     // 4-cycles, each counted at its highest vertex
  kNeedPairs = 16u, // every pair's common neighbours (C4 counted twice)
  kNeedW4 = 32u,
  kNeedK23 = 64u,   // with kNeedPairs: K2,3 and degrees on 4-cycles
  kNeedWork = 128u, // motif_outweighs is asked
};

__host__ __device__ constexpr unsigned motif_needs(int pattern) {
  return pattern == 1   ? 0u
         : pattern == 2 ? kNeedTau | kNeedD2 | kNeedT | kNeedPairs | kNeedW4 | kNeedK23 | kNeedWork
         : pattern == 3 ? kNeedTau | kNeedT | kNeedW4 | kNeedWork
         : pattern == 4 ? kNeedC4
         : pattern == 5 ? kNeedTau | kNeedPairs | kNeedW4 | kNeedWork
         : pattern == 6 ? kNeedTau | kNeedW4
                        : (unsigned)kNeedTau;
}

__device__ __forceinline__ u64 c2(u64 x) { return x * (x - 1) / 2; }  // 0 at 0 and 1
__device__ __forceinline__ u64 c3(long long x) {
  return x < 3 ? 0ull : (u64)x * (u64)(x - 1) / 2 * (u64)(x - 2) / 3;
}
// C(x, 4) below 2^64 for x up to 46,341: C(x, 3) (x - 3) is at most 8e17.
__device__ __forceinline__ u64 c4(long long x) {
  return x < 4 ? 0ull : c3(x) * (u64)(x - 3) / 4;
}

// Bits above position j of a row's word w.
__device__ __forceinline__ unsigned above(int j, int w) {
  const int s = j + 1 - 32 * w;
  return s <= 0 ? kFull : (s >= 32 ? 0u : kFull << s);
}

// P2, P3 and P5 above 512 vertices, known once the triangles are: the wheel stage
// and X7 visit the sum of a^2 over the entries, some cliques' whole cost, while the
// per-edge formulas test the neighbours that an edge's ends do not share (x and y
// of them), next to none in a clique.  True where the formulas are the shorter
// way, by the sums of a^2, a, x^2 and a x over the entries, which follow from those
// of the vertices (an entry of v has x = d - 1 - a, and a adds up to 2 t along v's
// row).  The weights, in ps, are fitted to whole calls (formulas / sums, ms): three
// complete graphs of 400 vertices, P2, P3, P5: 10 / 864, 1.3 / 395, 109 / 868; one of
// 300 beside the Chung-Lu graph of 100,000: 34 / 445, 10 / 73, 25 / 436; a random
// graph of 800 vertices with 70% of all edges: 645 / 1,069, 542 / 251, above 2,500 /
// 1,066; 2,000 vertices, 10%: 56 / 4.4, 23 / 2.0, 96 / 4.3; the Chung-Lu graph of
// 20,000 with hubs of 5,000: above 2,500 / 140, 24 and 138.
constexpr u64 kOutweighFloor = 20000000;  // some 0.1 ms
__host__ __device__ inline bool motif_outweighs(int pattern, const u64 *s) {
  const u64 a = 6 * s[kT], a2 = s[kA2] ? 2 * s[kA2] : 4 * s[kD] + a;
  if (a2 < kOutweighFloor) return false;
  const u64 da = 2 * (s[kVtd] - 3 * s[kT]);  // sum of (d - 1) a
  const u64 d3 = 6 * s[kVd3] + a2;           // of (d - 1)^2 + a^2, but for sum of d (d - 1)
  const u64 q = (d3 > 2 * da ? d3 - 2 * da : 0) >> 6, m = (da > a2 ? da - a2 : 0) >> 6;
  const u64 e = a >> 6, w = a2 >> 6;
  switch (pattern) {
    case 2: return 15 * w > 5 * q + 19 * m + 80 * e;
    case 3: return 6 * w > q + 16 * m + 8 * e;
    case 5: return 20 * w > 2 * q + 200 * m + 500 * e;
    default: return false;
  }
}

// Per-block totals of the sums a kernel adds to.
struct BlockSums {
  u64 *s;
  __device__ __forceinline__ void init() const {
    for (int i = threadIdx.x; i < kSums; i += blockDim.x) s[i] = 0;
    __syncthreads();
  }
  // Every lane of the warp takes part.
  __device__ __forceinline__ void add(int which, u64 v) const {
    v = warp_sum_u64(v);
    if ((threadIdx.x & (kWarp - 1)) == 0 && v) atomicAdd(s + which, v);
  }
  __device__ __forceinline__ void flush(u64 *acc) const {
    __syncthreads();
    for (int i = threadIdx.x; i < kSums; i += blockDim.x)
      if (s[i]) atomicAdd(acc + i, s[i]);
  }
};

// The pattern's count from the sums, modulo 2^64: non-induced counts of the
// subgraphs on five vertices that contain the pattern, each with the signed
// number of the pattern's copies in it.
__host__ __device__ inline u64 motif_combine(int pattern, const u64 *s) {
  const u64 K4 = s[kK4], K5 = s[kK5], D = s[kD], T = s[kT];
  // C4 family: the ordered walk counts each cycle once, the pair walk twice.
  const u64 ka = s[kKa] - 24 * K4;   // 2 x K5 minus a path of 3 vertices
  const u64 kd = s[kKd] - 36 * K4;   // 3 x tailed K4
  const u64 third = 0xaaaaaaaaaaaaaaabull;  // 1/3 modulo 2^64
  const u64 tk4 = kd * third;
  const u64 claw = s[kVd3] - s[kVtd] + 6 * T + 2 * D - 4 * K4;
  const u64 gem = s[kGem] - 12 * K4, kite = s[kKite] - 12 * K4;
  const u64 butterfly = s[kVt2] - 2 * D;
  switch (pattern) {
    case 1: return claw;
    case 2:
      // banner = C4d / 2 - 8 (C4 / 2) - 2 D and house = C4a / 2 - 4 D, with
      // the doubled sums of the pair walk.
      return s[kEfork] - 2 * s[kCricket] - 2 * s[kBull] - s[kLolli] - (s[kC4d] - 8 * s[kC4] - 4 * D) +
             6 * s[kK23] + 5 * s[kEdart] + 4 * kite + (2 * s[kC4a] - 16 * D) + 4 * butterfly -
             10 * gem - 10 * s[kX7] + 20 * s[kW4] - 3 * kd + 10 * ka - 12 * s[kC3] - 36 * s[kKk] +
             60 * K5;
    case 3: {
      const u64 star = s[kVd4] - s[kCricket] + s[kEdart] + butterfly - gem + s[kW4] - tk4 -
                       2 * s[kC3] - 3 * s[kKk] + 5 * K5;  // + 2 (K5 - P3), added below
      return 4 * star + 4 * ka + 3 * claw;
    }
    case 4: return s[kEp4] - 4 * s[kC4] + 4 * D - 12 * K4;
    case 5:
      return 2 * s[kBull] - 4 * s[kEdart] - 4 * kite - (s[kC4a] - 8 * D) + 10 * gem + 8 * s[kX7] -
             24 * s[kW4] + 4 * kd - 14 * ka + 12 * s[kC3] + 60 * s[kKk] - 120 * K5;
    case 6: {
      const u64 paw = s[kVtd] - 6 * T - 4 * (D - 6 * K4) - 12 * K4;
      return 2 * paw + 2 * s[kEdart] - 4 * gem + 8 * s[kW4] - 2 * kd + 10 * ka - 12 * s[kC3] -
             48 * s[kKk] + 120 * K5;
    }
    case 7: return 2 * s[kC3] - ka + 6 * s[kKk] - 20 * K5;
    default: return kd - 3 * ka + 18 * s[kKk] - 60 * K5;
  }
}

}  // namespace mc
