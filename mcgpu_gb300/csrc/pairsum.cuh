// pairsum.cuh -- the pieces of the FP64 system-energy kernels: a CTA takes a
// group of up to kPsGroup consecutive molecules m and sums E(m, j > m).
//
// Every candidate j is loaded once for the whole group (one load of its
// primaries for kPsGroup tests; a CTA per molecule loaded every candidate for
// every molecule, which bounded the sum on large boxes), the in-range (m, j)
// go to a ring per warp, and full rings are evaluated as items (entry,
// neighbour atom) that fill the lanes, as the trial-move batches do
// (kernels.cuh): the FP64 pipe is what is left to bound the kernel.
#pragma once

#include "kernels.cuh"

namespace mcgpu {

constexpr int kPsGroup = 8;        // molecules per CTA at most
constexpr int kPsThreads = 128;
constexpr int kPsWarps = kPsThreads / 32;
constexpr int kPsPitch = kMaxA + 1;  // odd pitch: lanes on different molecules of
                                     // the group read different banks
static_assert(kPsGroup == 8, "ring entries hold the molecule in three bits");

// The group's staged atoms: positions, blending factors (blend64), charge.
struct PsGroup {
  double x[kPsGroup * kPsPitch], y[kPsGroup * kPsPitch], z[kPsGroup * kPsPitch];
  double sd[kPsGroup * kPsPitch], ed[kPsGroup * kPsPitch], qd[kPsGroup * kPsPitch];
  int len[kPsGroup];
  int ring[kPsWarps][kRing];
  double red[kPsWarps];
};

// Whether the group's n staged molecules have one length and the same skipped
// sites, as the lanes of ps_items must for pair_sum64's votes.  Every thread of the
// CTA calls it once the rows are staged, and gets the same answer.
__device__ __forceinline__ bool ps_alike(const PsGroup& G, int n) {
  if (n == 1) return true;
  bool differ = false;
  for (int g = 1; g < n; g++) {
    differ = differ || G.len[g] != G.len[0];
    for (int i = threadIdx.x; i < min(G.len[0], G.len[g]); i += kPsThreads)
      differ = differ || blend_skipped(G.sd[g * kPsPitch + i]) != blend_skipped(G.sd[i]);
  }
  return !__syncthreads_or(differ);
}

// Evaluates `count` (1..32) ring entries (j << 3 | group molecule) from
// `head`: this lane's share of the sum.  rows: len(j), start(j) of molecule
// j and its atoms' position and factors.  alike: ps_alike's answer; FINE: pair_sum64's.
template <bool FINE, class Rows>
__device__ __forceinline__ double ps_items(const PsGroup& G, const Rows& rows, const int* rj,
                                           int head, int count, int lane, bool alike, double Lx,
                                           double Ly, double Lz) {
  int len = 0;
  if (lane < count) len = rows.len(rj[(head + lane) & (kRing - 1)] >> 3);
  const int len0 = __shfl_sync(~0u, len, 0);
  const bool same = __all_sync(~0u, lane >= count || len == len0);
  int pref = len, total;
  if (same) {
    total = count * len0;
  } else {
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int v = __shfl_up_sync(~0u, pref, off);
      if (lane >= off) pref += v;
    }
    total = __shfl_sync(~0u, pref, 31);
    pref -= len;
  }
  double acc = 0.0;
  for (int base = 0; base < total; base += 32) {
    const int it = base + lane;
    int e, k;
    if (same) {
      // atom by atom over the entries: the lanes of a round share the atom
      k = it / count;
      e = it - k * count;
    } else {
      e = 0;
#pragma unroll
      for (int step = 16; step > 0; step >>= 1) {
        const int at = e + step;
        const int v = __shfl_sync(~0u, pref, at & 31);
        if (at < count && v <= it) e = at;
      }
      k = it - __shfl_sync(~0u, pref, e);
    }
    if (it >= total) continue;
    const int jm = rj[(head + e) & (kRing - 1)];
    const int o = (jm & 7) * kPsPitch;
    double xb, yb, zb, sb, eb, qb;
    rows.atom(rows.start(jm >> 3) + k, xb, yb, zb, sb, eb, qb);
    if (alike)
      acc += pair_sum64<true, FINE>(G.x + o, G.y + o, G.z + o, G.sd + o, G.ed + o, G.qd + o, G.len[0],
                                    xb, yb, zb, sb, eb, qb, Lx, Ly, Lz);
    else
      acc += pair_sum64<false, FINE>(G.x + o, G.y + o, G.z + o, G.sd + o, G.ed + o, G.qd + o,
                                     G.len[jm & 7], xb, yb, zb, sb, eb, qb, Lx, Ly, Lz);
  }
  return acc;
}

// Block sum of acc in a fixed order, valid in thread 0.
__device__ __forceinline__ double ps_block_sum(PsGroup& G, double acc) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(~0u, acc, off);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) G.red[threadIdx.x >> 5] = acc;
  __syncthreads();
  double sum = 0.0;
  if (threadIdx.x == 0)
    for (int w = 0; w < kPsWarps; w++) sum += G.red[w];
  return sum;
}

// Molecules per CTA for a box of n: as many as leave eight CTAs for each of the
// 152 SMs (their shares of the in-range pairs are uneven; 286 CTAs of 7 of
// 1,999 16-atom molecules left the busiest SM 1.6 times the mean).  In a batch the
// other chains fill the SMs, and a chain's groups are larger: 152 chains of 2,000
// waters 3.05 ms, 6.6 by the boxes' rule (one chain of 700: 76 us, 54).  Either way
// the groups follow from the chain's own size -- the card's 152 SMs are a constant
// here -- so its sum is the same alone and among others.
constexpr int kPsPerBox = 152 * 8, kPsPerBatch = 128;
__host__ __device__ inline int ps_group(int n, int per) {
  const int g = n / per;
  return g < 1 ? 1 : g > kPsGroup ? kPsGroup : g;
}

}  // namespace mcgpu
