// mpm_pairs.cuh -- the node-sorted pair list of the FP64 forms: for every node
// (SGMP: centre node) its (particle, slot) pairs in ascending order, which is
// the reference's summation order.
//
// The locate kernel counts the pairs per node; here the counts are scanned into
// segment ends (mpm_sort.cuh), every pair takes a place in its node's segment
// through a per-node fill counter, and each segment is put in ascending order of
// (particle << 5 | slot) by one warp (a bitonic network over its registers up to
// 256 pairs), one block beyond. The result is what a stable radix sort of all
// pairs by node gives, whatever order the placement's atomics ran in. A radix
// sort moved 27 slots per particle (unused ones under a sentinel) five times
// through memory; this moves each used pair once. One step's pairs, before and
// after, GB300: slope 159 k particles 115 -> 58 us, dam break 31 k
// 50 -> 31, Taylor bar 17 k 39 -> 20, Cook 5.8 k 40 -> 20. The order in which
// the transfers take the nodes is made beside it (1.5 us of each).
#pragma once

#include "mpm_kernels.cuh"
#include "mpm_sort.cuh"

namespace mpm {

__global__ void k_zero_words(int* w, long long n) {
  chain_entry();
  for (long long i = gtid(); i < n; i += (long long)gridDim.x * blockDim.x) w[i] = 0;
}

// The order the transfers take the nodes in (pair_walk): by classes of the
// number of eights of pairs in a segment, longest first, empty segments
// last, about the grid's order within a class. The order has no bearing on
// results.
__device__ __forceinline__ int walk_class(int n) {
  return kWalkClasses - 1 - min((n + 7) / 8, kWalkClasses - 1);
}

// per-node counts scanned in place into segment ends, the fill counters and
// the class counters (nodes of each class, then nodes placed) zeroed on the way
struct PairScan {
  using T = int;
  using Op = bm::ScanSum;
  int* seg;
  int* fill;
  int* wcnt;
  long long n;
  __device__ __forceinline__ int load(long long g) const { return seg[g]; }
  __device__ __forceinline__ void store(long long g, int v, int) const {
    seg[g] = v;
    fill[g] = 0;
    if (g == 0)
      for (int c = 0; c < 2 * kWalkClasses; ++c) wcnt[c] = 0;
  }
};

constexpr int kWarpPairs = 256;  // longest segment a warp orders

// a place in its node's segment for each pair (thread = particle; rows of blocks,
// one per slot: every pair's atomic in flight at once). Neighbouring particles
// often share a slot's node: one atomic per node and warp. The blocks after the
// last row, by the number of nodes, count the nodes of each class.
__global__ void __launch_bounds__(256) k_pair_place(const int* snode, const int* seg, int* fill, unsigned* val,
                                                    long long np, int K, long long nk, int* wcnt, int* nbig) {
  chain_entry();
  const int row = (int)((np + 255) / 256), lane = threadIdx.x & 31;
  const int k = min((int)blockIdx.x / row, K), at = blockIdx.x - k * row;  // (slot K: the counting blocks)
  const long long p = (long long)at * 256 + threadIdx.x;
  if (p == 0 && k == 0) *nbig = 0;
  if (k == K) {
    __shared__ int hist[kWalkClasses];
    if (threadIdx.x < kWalkClasses) hist[threadIdx.x] = 0;
    __syncthreads();
    for (long long n0 = p - threadIdx.x; n0 < nk; n0 += (long long)(gridDim.x - K * row) * 256) {
      const long long n = n0 + threadIdx.x;
      const int c = n < nk ? walk_class(seg[n] - (n == 0 ? 0 : seg[n - 1])) : -1;
      const unsigned grp = __match_any_sync(0xffffffffu, c);
      if (c >= 0 && lane == __ffs(grp) - 1) atomicAdd(&hist[c], __popc(grp));
    }
    __syncthreads();
    if (threadIdx.x < kWalkClasses && hist[threadIdx.x]) atomicAdd(&wcnt[threadIdx.x], hist[threadIdx.x]);
    return;
  }
  const int nd = p < np ? snode[k * np + p] : -1;
  const unsigned grp = __match_any_sync(0xffffffffu, nd);
  const int leader = __ffs(grp) - 1, rank = __popc(grp & ((1u << lane) - 1u));
  int base = 0;
  if (lane == leader && nd >= 0) base = atomicAdd(&fill[nd], __popc(grp));
  base = __shfl_sync(0xffffffffu, base, leader);
  if (nd >= 0) val[(nd == 0 ? 0 : seg[nd - 1]) + base + rank] = ((unsigned)p << 5) | (unsigned)k;
}

// ascending order of n <= 32 R values at v by one warp, lane l holding the
// elements l, l + 32, ...: a bitonic network, comparators at distances below
// 32 across lanes, the others within a lane's registers
template <int R>
__device__ __forceinline__ void warp_order(unsigned* v, int n) {
  const int lane = threadIdx.x & 31;
  unsigned x[R];
#pragma unroll
  for (int r = 0; r < R; ++r) x[r] = r * 32 + lane < n ? v[r * 32 + lane] : 0xffffffffu;
#pragma unroll
  for (int k = 2; k <= 32 * R; k <<= 1) {
#pragma unroll
    for (int s = k >> 1; s > 0; s >>= 1) {
      if (s >= 32) {
        const int d = s >> 5;
#pragma unroll
        for (int r = 0; r < R; ++r) {
          if (r & d) continue;
          const bool up = ((r * 32 + lane) & k) == 0;
          const unsigned a = x[r], b = x[r | d];
          x[r] = up ? min(a, b) : max(a, b);
          x[r | d] = up ? max(a, b) : min(a, b);
        }
      } else {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const bool up = ((r * 32 + lane) & k) == 0, low = (lane & s) == 0;
          const unsigned o = __shfl_xor_sync(0xffffffffu, x[r], s);
          x[r] = up == low ? min(x[r], o) : max(x[r], o);
        }
      }
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (r * 32 + lane < n) v[r * 32 + lane] = x[r];
}

// each node's segment in ascending order, a warp taking share (1 .. 32) nodes,
// of which it looks at all together; segments longer than kWarpPairs are listed
// for k_pair_long. share keeps the warps of a large grid, most of whose nodes
// have nothing to order, to about kOrderWarps.
constexpr long long kOrderWarps = 65536;
inline int order_share(long long nk) {
  int s = 1;
  while (s < 32 && nk > s * kOrderWarps) s *= 2;
  return s;
}
__global__ void k_pair_order(const int* seg, long long nk, unsigned* val, int* big, int* nbig, int share) {
  chain_entry();
  const int lane = threadIdx.x & 31;
  const long long k0 = (gtid() >> 5) * share, kl = k0 + lane;
  const bool own = lane < share && kl < nk;
  const int al = own && kl > 0 ? seg[kl - 1] : 0, nl = own ? seg[kl] - al : 0;
  unsigned rest = __ballot_sync(0xffffffffu, nl > 1);
  while (rest) {
    const int l = __ffs(rest) - 1;
    rest &= rest - 1;
    const int a = __shfl_sync(0xffffffffu, al, l), n = __shfl_sync(0xffffffffu, nl, l);
    unsigned* v = val + a;
    if (n <= 32) warp_order<1>(v, n);
    else if (n <= 64) warp_order<2>(v, n);
    else if (n <= 128) warp_order<4>(v, n);
    else if (n <= kWarpPairs) warp_order<8>(v, n);
    else if (lane == 0) big[atomicAdd(nbig, 1)] = (int)(k0 + l);
  }
}

// the segments listed in big in ascending order, and the nodes into walk
__global__ void __launch_bounds__(bm::kSortThreads) k_pair_long(const int* seg, unsigned* val, const int* big,
                                                                const int* nbig, long long nk, int* wcnt, int* walk) {
  chain_entry();
  __shared__ unsigned sm[bm::kSmemSeg];
  bm::sort_long(seg, val, big, nbig, sm, [](int, unsigned* v, int n) { bm::block_bitonic(v, n); });

  constexpr int NW = bm::kSortThreads / 32;
  static_assert(kWalkClasses == 32, "a lane per class");
  __shared__ int cnt[NW][kWalkClasses], base[kWalkClasses];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int start = 0;  // of the lane's class (first warp)
  if (warp == 0) {
    const int own = wcnt[lane];
    start = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, start, o);
      if (lane >= o) start += u;
    }
    start -= own;
  }
  for (long long n0 = (long long)blockIdx.x * bm::kSortThreads; n0 < nk; n0 += (long long)gridDim.x * bm::kSortThreads) {
    const long long n = n0 + threadIdx.x;
    const int c = n < nk ? walk_class(seg[n] - (n == 0 ? 0 : seg[n - 1])) : -1;
    const unsigned grp = __match_any_sync(0xffffffffu, c);
    cnt[warp][lane] = 0;
    __syncwarp();
    if (c >= 0 && lane == __ffs(grp) - 1) cnt[warp][c] = __popc(grp);
    __syncthreads();
    if (warp == 0) {  // lane = class: the warps' offsets, and the tile's place in the class
      int tot = 0;
      for (int q = 0; q < NW; ++q) {
        const int v = cnt[q][lane];
        cnt[q][lane] = tot;
        tot += v;
      }
      base[lane] = start + (tot ? atomicAdd(&wcnt[kWalkClasses + lane], tot) : 0);
    }
    __syncthreads();
    if (c >= 0) walk[base[c] + cnt[warp][c] + __popc(grp & ((1u << lane) - 1u))] = (int)n;
    __syncthreads();
  }
}

}  // namespace mpm
