// mpm_sort.cuh -- the batched engine's counting sort of particles by sort
// key, and the tile scans it uses. It runs on the scenes whose order has
// become stale (step_tick), whose keys and particles are numbered without gaps;
// the others take no part.
//
// (On a scene's first step the particles are in the deck's order.) Later on
// they arrive in the last sort's key order with a few per cent moved
// to a neighbouring key, so a key's particles are nearly contiguous already
// and a key holds a handful of particles (about 8 at 8 particles per cell).
// The sort is a counting sort: per-key counts (taken by sort_keys),
// an inclusive scan of the counts into segment ends, placement of every
// particle into its key's segment through a per-key fill counter (one
// atomic per key and warp), then the order inside each segment restored to
// ascending particle index -- the stable order -- by one thread per short
// segment and one block per long one. The result is the permutation a
// stable radix sort by key would give, whatever order the placement atomics
// ran in, so the step stays deterministic.
#pragma once

#include <climits>

namespace mpm {
namespace bm {

// ------------------------------------------------------------------ scans
// Inclusive scans in tiles of kScanTile items: per-tile totals, an exclusive
// scan of the totals by one block, then each tile scanned with its carry. A
// source policy S gives the value type (S::T), the operation (S::Op), the
// item count, the load of item g and the store of its inclusive prefix; a
// block reads its whole tile before it stores into it and touches no other
// tile, so in-place scans are safe.
constexpr int kScanThreads = 256;
constexpr int kScanItems = 16;
constexpr long long kScanTile = (long long)kScanThreads * kScanItems;

inline long long scan_tiles(long long n) { return (n + kScanTile - 1) / kScanTile; }

struct ScanSum {
  template <class T>
  __device__ __forceinline__ static T id() { return (T)0; }
  template <class T>
  __device__ __forceinline__ static T op(T a, T b) { return a + b; }
};
struct ScanMax {
  template <class T>
  __device__ __forceinline__ static T id() { return (T)INT_MIN; }
  template <class T>
  __device__ __forceinline__ static T op(T a, T b) { return a > b ? a : b; }
};

// Block-wide scan of one value per thread: thr[t] receives the inclusive
// prefix of threads 0..t; returns the exclusive prefix of this thread. Every
// thread of the block calls it; blockDim.x is a multiple of 32, at most 1024.
template <class T, class Op>
__device__ __forceinline__ T block_scan(T v, T* thr, T* wsum) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const T u = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v = Op::op(u, v);
  }
  if (lane == 31) wsum[warp] = v;
  __syncthreads();
  if (warp == 0) {
    T w = lane < nw ? wsum[lane] : Op::template id<T>();
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const T u = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w = Op::op(u, w);
    }
    if (lane < nw) wsum[lane] = w;
  }
  __syncthreads();
  if (warp > 0) v = Op::op(wsum[warp - 1], v);
  thr[threadIdx.x] = v;
  __syncthreads();
  const T ex = threadIdx.x ? thr[threadIdx.x - 1] : Op::template id<T>();
  __syncthreads();  // thr and wsum are reused by the next call
  return ex;
}

// tile t into shared memory (coalesced); each thread then owns kScanItems
// consecutive items
template <class S>
__device__ __forceinline__ void load_tile(const S& src, long long t, typename S::T* tile) {
  const long long base = t * kScanTile;
  for (int e = threadIdx.x; e < kScanTile; e += blockDim.x) {
    const long long g = base + e;
    tile[e] = g < src.n ? src.load(g) : S::Op::template id<typename S::T>();
  }
  __syncthreads();
}

template <class S>
__global__ void __launch_bounds__(kScanThreads) ks_tile_total(S src, typename S::T* tiles) {
  chain_entry();
  using T = typename S::T;
  using Op = typename S::Op;
  __shared__ T tile[kScanTile];
  __shared__ T thr[kScanThreads], wsum[32];
  load_tile(src, blockIdx.x, tile);
  T v = Op::template id<T>();
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) v = Op::op(v, tile[threadIdx.x * kScanItems + k]);
  block_scan<T, Op>(v, thr, wsum);
  if (threadIdx.x == 0) tiles[blockIdx.x] = thr[kScanThreads - 1];
}

// exclusive scan of the nt tile totals in place, by one block of
// kScanThreads threads
template <class T, class Op>
__global__ void __launch_bounds__(kScanThreads) ks_tile_prefix(T* tiles, long long nt) {
  chain_entry();
  __shared__ T thr[kScanThreads], wsum[32];
  T carry = Op::template id<T>();
  for (long long b0 = 0; b0 < nt; b0 += kScanThreads) {
    const long long t = b0 + threadIdx.x;
    const T v = t < nt ? tiles[t] : Op::template id<T>();
    const T ex = block_scan<T, Op>(v, thr, wsum);
    const T total = thr[kScanThreads - 1];  // thr is not written again before the barrier below
    if (t < nt) tiles[t] = Op::op(carry, ex);
    carry = Op::op(carry, total);
    __syncthreads();
  }
}

// FUSED: tiles hold the tile totals themselves (no ks_tile_prefix launch):
// every block reduces the totals of the tiles before it (for up to
// kFusedTiles tiles, a few loads per thread)
constexpr long long kFusedTiles = 4096;
template <class S, bool FUSED>
__global__ void __launch_bounds__(kScanThreads) ks_tile_scan(S src, const typename S::T* tiles) {
  chain_entry();
  using T = typename S::T;
  using Op = typename S::Op;
  __shared__ T tile[kScanTile];
  __shared__ T thr[kScanThreads], wsum[32];
  T carry;
  if (FUSED) {
    T v = Op::template id<T>();
    for (long long t = threadIdx.x; t < blockIdx.x; t += blockDim.x) v = Op::op(v, tiles[t]);
    block_scan<T, Op>(v, thr, wsum);
    carry = thr[kScanThreads - 1];  // (thr is rewritten only after the next scan's first barrier)
  } else {
    carry = tiles[blockIdx.x];
  }
  load_tile(src, blockIdx.x, tile);
  T r[kScanItems];
  T v = Op::template id<T>();
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    v = Op::op(v, tile[threadIdx.x * kScanItems + k]);
    r[k] = v;
  }
  const T pre = Op::op(carry, block_scan<T, Op>(v, thr, wsum));
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) tile[threadIdx.x * kScanItems + k] = Op::op(pre, r[k]);
  __syncthreads();
  const long long base = (long long)blockIdx.x * kScanTile;
  for (int e = threadIdx.x; e < kScanTile; e += blockDim.x) {
    const long long g = base + e;
    if (g < src.n) src.store(g, tile[e], e ? tile[e - 1] : carry);
  }
}

// an int array scanned into another (or itself); store(g, v, prev) receives
// the inclusive prefixes of items g and g - 1 (sources that also derive
// something from each item's own value use prev)
template <class O>
struct IntScan {
  using T = int;
  using Op = O;
  const int* in;
  int* out;
  long long n;
  __device__ __forceinline__ int load(long long g) const { return in[g]; }
  __device__ __forceinline__ void store(long long g, int v, int) const { out[g] = v; }
};

// ------------------------------------------------------------ grid barrier
// Barrier over the blocks of one cooperative launch. bar[0] counts arrivals
// (zero when the launch starts, never reset inside it), so round r is complete
// at r * gridDim.x arrivals; bar[1] is set when a wait runs out of polls, after
// which every block leaves its launch at its next barrier. Returns false then,
// and the host finds *stall (its own memory, mapped) set.
// The work between two barriers is linear in the particles and keys (the
// longest segment included, order_segment), so the limit is too: a fixed part of
// 1.6 s (a poll takes 0.38 us), far above any phase of a small scene, and one poll
// for every 64 particles, 6 ns for each of them (order_segment takes 2 at most,
// where its network sorts a 64th of a scene).
constexpr int kBarrierPolls = 1 << 22;
inline int barrier_polls(long long np) { return np / 64 < INT_MAX - kBarrierPolls ? kBarrierPolls + (int)(np / 64) : INT_MAX; }

__device__ __forceinline__ bool grid_barrier(unsigned* bar, unsigned round, int polls, volatile int* stall) {
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(&bar[0], 1u);
    const unsigned want = round * gridDim.x;
    volatile unsigned* v = bar;
    int spins = 0;
    while (v[0] < want && v[1] == 0u && ++spins < polls) __nanosleep(100);
    if (v[0] < want) {
      atomicExch(&bar[1], 1u);
      *stall = 1;
    }
    ok = v[1] == 0u;
    __threadfence();
  }
  __syncthreads();
  const bool r = ok != 0;
  __syncthreads();  // ok is written again by the next barrier
  return r;
}

// ---------------------------------------------------------- counting sort
// The phases of the sort as device functions over the whole grid of one
// cooperative kernel (kb_resort), a grid barrier between them.
constexpr int kRegSeg = 32;         // segments up to this length are ordered by one thread
constexpr int kSortThreads = 256;   // threads of a block
constexpr int kSmemSeg = 8192;      // long segments up to this length are ordered in shared memory

constexpr unsigned kNoKey = 0xffffffffu;  // a particle that is not sorted

// seg (per-key counts) into inclusive segment ends in three phases over tiles
// of kScanTile keys, fill zeroed on the way; tile = kScanTile ints and thr,
// wsum of block_scan in shared memory
__device__ __forceinline__ void sort_tile_totals(const int* seg, long long nk, int* tiles, int* thr, int* wsum) {
  const long long nt = (nk + kScanTile - 1) / kScanTile;
  for (long long t = blockIdx.x; t < nt; t += gridDim.x) {
    const long long base = t * kScanTile;
    int v = 0;
    for (int e = threadIdx.x; e < kScanTile; e += kSortThreads)
      if (base + e < nk) v += seg[base + e];
    block_scan<int, ScanSum>(v, thr, wsum);
    if (threadIdx.x == 0) tiles[t] = thr[kSortThreads - 1];
    __syncthreads();
  }
}

// exclusive prefixes of the tile totals, by the first block
__device__ __forceinline__ void sort_tile_prefix(long long nk, int* tiles, int* thr, int* wsum) {
  if (blockIdx.x != 0) return;
  const long long nt = (nk + kScanTile - 1) / kScanTile;
  int carry = 0;
  for (long long b0 = 0; b0 < nt; b0 += kSortThreads) {
    const long long t = b0 + threadIdx.x;
    const int ex = block_scan<int, ScanSum>(t < nt ? tiles[t] : 0, thr, wsum);
    const int total = thr[kSortThreads - 1];
    if (t < nt) tiles[t] = carry + ex;
    carry += total;
    __syncthreads();
  }
}

__device__ __forceinline__ void sort_tile_scan(int* seg, int* fill, long long nk, const int* tiles, int* tile, int* thr,
                                               int* wsum) {
  const long long nt = (nk + kScanTile - 1) / kScanTile;
  for (long long t = blockIdx.x; t < nt; t += gridDim.x) {
    const long long base = t * kScanTile;
    for (int e = threadIdx.x; e < kScanTile; e += kSortThreads) tile[e] = base + e < nk ? seg[base + e] : 0;
    __syncthreads();
    int r[kScanItems], v = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) r[k] = v += tile[threadIdx.x * kScanItems + k];
    const int pre = tiles[t] + block_scan<int, ScanSum>(v, thr, wsum);
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) tile[threadIdx.x * kScanItems + k] = pre + r[k];
    __syncthreads();
    for (int e = threadIdx.x; e < kScanTile; e += kSortThreads)
      if (base + e < nk) {
        seg[base + e] = tile[e];
        fill[base + e] = 0;  // the placement's slots start at zero
      }
    __syncthreads();
  }
}

// perm[seg start + slot] = i for a warp's particles i with key k (kNoKey: none),
// the slot taken from the key's fill counter (one atomic per key and warp; lanes
// of a warp with the same key take consecutive slots in lane order)
__device__ __forceinline__ void sort_place(unsigned k, long long i, const int* seg, int* fill, int* perm) {
  const int lane = threadIdx.x & 31;
  const unsigned grp = __match_any_sync(0xffffffffu, k);
  const int leader = __ffs(grp) - 1, rank = __popc(grp & ((1u << lane) - 1u));
  int base = 0;
  if (lane == leader && k != kNoKey) base = atomicAdd(&fill[k], __popc(grp));
  base = __shfl_sync(0xffffffffu, base, leader);
  if (k != kNoKey) perm[(k == 0 ? 0 : seg[k - 1]) + base + rank] = (int)i;
}

// Ascending order of perm inside each key's segment: segments of up to
// kRegSeg particles by one thread (insertion sort, skipped when already in
// order -- the common case), longer ones listed in big for sort_long.
__device__ __forceinline__ void sort_segments(const int* seg, long long nk, int* perm, int* big, int* nbig) {
  for (long long k = (long long)blockIdx.x * kSortThreads + threadIdx.x; k < nk;
       k += (long long)gridDim.x * kSortThreads) {
    const int a = k == 0 ? 0 : seg[k - 1], e = seg[k];
    const int n = e - a;
    if (n <= 1) continue;
    if (n > kRegSeg) {
      big[atomicAdd(nbig, 1)] = (int)k;
      continue;
    }
    int* p = perm + a;
    bool sorted = true;
    int prev = p[0];
    for (int j = 1; j < n; ++j) {
      const int c = p[j];
      sorted = sorted && prev < c;
      prev = c;
    }
    if (sorted) continue;
    int v[kRegSeg];
    for (int j = 0; j < n; ++j) {
      const int c = p[j];
      int m = j;
      while (m > 0 && v[m - 1] > c) {
        v[m] = v[m - 1];
        --m;
      }
      v[m] = c;
    }
    for (int j = 0; j < n; ++j) p[j] = v[j];
  }
}

// ascending sort of d[0, n) (distinct values) by one block: a bitonic
// network over the next power of two whose every comparator puts the smaller
// value first (the first merge step of each stage compares mirrored
// partners), so the virtual elements past n (taken as +infinity) never move
// and are never touched
template <class T>
__device__ __forceinline__ void block_bitonic(T* d, int n) {
  int N = 1;
  while (N < n) N <<= 1;
  for (int k = 2; k <= N; k <<= 1) {
    for (int s = k >> 1; s > 0; s >>= 1) {
      for (int t = threadIdx.x; t < (N >> 1); t += blockDim.x) {
        int i, j;
        if (s == (k >> 1)) {  // mirrored partner within the block of k
          const int blk = t / s, o = t - blk * s;
          i = blk * k + o;
          j = blk * k + k - 1 - o;
        } else {
          i = (t / s) * 2 * s + (t % s);
          j = i + s;
        }
        if (j < n) {
          const T x = d[i], y = d[j];
          if (x > y) {
            d[i] = y;
            d[j] = x;
          }
        }
      }
      __syncthreads();
    }
  }
}

// the long segments: one block per segment (grid-stride over the list), in
// shared memory (sm, kSmemSeg values) up to kSmemSeg values; beyond, by
// longer(k, p, n)
template <class T, class Longer>
__device__ __forceinline__ void sort_long(const int* seg, T* perm, const int* big, const int* nbig, T* sm,
                                          Longer longer) {
  const int nb = *nbig;
  for (int b = blockIdx.x; b < nb; b += gridDim.x) {
    const int k = big[b];
    const int a = k == 0 ? 0 : seg[k - 1], n = seg[k] - a;
    T* p = perm + a;
    if (n <= kSmemSeg) {
      for (int j = threadIdx.x; j < n; j += blockDim.x) sm[j] = p[j];
      __syncthreads();
      block_bitonic(sm, n);
      for (int j = threadIdx.x; j < n; j += blockDim.x) p[j] = sm[j];
    } else {
      longer(k, p, n);
    }
    __syncthreads();
  }
}

// Ascending order of the n > kSmemSeg particles p of key k by one block: the
// particles between the first and the last of them that have the key, in
// order. A scene's particles outside its grid all share one key, so n reaches
// the scene's size; a bitonic network in global memory over 1.0, 4.1 and 8.0 M
// particles took 91, 443 and 951 ms, this the whole step 0.7, 2.3 and 4.4 ms
// (27 M: over 5 s and 17 ms). Where the key's particles are strewn over more
// than kScanRatio times their number (the order of a deck; a sorted scene has
// them close together) the network is shorter.
constexpr int kScanRatio = 64;

__device__ __forceinline__ void order_segment(const unsigned* key, unsigned k, int* p, int n) {
  constexpr int NW = kSortThreads / 32, Q = 16;
  __shared__ int range[2], cnt[2][NW];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x < 2) range[threadIdx.x] = p[0];
  __syncthreads();
  int lo = p[0], hi = p[0];
  for (int j = threadIdx.x; j < n; j += kSortThreads) {
    lo = min(lo, p[j]);
    hi = max(hi, p[j]);
  }
  lo = __reduce_min_sync(0xffffffffu, lo);
  hi = __reduce_max_sync(0xffffffffu, hi);
  if (lane == 0) {
    atomicMin(&range[0], lo);
    atomicMax(&range[1], hi);
  }
  __syncthreads();
  lo = range[0];
  hi = range[1];
  if ((long long)hi - lo >= (long long)kScanRatio * n) {
    block_bitonic(p, n);
    return;
  }
  // tiles of Q rows of 32 particles per warp; the rows' votes give the places
  int done = 0;
  for (long long i0 = lo, t = 0; i0 <= hi; i0 += kSortThreads * Q, ++t) {
    const long long w0 = i0 + warp * (32 * Q) + lane;
    unsigned row[Q];
    int mine = 0;
#pragma unroll
    for (int q = 0; q < Q; ++q) row[q] = w0 + 32 * q <= hi ? key[w0 + 32 * q] : kNoKey;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      row[q] = __ballot_sync(0xffffffffu, row[q] == k);
      mine += __popc(row[q]);
    }
    if (lane == 0) cnt[t & 1][warp] = mine;
    __syncthreads();  // (one a tile: this half of cnt is written again after the next one)
    int at = done;
#pragma unroll
    for (int w = 0; w < NW; ++w) {
      if (w < warp) at += cnt[t & 1][w];
      done += cnt[t & 1][w];
    }
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      if (row[q] >> lane & 1u) p[at + __popc(row[q] & ((1u << lane) - 1u))] = (int)(w0 + 32 * q);
      at += __popc(row[q]);
    }
  }
}

}  // namespace bm
}  // namespace mpm
