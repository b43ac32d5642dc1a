// mpm_reduce.cuh -- the block reduction of the energy sums, shared by the step's
// reduction (mpm_kernels.cuh) and the allocation-free one (mpm_noalloc.cu),
// whose results agree bit for bit.
#pragma once

namespace mpm {

// A block's NV sums (the last one a maximum) of its NT threads' values in a
// fixed order, in out: a warp per value, a lane adds NT / 32 threads' and the
// lanes are joined in a tree (13 FP64 instructions in series; a tree over the
// block's threads had one warp execute 48 of them, 64 cycles each on this
// FP64 pipe, between barriers: the step's reduction of Cook's 5.8 k particles
// 19 -> 13.5 us).
template <int NV, int NT>
__device__ __forceinline__ void reduce_block(double (*sh)[NT], const double* v, double* out) {
  constexpr int NW = NT / 32;
  static_assert(NV <= NW, "a warp per value");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int i = 0; i < NV; ++i) sh[i][threadIdx.x] = v[i];
  __syncthreads();
  if (warp < NV) {
    const bool mx = warp == NV - 1;
    double a = sh[warp][lane];
#pragma unroll
    for (int j = 1; j < NW; ++j) {
      const double b = sh[warp][lane + 32 * j];
      a = mx ? (b > a ? b : a) : a + b;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double b = __shfl_down_sync(0xffffffffu, a, o);
      a = mx ? (b > a ? b : a) : a + b;
    }
    if (lane == 0) out[warp] = a;
  }
  __syncthreads();
}

}  // namespace mpm
