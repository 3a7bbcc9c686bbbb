// Bounding boxes of particle positions reduced over a CTA and merged into
// device-wide boxes held as ordered-integer doubles (see dbl_ord).
#pragma once

#include "common.cuh"

namespace csrst {

__device__ __forceinline__ void warp_bbox(double &mn0, double &mn1, double &mx0, double &mx1) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    mn0 = fmin(mn0, __shfl_xor_sync(0xffffffffu, mn0, o));
    mn1 = fmin(mn1, __shfl_xor_sync(0xffffffffu, mn1, o));
    mx0 = fmax(mx0, __shfl_xor_sync(0xffffffffu, mx0, o));
    mx1 = fmax(mx1, __shfl_xor_sync(0xffffffffu, mx1, o));
  }
}

// Reduce a per-thread box over the CTA and merge it into dst[4] with atomics;
// sb is shared scratch of 4 x 32 doubles.
__device__ __forceinline__ void block_bbox(double mn0, double mn1, double mx0, double mx1, long long *dst,
                                           double (*sb)[32]) {
  warp_bbox(mn0, mn1, mx0, mx1);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  if (lane == 0) { sb[0][w] = mn0; sb[1][w] = mn1; sb[2][w] = mx0; sb[3][w] = mx1; }
  __syncthreads();
  if (w == 0) {
    mn0 = lane < nw ? sb[0][lane] : INFINITY;
    mn1 = lane < nw ? sb[1][lane] : INFINITY;
    mx0 = lane < nw ? sb[2][lane] : -INFINITY;
    mx1 = lane < nw ? sb[3][lane] : -INFINITY;
    warp_bbox(mn0, mn1, mx0, mx1);
    if (lane == 0 && mn0 <= mx0) {
      atomicMin(&dst[0], dbl_ord(mn0));
      atomicMin(&dst[1], dbl_ord(mn1));
      atomicMax(&dst[2], dbl_ord(mx0));
      atomicMax(&dst[3], dbl_ord(mx1));
    }
  }
  __syncthreads();
}

// Smallest ordered-integer double of a warp: its high words, then the low
// words of the lanes that hold that high word.
__device__ __forceinline__ long long warp_min_ord(long long v) {
  const int hi = (int)(v >> 32), mh = __reduce_min_sync(0xffffffffu, hi);
  const unsigned ml = __reduce_min_sync(0xffffffffu, hi == mh ? (unsigned)v : 0xffffffffu);
  return ((long long)mh << 32) | ml;
}

// The boxes of one push, merged over a CTA into ws->bball (v[0 .. 3]: R0 u R2)
// and the next push's slot (v[4 .. 7]), as ordered-integer doubles, the maxima
// complemented (~x reverses the order), so that everything is a minimum; sb is
// shared scratch.  Ends with a barrier.
__device__ __forceinline__ void merge_boxes(const long long (&v)[8], WinState *ws, long long (*sb)[32]) {
  const int w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const long long m = warp_min_ord(v[k]);
    if ((threadIdx.x & 31) == 0) sb[k][w] = m;
  }
  __syncthreads();
  if (threadIdx.x < 8) {
    const int k = threadIdx.x;
    long long m = sb[k][0];
    for (int q = 1; q < nw; ++q) m = sb[k][q] < m ? sb[k][q] : m;
    long long *dst = (k < 4 ? ws->bball : ws->bb[1 - ws->cur]) + (k & 3);
    if ((k & 3) < 2) atomicMin(dst, m);
    else atomicMax(dst, ~m);
  }
  __syncthreads();
}

// Shared scratch of one push CTA, declared once per kernel so that a kernel
// that inlines several push variants does not hold one copy per variant.
struct PushShared {
  long long sb[8][32];  // merge_boxes
  int tb[4];         // touched box of the CTA (window cells)
  int err;           // the member's sticky error at entry
  bool last;         // this CTA ends its push last
};

__device__ __forceinline__ void bbox_reset(long long *b) {
  b[0] = dbl_ord(INFINITY); b[1] = dbl_ord(INFINITY);
  b[2] = dbl_ord(-INFINITY); b[3] = dbl_ord(-INFINITY);
}

}  // namespace csrst
