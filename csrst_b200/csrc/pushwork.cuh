// How a push's particles are shared out over its warps, and the end of a
// single-member push.
#pragma once

#include "bbox.cuh"
#include "common.cuh"

namespace csrst {

constexpr int kPushThreads = 256;  // threads of every push CTA

// The rounds of one CTA: in each, its warps take 256 consecutive particles (the
// bunch is sorted by y slice and x, so a CTA's warps read the same cells and
// adjacent lines).  run(k): the k-th run of rounds, from particle n in steps of
// step up to end; false: no more runs.
//
// One contiguous share [beg, end) (a member of a batch).
struct ShareWork {
  long long b, e;
  __device__ __forceinline__ bool run(int k, long long &n, long long &end, long long &step) const {
    n = b; end = e; step = kPushThreads;
    return k == 0;
  }
};

// The whole bunch over the grid.  The particles at the bunch's rim (the first
// and last y slices) change cell every few groups, and each change drains a
// tile, so the CTAs that held the rim in equal contiguous shares ended last
// (8192 x 1024 mesh, 4e6 TSC particles: 282 tile drains in the first and last
// CTA, 16 in the median one).  The rim, 1/32 of the bunch on each side, is
// therefore dealt out round by round, the rest in contiguous shares (that
// bunch, FP32: 509 -> 483 us per step).  With fewer than kMinRounds rounds per
// CTA the extra rim rounds of some CTAs cost more than the drains (1.5e5 cubic
// particles, 2 rounds per CTA: 116 -> 136 us per step): contiguous shares only.
// A queue of runs handed out by a counter, per warp, was slower than either
// (516 us): a run of one warp drains its tile more often than a CTA's.
struct BunchWork {
  static constexpr unsigned kMinRounds = 16;
  long long N;
  __device__ __forceinline__ bool run(int k, long long &n, long long &end, long long &step) const {
    const unsigned b = blockIdx.x, G = gridDim.x, T = (unsigned)((N + kPushThreads - 1) / kPushThreads);
    const unsigned rim = T >= kMinRounds * G ? T / 32 : 0u, mid = T - 2 * rim;
    unsigned r0, r1, s = 1;
    if (k == 0) {
      r0 = rim + (unsigned)((unsigned long long)mid * b / G);
      r1 = rim + (unsigned)((unsigned long long)mid * (b + 1) / G);
    } else if (k < 3 && rim > 0) {
      r0 = (k == 1 ? 0 : T - rim) + b;
      r1 = k == 1 ? rim : T;
      s = G;
    } else {
      return false;
    }
    n = (long long)r0 * kPushThreads;
    end = (long long)r1 * kPushThreads;
    if (end > N) end = N;
    step = (long long)s * kPushThreads;
    return true;
  }
};

// CTAs of a single-member push: one round each for a small bunch, at most `most`.
inline int push_ctas(long long n, int most) {
  const long long want = (n + kPushThreads - 1) / kPushThreads;
  return (int)(want < 1 ? 1 : want < most ? want : most);
}

// The member's sticky error at entry, or its bunch not fitting the window as
// the set-up after the last push or move found (PushCtl::nofit), read by one
// thread for the CTA; a CTA that sees one leaves as a whole.
__device__ __forceinline__ bool entry_error(WinState *ws, PushShared &sh) {
  if (threadIdx.x == 0) {
    sh.err = *(volatile int *)&ws->err;
    if (!sh.err && *(volatile int *)&push_ctl(ws)->nofit) {
      set_err(ws, kErrWindowFit);
      sh.err = kErrWindowFit;
    }
  }
  __syncthreads();
  return sh.err != 0;
}

// True in the CTA that ends a single-member push last, with every other CTA's
// boxes and sums visible to it; resets the launch's counters.
__device__ __forceinline__ bool last_cta(WinState *ws, PushShared &sh) {
  __syncthreads();
  if (threadIdx.x == 0) {
    PushCtl *ctl = push_ctl(ws);
    __threadfence();
    sh.last = atomicAdd(&ctl->done, 1u) == gridDim.x - 1;
    if (sh.last) {
      __threadfence();
      ctl->done = 0;
    }
  }
  __syncthreads();
  return sh.last;
}

}  // namespace csrst
