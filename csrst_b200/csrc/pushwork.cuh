// How a push's particles are shared out over its warps, and the end of a
// single-member push.
#pragma once

#include "accum.cuh"
#include "bbox.cuh"
#include "common.cuh"

namespace csrst {

// The work of one warp as runs of rounds of 32 particles: in the k-th run lane
// l's particles are n + l, n + l + step, ... below end; false: no more runs.
// run() is called by the whole warp together.
//
// One contiguous share [beg, end) of a CTA (a member of a batch): in each round
// its warps take 256 consecutive particles (the bunch is sorted by y slice and
// x, so they read the same cells and adjacent lines).
struct ShareWork {
  long long b, e;
  __device__ __forceinline__ bool run(int k, long long &n, long long &end, long long &step) const {
    n = b + (threadIdx.x & ~31u); end = e; step = kPushThreads;
    return k == 0;
  }
};

// The whole bunch over the grid: 13/16 of it in contiguous shares per CTA, the
// rest handed out to the warps by a counter, kGroups groups of 32 at a time.  With
// equal shares alone the CTA that an SM started last ends well after the
// others (its warps come last in the schedulers' order), and so do the CTAs
// whose share crosses from one y slice to the next, where the bunch is sparse
// and every round drains the tile: the middle CTA ended after 132 us, the last
// after 178 (8192 x 1024 mesh, 4e6 TSC particles, FP32).  Per step of that
// bunch, FP32 / FP64: shares alone 412 / 661 us, 13/16 and two groups 381 / 638,
// half and two groups 425 / 661 (a run's end drains the tile too), one group
// 389 / 655.  Below kMinRounds rounds per CTA the counter costs as much as it
// saves: shares alone.
struct BunchWork {
  static constexpr unsigned kMinRounds = 8, kGroups = 2;
  long long N;
  PushCtl *ctl;
  __device__ __forceinline__ bool run(int k, long long &n, long long &end, long long &step) const {
    const unsigned G = gridDim.x, T = (unsigned)((N + kPushThreads - 1) / kPushThreads);
    const unsigned shared = T >= kMinRounds * G ? T - T / 16 * 3 : T;  // rounds in shares
    if (k == 0) {
      n = (long long)((unsigned long long)shared * blockIdx.x / G) * kPushThreads + (threadIdx.x & ~31u);
      end = (long long)((unsigned long long)shared * (blockIdx.x + 1) / G) * kPushThreads;
      step = kPushThreads;
    } else {
      if (shared == T) return false;
      unsigned c = 0;
      if ((threadIdx.x & 31) == 0) c = atomicAdd(&ctl->next, 1u);
      c = __shfl_sync(0xffffffffu, c, 0);
      n = (long long)shared * kPushThreads + (long long)c * (kGroups * 32);
      end = n + kGroups * 32;
      step = 32;
      if (n >= N) return false;
    }
    if (end > N) end = N;
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
      ctl->next = 0;
    }
  }
  __syncthreads();
  return sh.last;
}

// Before a push: derive the gather patches from the particle box of the
// positions the push will gather at (PartBunch::getLocalPDomain and
// getFields), and reset the accumulators the push will fill.
// em: getExtraMarginEdge (x first, x last, y first, y last); cm: getExtraMarginCell.
// defer: a bunch that does not fit is reported by the next push (PushCtl).
__device__ __forceinline__ void push_prep_body(WinState *ws, double h0, double h1, int em0, int em2, int cm0,
                                               bool defer) {
  const int c = ws->cur;
  const double mn0 = ord_dbl(ws->bb[c][0]), mn1 = ord_dbl(ws->bb[c][1]);
  const double mx0 = ord_dbl(ws->bb[c][2]), mx1 = ord_dbl(ws->bb[c][3]);
  int lp[4];
  if (mn0 <= mx0) {
    lp[0] = (int)floor((mn0 - ws->mo0) / h0); lp[1] = (int)floor((mx0 - ws->mo0) / h0);
    lp[2] = (int)floor((mn1 - ws->mo1) / h1); lp[3] = (int)floor((mx1 - ws->mo1) / h1);
  } else {  // no particles: PartBunch::getLocalPDomain with Rmin = Rmax = 0
    lp[0] = lp[1] = (int)floor((0.0 - ws->mo0) / h0);
    lp[2] = lp[3] = (int)floor((0.0 - ws->mo1) / h1);
  }
  for (int k = 0; k < 4; ++k) ws->lp[k] = lp[k];
  // Every gather tap lies within [lp - 2, lp + 2] (the cubic edge stencil
  // reaches furthest); the window planes hold one guard cell.  A bunch that
  // no longer fits stops the run instead of reading outside the window.
  const int nofit = mn0 <= mx0 && (lp[0] - 2 < -1 || lp[1] + 2 > ws->L0 || lp[2] - 2 < -1 || lp[3] + 2 > ws->L1);
  if (nofit && !defer) set_err(ws, kErrWindowFit);
  push_ctl(ws)->nofit = defer ? nofit : 0;
  const double po0 = ws->mo0 + lp[0] * h0, po1 = ws->mo1 + lp[2] * h1;
  ws->hz_o0 = po0 + cm0 * h0; ws->hz_o1 = po1 + cm0 * h1;
  ws->ex_o0 = po0 + em0 * h0; ws->ex_o1 = po1 + em2 * h1;
  ws->ey_o0 = po0 + em2 * h0; ws->ey_o1 = po1 + em0 * h1;
  ws->hz_I = lp[0] + cm0; ws->hz_J = lp[2] + cm0;
  ws->ex_I = lp[0] + em0; ws->ex_J = lp[2] + em2;
  ws->ey_I = lp[0] + em2; ws->ey_J = lp[2] + em0;
  bbox_reset(ws->bb[1 - c]);
  bbox_reset(ws->bball);
}

// FP32 mode's set-up.  Gather-patch set-up and the window-fit check from the box of the next
// push's gather positions (cells of the static mesh).  defer: a bunch that does
// not fit is reported by the next push, not at once (PushCtl).
__device__ __forceinline__ void prep32_body(WinState *ws, int reach, bool defer) {
  const int c = ws->cur;
  const double mn0 = ord_dbl(ws->bb[c][0]), mn1 = ord_dbl(ws->bb[c][1]);
  const double mx0 = ord_dbl(ws->bb[c][2]), mx1 = ord_dbl(ws->bb[c][3]);
  int nofit = 0;
  if (mn0 <= mx0) {
    const int lp[4] = {(int)floor(mn0) - ws->P0, (int)floor(mx0) - ws->P0, (int)floor(mn1) - ws->P1,
                       (int)floor(mx1) - ws->P1};
    for (int k = 0; k < 4; ++k) ws->lp[k] = lp[k];
    // every gather tap lies within [lp - reach, lp + reach]
    nofit = lp[0] - reach < -1 || lp[1] + reach > ws->L0 || lp[2] - reach < -1 || lp[3] + reach > ws->L1;
    if (nofit && !defer) set_err(ws, kErrWindowFit);
  }
  push_ctl(ws)->nofit = defer ? nofit : 0;
  bbox_reset(ws->bb[1 - c]);
  bbox_reset(ws->bball);
}

}  // namespace csrst
