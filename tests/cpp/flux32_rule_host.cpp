// Host build of the FP32 deposit's choice of form (csrst_b200/csrc/flux32.cuh).
#include <math.h>
#include <stdint.h>

#define __device__
#define __forceinline__ inline
static inline long long __double2ll_rn(double x) { return llrint(x); }
static inline long long __float2ll_rn(float x) { return llrintf(x); }

#include "../../csrst_b200/csrc/flux32.cuh"

extern "C" int compact_form_host(int order, float a0, float a1, int dc0, int dc1, float b0, float b1, double K) {
  return order == 0   ? csrst::compact_form<0>(a0, a1, dc0, dc1, b0, b1, K)
         : order == 1 ? csrst::compact_form<1>(a0, a1, dc0, dc1, b0, b1, K)
                      : csrst::compact_form<2>(a0, a1, dc0, dc1, b0, b1, K);
}
