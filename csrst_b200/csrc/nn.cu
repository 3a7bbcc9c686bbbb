// Element-wise and reduction kernels of the wake surrogate's training and
// inference (the products are the tensor-core GEMM of gemm.cu).  Reductions
// run in a fixed order, so a training run repeats bit for bit.
//
// All are bound by memory or, at the sizes of a training step (R = 16384 rows
// of 128), by a launch's latency: each thread has its loads in flight together, and
// launches follow one another through chain.cuh.
#include <cuda_bf16.h>
#include <stdint.h>

#include "../../include/csrst.h"
#include "chain.cuh"
#include "nn.h"

namespace csrst {
namespace {

__device__ __forceinline__ long long gtid() { return blockIdx.x * (long long)blockDim.x + threadIdx.x; }
inline unsigned grid_of(long long n) { return (unsigned)((n + 255) / 256 < 65535 * 16 ? (n + 255) / 256 : 65535 * 16); }

// [z][r][c] -> [z][c][r] (dst rows ldd apart) through 32 x 32 shared-memory
// tiles; T is a BF16 value or a 32-bit pair of them.
template <class T>
__global__ void k_transpose(const T *src, T *dst, int rows, int cols, int ldd) {
  chain_next();
  chain_wait();
  __shared__ T t[32][33];
  const long long z = blockIdx.z;
  src += z * (long long)rows * cols;
  dst += z * (long long)ldd * cols;
  const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
  for (int k = threadIdx.y; k < 32; k += 8) {
    const int r = r0 + k, c = c0 + threadIdx.x;
    if (r < rows && c < cols) t[k][threadIdx.x] = src[(long long)r * cols + c];
  }
  __syncthreads();
  for (int k = threadIdx.y; k < 32; k += 8) {
    const int c = c0 + k, r = r0 + threadIdx.x;
    if (r < rows && c < cols) dst[(long long)c * ldd + r] = t[threadIdx.x][k];
  }
}

// Whole 64 x 64 tiles of BF16 values: a tile is held as 64 rows of 32 words
// (column pairs; 33 apart), and thread (w, g) of 32 x 8 turns words w of rows
// 8g .. 8g + 7 into 16 bytes of columns 2w and 2w + 1.
__device__ __forceinline__ void store_columns(const uint32_t (*t)[33], __nv_bfloat16 *dst, int ldd) {
  const int w = threadIdx.x & 31, g = threadIdx.x >> 5;
  uint32_t v[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) v[k] = t[8 * g + k][w];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    uint4 o;
    const unsigned sel = h ? 0x7632 : 0x5410;
    o.x = __byte_perm(v[0], v[1], sel);
    o.y = __byte_perm(v[2], v[3], sel);
    o.z = __byte_perm(v[4], v[5], sel);
    o.w = __byte_perm(v[6], v[7], sel);
    *reinterpret_cast<uint4 *>(dst + (long long)(2 * w + h) * ldd + 8 * g) = o;
  }
}

__global__ void __launch_bounds__(256) k_transpose64(const __nv_bfloat16 *src, __nv_bfloat16 *dst, int rows, int cols,
                                                     int ldd) {
  chain_next();
  chain_wait();
  __shared__ uint32_t t[64][33];
  const long long z = blockIdx.z;
  const int c0 = blockIdx.x * 64, r0 = blockIdx.y * 64, q = threadIdx.x & 7, r = threadIdx.x >> 3;
  src += z * (long long)rows * cols + (long long)r0 * cols + c0 + 8 * q;
  const uint4 a = *reinterpret_cast<const uint4 *>(src + (long long)r * cols);
  const uint4 b = *reinterpret_cast<const uint4 *>(src + (long long)(r + 32) * cols);
  uint32_t *ta = &t[r][4 * q], *tb = &t[r + 32][4 * q];
  ta[0] = a.x, ta[1] = a.y, ta[2] = a.z, ta[3] = a.w;
  tb[0] = b.x, tb[1] = b.y, tb[2] = b.z, tb[3] = b.w;
  __syncthreads();
  store_columns(t, dst + z * (long long)ldd * cols + (long long)c0 * ldd + r0, ldd);
}

// 32-bit elements, rows a multiple of 32: 32 x 128 tiles, sixteen loads of a
// thread in flight, 16-byte stores (the tile's columns are 129 words apart, which
// keeps both sides free of bank conflicts).
__global__ void __launch_bounds__(256) k_transpose32x128(const uint32_t *src, uint32_t *dst, int rows, int cols,
                                                         int ldd) {
  chain_next();
  chain_wait();
  __shared__ uint32_t t[32][129];
  const long long z = blockIdx.z;
  const int c0 = blockIdx.x * 128, r0 = blockIdx.y * 32, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  src += z * (long long)rows * cols;
  dst += z * (long long)ldd * cols;
  uint32_t v[4][4];
#pragma unroll
  for (int k = 0; k < 4; ++k)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = c0 + 32 * j + lane;
      v[k][j] = c < cols ? src[(long long)(r0 + 8 * k + warp) * cols + c] : 0u;
    }
#pragma unroll
  for (int k = 0; k < 4; ++k)
#pragma unroll
    for (int j = 0; j < 4; ++j) t[8 * k + warp][32 * j + lane] = v[k][j];
  __syncthreads();
  const int rq = 4 * (lane & 7);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int c = 32 * k + 4 * warp + (lane >> 3);
    if (c0 + c < cols)
      *reinterpret_cast<uint4 *>(dst + (long long)(c0 + c) * ldd + r0 + rq) =
          make_uint4(t[rq][c], t[rq + 1][c], t[rq + 2][c], t[rq + 3][c]);
  }
}

// d/dx of 0.5 x (1 + erf(x / sqrt 2)) = 0.5 (1 + erf(x / sqrt 2)) + x exp(-x^2 / 2) / sqrt(2 pi)
__device__ __forceinline__ float gelu_grad(float x) {
  return 0.5f * (1.0f + erff(x * 0.70710678118654752f)) + x * expf(-0.5f * x * x) * 0.3989422804014327f;
}

__global__ void k_gelu_bwd(const float *dy, const float *pre, float *dx32, __nv_bfloat16 *dx16, long long n) {
  chain_next();
  chain_wait();
  for (long long i = gtid(); i < n; i += (long long)gridDim.x * blockDim.x) {
    const float v = dy[i] * gelu_grad(pre[i]);
    if (dx32) dx32[i] = v;
    if (dx16) dx16[i] = __float2bfloat16(v);
  }
}

__device__ __forceinline__ uint32_t pair16(float lo, float hi) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t *>(&h);
}

// The gradient of a layer's output through its activation in the three forms
// the products and sums after it read, in one pass over 64 x 64 tiles (R = 16384 x
// 128: 8.3 us for 13 + 6 us as an element-wise pass and a transpose).
template <bool GELU>
__global__ void __launch_bounds__(256) k_backward_rows(const float *dy, const float *pre, float *dx32,
                                                       __nv_bfloat16 *dx16, __nv_bfloat16 *dxT16, int rows, int cols) {
  chain_next();
  chain_wait();
  __shared__ uint32_t t[64][33];
  const int c0 = blockIdx.x * 64, r0 = blockIdx.y * 64, q = threadIdx.x & 15, r = threadIdx.x >> 4;
  const long long o = (long long)(r0 + r) * cols + c0 + 4 * q;
  float4 d[4], p[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    d[k] = *reinterpret_cast<const float4 *>(dy + o + (long long)(16 * k) * cols);
    if (GELU) p[k] = *reinterpret_cast<const float4 *>(pre + o + (long long)(16 * k) * cols);
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    float4 v = d[k];
    if (GELU) {
      v.x *= gelu_grad(p[k].x);
      v.y *= gelu_grad(p[k].y);
      v.z *= gelu_grad(p[k].z);
      v.w *= gelu_grad(p[k].w);
    }
    const long long i = o + (long long)(16 * k) * cols;
    if (dx32) *reinterpret_cast<float4 *>(dx32 + i) = v;
    const uint2 w = make_uint2(pair16(v.x, v.y), pair16(v.z, v.w));
    *reinterpret_cast<uint2 *>(dx16 + i) = w;
    t[r + 16 * k][2 * q] = w.x;
    t[r + 16 * k][2 * q + 1] = w.y;
  }
  __syncthreads();
  store_columns(t, dxT16 + (long long)c0 * rows + r0, rows);
}

__global__ void k_cast(const float *x, __nv_bfloat16 *y, long long n) {
  chain_next();
  chain_wait();
  for (long long i = gtid(); i < n; i += (long long)gridDim.x * blockDim.x) y[i] = __float2bfloat16(x[i]);
}
__global__ void k_cast4(const float4 *x, uint2 *y, long long n4) {
  chain_next();
  chain_wait();
  for (long long i = gtid(); i < n4; i += (long long)gridDim.x * blockDim.x) {
    const float4 v = x[i];
    y[i] = make_uint2(pair16(v.x, v.y), pair16(v.z, v.w));
  }
}

// s + x[0] + x[stride] + ... in that order, the loads 32 at a time ahead of
// the additions that wait for one another.
__device__ __forceinline__ float sum_in_order(float s, const float *x, long long stride, int n) {
  int k = 0;
  for (; k + 32 <= n; k += 32) {
    float v[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = x[(long long)(k + j) * stride];
#pragma unroll
    for (int j = 0; j < 32; ++j) s += v[j];
  }
  for (; k < n; ++k) s += x[(long long)k * stride];
  return s;
}

// out[c] (+)= sum_r x[r][c]: each block sums a 256-row slab per column, a
// second pass adds the slabs in order; one slab goes straight to `out`.  A chain
// of loads and additions per column: one warp a block spreads 128 columns over
// 256 blocks (16384 x 128: 6.5 us for 12.9 with one load at a time).
__global__ void __launch_bounds__(32) k_colsum_part(const float *x, int rows, int cols, float *part, int accumulate) {
  chain_next();
  chain_wait();
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= cols) return;
  const int r0 = blockIdx.y * 256, r1 = min(rows, r0 + 256);
  const float s = sum_in_order(0.0f, x + (long long)r0 * cols + c, cols, r1 - r0);
  float *o = part + (long long)blockIdx.y * cols + c;
  *o = accumulate ? *o + s : s;
}
__global__ void __launch_bounds__(32) k_colsum_final(const float *part, int slabs, int cols, float *out, int accumulate) {
  chain_next();
  chain_wait();
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= cols) return;
  const float s = sum_in_order(0.0f, part + c, cols, slabs);
  out[c] = accumulate ? out[c] + s : s;
}

// Mean squared error, optionally weighted per output (a 0/1 weight leaves
// an output out): grad = 2 w^2 (pred - target) / n (written through gmap:
// index (i / gd) * g0 + (i % gd) * g1, so that the gradient lands in the layout
// of the last product), partial sums per block, then the total in order.
__global__ void k_mse(const float *pred, const float *target, const float *weight, long long n, float *grad, int gd,
                      long long g0, long long g1, double *part) {
  chain_next();
  chain_wait();
  __shared__ double sh[256];
  double s = 0.0;
  for (long long i = gtid(); i < n; i += (long long)gridDim.x * blockDim.x) {
    const float e = weight ? (pred[i] - target[i]) * weight[i] : pred[i] - target[i];
    s += (double)e * e;
    const long long q = n <= 0x7fffffffll ? (long long)((unsigned)i / (unsigned)gd) : i / gd;
    if (grad) grad[q * g0 + (i - q * gd) * g1] = 2.0f * (weight ? weight[i] : 1.0f) * e / (float)n;
  }
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w) sh[threadIdx.x] += sh[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = sh[0];
}
// The blocks' partial sums: lanes in turn, then the lanes, in a fixed order.
__global__ void k_sum_final(const double *part, int np, long long n, double *out) {
  chain_next();
  chain_wait();
  double s = 0.0;
  for (int k = threadIdx.x; k < np; k += 32) s += part[k];
  for (int d = 16; d > 0; d >>= 1) s += __shfl_down_sync(0xffffffffu, s, d);
  if (threadIdx.x == 0) *out = s / (double)n;
}

// Adam (Kingma & Ba 2015) with bias correction.  The step counter and the
// schedule live on the device, so a captured training step replays as is:
// k_adam_tick advances t and writes {lr_t, 1 - b1^t, 1 - b2^t}, the learning
// rate following a cosine from lr0 to lr_min over `total` steps.
__global__ void k_adam_tick(int *t, float *coef, float lr0, float lr_min, int total, float b1, float b2) {
  chain_next();
  chain_wait();
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  const int k = ++*t;
  const float f = k >= total ? 1.0f : (float)k / (float)total;
  coef[0] = lr_min + 0.5f * (lr0 - lr_min) * (1.0f + cospif(f));
  coef[1] = 1.0f - powf(b1, (float)k);
  coef[2] = 1.0f - powf(b2, (float)k);
}

__device__ __forceinline__ void adam_one(float &w, float gi, float &m, float &v, float lr, float c1, float c2,
                                         float b1, float b2, float eps) {
  const float mi = b1 * m + (1.0f - b1) * gi;
  const float vi = b2 * v + (1.0f - b2) * gi * gi;
  m = mi;
  v = vi;
  w -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

// n4 elements of four, then the n - 4 n4 that are left.
__global__ void k_adam(float *w, const float *g, float *m, float *v, long long n, long long n4, const float *coef,
                       float b1, float b2, float eps) {
  chain_next();
  chain_wait();
  const float lr = coef[0], c1 = coef[1], c2 = coef[2];
  for (long long i = gtid(); i < n4; i += (long long)gridDim.x * blockDim.x) {
    float4 wi = reinterpret_cast<float4 *>(w)[i], mi = reinterpret_cast<float4 *>(m)[i];
    float4 vi = reinterpret_cast<float4 *>(v)[i];
    const float4 gi = reinterpret_cast<const float4 *>(g)[i];
    adam_one(wi.x, gi.x, mi.x, vi.x, lr, c1, c2, b1, b2, eps);
    adam_one(wi.y, gi.y, mi.y, vi.y, lr, c1, c2, b1, b2, eps);
    adam_one(wi.z, gi.z, mi.z, vi.z, lr, c1, c2, b1, b2, eps);
    adam_one(wi.w, gi.w, mi.w, vi.w, lr, c1, c2, b1, b2, eps);
    reinterpret_cast<float4 *>(w)[i] = wi;
    reinterpret_cast<float4 *>(m)[i] = mi;
    reinterpret_cast<float4 *>(v)[i] = vi;
  }
  for (long long i = 4 * n4 + gtid(); i < n; i += (long long)gridDim.x * blockDim.x)
    adam_one(w[i], g[i], m[i], v[i], lr, c1, c2, b1, b2, eps);
}

// Complex spectral weights W_k = Wr + i Wi ([modes][cin][cout]) as the real
// block matrices the products take: Mk[2o + p][2c + q] (Z = U Mk^T) and its
// transpose MkT[2c + q][2o + p] (dU = dZ Mk).  32 x 32 tiles of (c, o): MkT's pairs
// (p = 0, 1) go out along o as they were read, Mk's pairs (q = 0, 1) along c through
// shared memory (32 modes of 128 x 128: 6.1 us for 23 with Mk's values written
// one at a time down its columns).
template <bool PAIRS>
__device__ __forceinline__ void put_pair(__nv_bfloat16 *o, float lo, float hi) {
  if (PAIRS) {
    *reinterpret_cast<uint32_t *>(o) = pair16(lo, hi);
  } else {
    o[0] = __float2bfloat16(lo);
    o[1] = __float2bfloat16(hi);
  }
}
template <bool PAIRS>
__global__ void k_spectral_pack(const float *wr, const float *wi, int ch, __nv_bfloat16 *mk, __nv_bfloat16 *mkt) {
  chain_next();
  chain_wait();
  __shared__ float tr[32][33], ti[32][33];
  const long long k = blockIdx.z, w2 = 2 * ch;
  const int o0 = blockIdx.x * 32, c0 = blockIdx.y * 32, x = threadIdx.x;
  wr += k * ch * ch;
  wi += k * ch * ch;
  mk += k * w2 * w2;
  mkt += k * w2 * w2;
  for (int y = threadIdx.y; y < 32; y += 8) {
    const int c = c0 + y, o = o0 + x;
    if (c >= ch || o >= ch) continue;
    const float r = wr[(long long)c * ch + o], im = wi[(long long)c * ch + o];
    tr[y][x] = r;
    ti[y][x] = im;
    put_pair<PAIRS>(mkt + (long long)(2 * c) * w2 + 2 * o, r, im);
    put_pair<PAIRS>(mkt + (long long)(2 * c + 1) * w2 + 2 * o, -im, r);
  }
  __syncthreads();
  for (int y = threadIdx.y; y < 32; y += 8) {
    const int c = c0 + x, o = o0 + y;
    if (c >= ch || o >= ch) continue;
    const float r = tr[x][y], im = ti[x][y];
    put_pair<PAIRS>(mk + (long long)(2 * o) * w2 + 2 * c, r, -im);
    put_pair<PAIRS>(mk + (long long)(2 * o + 1) * w2 + 2 * c, im, r);
  }
}

// dWr[c][o] = dMk[2o][2c] + dMk[2o+1][2c+1], dWi[c][o] = dMk[2o+1][2c] - dMk[2o][2c+1],
// read along c and turned through shared memory (5.8 us for 12.3 with reads down
// dMk's columns).
__global__ void k_spectral_unpack(const float *dmk, int ch, float *dwr, float *dwi) {
  chain_next();
  chain_wait();
  __shared__ float tr[32][33], ti[32][33];
  const long long k = blockIdx.z, w2 = 2 * ch;
  const int o0 = blockIdx.x * 32, c0 = blockIdx.y * 32, x = threadIdx.x;
  dmk += k * w2 * w2;
  dwr += k * ch * ch;
  dwi += k * ch * ch;
  for (int y = threadIdx.y; y < 32; y += 8) {
    const int c = c0 + x, o = o0 + y;
    if (c >= ch || o >= ch) continue;
    const float *d0 = dmk + (long long)(2 * o) * w2 + 2 * c, *d1 = d0 + w2;
    tr[y][x] = d0[0] + d1[1];
    ti[y][x] = d1[0] - d0[1];
  }
  __syncthreads();
  for (int y = threadIdx.y; y < 32; y += 8) {
    const int c = c0 + y, o = o0 + x;
    if (c >= ch || o >= ch) continue;
    dwr[(long long)c * ch + o] = tr[x][y];
    dwi[(long long)c * ch + o] = ti[x][y];
  }
}

bool aligned16(const void *p) { return !((uintptr_t)p & 15); }
int done(bool ok) { return ok ? CSRST_OK : CSRST_E_CUDA; }

}  // namespace
int nn_backward_rows(const float *dy, const float *pre, float *dx32, void *dx16, void *dxT16, int rows, int cols,
                     void *stream) {
  if (!dy || !dx16 || !dxT16 || rows <= 0 || cols <= 0 || rows % 64 || cols % 64 || rows / 64 > 65535 ||
      !aligned16(dy) || !aligned16(pre) || !aligned16(dx32) || !aligned16(dx16) || !aligned16(dxT16))
    return CSRST_E_ARG;
  const dim3 g(cols / 64, rows / 64);
  return done(launch_chained(pre ? k_backward_rows<true> : k_backward_rows<false>, g, dim3(256), 0,
                             (cudaStream_t)stream, dy, pre, dx32, (__nv_bfloat16 *)dx16, (__nv_bfloat16 *)dxT16, rows,
                             cols));
}

}  // namespace csrst

using namespace csrst;

extern "C" {

// Whole 64 x 64 tiles with 16-byte rows go to k_transpose64, everything else to
// the 32 x 32 form (16384 x 128: 3.6 us, 6 there).
int csrst_nn_transpose_bf16(const void *src, void *dst, int batch, int rows, int cols, int ldd, void *stream) {
  if (!src || !dst || batch <= 0 || rows <= 0 || cols <= 0 || batch > 65535 || ldd < rows ||
      (rows + 31) / 32 > 65535)
    return CSRST_E_ARG;
  const __nv_bfloat16 *x = (const __nv_bfloat16 *)src;
  __nv_bfloat16 *y = (__nv_bfloat16 *)dst;
  if (rows % 64 == 0 && cols % 64 == 0 && ldd % 8 == 0 && aligned16(src) && aligned16(dst))
    return done(launch_chained(k_transpose64, dim3(cols / 64, rows / 64, batch), dim3(256), 0, (cudaStream_t)stream,
                               x, y, rows, cols, ldd));
  return done(launch_chained(k_transpose<__nv_bfloat16>, dim3((cols + 31) / 32, (rows + 31) / 32, batch), dim3(32, 8),
                             0, (cudaStream_t)stream, x, y, rows, cols, ldd));
}

// Rows in whole 32s with 16-byte destinations go to k_transpose32x128 (32 x
// 524288: 18.7 us, 45 with the 32 x 32 form).
int csrst_nn_transpose_b32(const void *src, void *dst, int batch, int rows, int cols, int ldd, void *stream) {
  if (!src || !dst || batch <= 0 || rows <= 0 || cols <= 0 || batch > 65535 || ldd < rows ||
      (rows + 31) / 32 > 65535 || ((uintptr_t)src & 3) || ((uintptr_t)dst & 3))
    return CSRST_E_ARG;
  const uint32_t *x = (const uint32_t *)src;
  uint32_t *y = (uint32_t *)dst;
  if (rows % 32 == 0 && ldd % 4 == 0 && aligned16(dst))
    return done(launch_chained(k_transpose32x128, dim3((cols + 127) / 128, rows / 32, batch), dim3(256), 0,
                               (cudaStream_t)stream, x, y, rows, cols, ldd));
  return done(launch_chained(k_transpose<uint32_t>, dim3((cols + 31) / 32, (rows + 31) / 32, batch), dim3(32, 8), 0,
                             (cudaStream_t)stream, x, y, rows, cols, ldd));
}

int csrst_nn_gelu_bwd(const float *dy, const float *pre, float *dx32, void *dx16, long long n, void *stream) {
  if (!dy || !pre || n <= 0) return CSRST_E_ARG;
  return done(launch_chained(k_gelu_bwd, dim3(grid_of(n)), dim3(256), 0, (cudaStream_t)stream, dy, pre, dx32,
                             (__nv_bfloat16 *)dx16, n));
}

// Four values a thread where both sides are 16-byte aligned (4.3e6 values: 7.3 us for 11.9).
int csrst_nn_cast_bf16(const float *x, void *y, long long n, void *stream) {
  if (!x || !y || n <= 0) return CSRST_E_ARG;
  if (n % 4 == 0 && aligned16(x) && aligned16(y))
    return done(launch_chained(k_cast4, dim3(grid_of(n / 4)), dim3(256), 0, (cudaStream_t)stream, (const float4 *)x,
                               (uint2 *)y, n / 4));
  return done(launch_chained(k_cast, dim3(grid_of(n)), dim3(256), 0, (cudaStream_t)stream, x, (__nv_bfloat16 *)y, n));
}

int csrst_nn_colsum(const float *x, int rows, int cols, float *part, float *out, int accumulate, void *stream) {
  if (!x || !part || !out || rows <= 0 || cols <= 0) return CSRST_E_ARG;
  const int slabs = (rows + 255) / 256;
  const dim3 g((cols + 31) / 32, slabs);
  cudaStream_t s = (cudaStream_t)stream;
  if (slabs == 1) return done(launch_chained(k_colsum_part, g, dim3(32), 0, s, x, rows, cols, out, accumulate));
  return done(launch_chained(k_colsum_part, g, dim3(32), 0, s, x, rows, cols, part, 0) &&
              launch_chained(k_colsum_final, dim3(g.x), dim3(32), 0, s, (const float *)part, slabs, cols, out,
                             accumulate));
}

int csrst_nn_mse(const float *pred, const float *target, const float *weight, long long n, float *grad, int gd,
                 long long g0, long long g1, double *part, double *loss, void *stream) {
  if (!pred || !target || !part || !loss || n <= 0 || gd <= 0) return CSRST_E_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  return done(launch_chained(k_mse, dim3(256), dim3(256), 0, s, pred, target, weight, n, grad, gd, g0, g1, part) &&
              launch_chained(k_sum_final, dim3(1), dim3(32), 0, s, (const double *)part, 256, n, loss));
}

int csrst_nn_adam_tick(int *t, float *coef, float lr0, float lr_min, int total, float b1, float b2, void *stream) {
  if (!t || !coef || total <= 0) return CSRST_E_ARG;
  return done(launch_chained(k_adam_tick, dim3(1), dim3(32), 0, (cudaStream_t)stream, t, coef, lr0, lr_min, total, b1,
                             b2));
}

int csrst_nn_adam(float *w, const float *g, float *m, float *v, long long n, const float *coef, float b1, float b2,
                  float eps, void *stream) {
  if (!w || !g || !m || !v || !coef || n <= 0) return CSRST_E_ARG;
  const long long n4 = aligned16(w) && aligned16(g) && aligned16(m) && aligned16(v) ? n / 4 : 0;
  return done(launch_chained(k_adam, dim3(grid_of(n4 ? n4 : n)), dim3(256), 0, (cudaStream_t)stream, w, g, m, v, n, n4,
                             coef, b1, b2, eps));
}

int csrst_nn_spectral_pack(const float *wr, const float *wi, int modes, int ch, void *mk, void *mkt, void *stream) {
  if (!wr || !wi || !mk || !mkt || modes <= 0 || ch <= 0) return CSRST_E_ARG;
  const bool pairs = !(((uintptr_t)mk | (uintptr_t)mkt) & 3);
  const unsigned t = (ch + 31) / 32;
  for (int k = 0; k < modes; k += 65535) {  // modes go to the grid's z
    const long long o = (long long)k * ch * ch;
    if (!launch_chained(pairs ? k_spectral_pack<true> : k_spectral_pack<false>,
                        dim3(t, t, modes - k < 65535 ? modes - k : 65535), dim3(32, 8), 0, (cudaStream_t)stream,
                        wr + o, wi + o, ch, (__nv_bfloat16 *)mk + 4 * o, (__nv_bfloat16 *)mkt + 4 * o))
      return CSRST_E_CUDA;
  }
  return CSRST_OK;
}

int csrst_nn_spectral_unpack(const float *dmk, int modes, int ch, float *dwr, float *dwi, void *stream) {
  if (!dmk || !dwr || !dwi || modes <= 0 || ch <= 0) return CSRST_E_ARG;
  const unsigned t = (ch + 31) / 32;
  for (int k = 0; k < modes; k += 65535) {
    const long long o = (long long)k * ch * ch;
    if (!launch_chained(k_spectral_unpack, dim3(t, t, modes - k < 65535 ? modes - k : 65535), dim3(32, 8), 0,
                        (cudaStream_t)stream, dmk + 4 * o, ch, dwr + o, dwi + o))
      return CSRST_E_CUDA;
  }
  return CSRST_OK;
}

}  // extern "C"
