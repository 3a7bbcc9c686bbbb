// Deposit accumulation of the push kernels.
//
// A thread walks the cell-sorted bunch with a stride of one CTA, so the
// particles it deposits one after another mostly start in the same cell, and
// the 32 lanes of a warp work on neighbouring particles of that cell.
// Adding every contribution straight into the CTA's window accumulator would
// make those lanes collide on the same addresses; aggregating them across the
// warp first costs more instructions than the deposit itself.
//
// Instead each thread owns a small tile of shared memory around a base cell
// shared by its warp and adds its contributions there with plain loads and
// stores: tile entry k of thread t sits at k * blockDim + t, so the lanes of a
// warp always use different banks and never contend.  When the warp moves on
// to particles that start in another cell, each lane sums one tile entry over
// the warp's tiles and adds it to the window accumulator.  Contributions
// that fall outside the tile (large moves) go to the window accumulator
// directly.  All sums are 64-bit integers, so the result does not depend on
// the order of the additions.
#pragma once

#include "common.cuh"

namespace csrst {

constexpr int kPushThreads = 256;  // threads of every push CTA

// TW x TH tile covering window cells [bi - OX, bi - OX + TW) x [bj - OY, bj - OY + TH)
// around a base cell that all 32 lanes of the warp share, so that a re-base
// is one collective step: lane k sums entry k over the warp's 32 tiles and adds
// it to the destination.  rebase() and flush() must be called by all lanes of
// the warp together; add() may be called by any subset.
template <int TW, int TH, int OX, int OY>
struct TileAcc {
  static constexpr int kSize = TW * TH, kTW = TW, kTH = TH, kOX = OX, kOY = OY;
  static_assert(kSize <= 32, "flush() gives every entry a lane");
  unsigned long long *tile;  // shared memory, kSize * kPushThreads entries, zeroed
  int bi, bj;                // warp-uniform base cell (window cells)
  bool live;                 // warp-uniform: the tile may hold non-zero entries
  int ti0, tj0, ti1, tj1;    // window cells this lane added to (touched box)

  __device__ __forceinline__ void init(unsigned long long *t, int L0, int L1) {
    tile = t + threadIdx.x;
    bi = bj = -(1 << 28);
    live = false;
    ti0 = L0; tj0 = L1; ti1 = -1; tj1 = -1;
  }

  template <bool SHARED>
  __device__ __forceinline__ void touch(int i, int j) {
    if (SHARED) { ti0 = min(ti0, i); tj0 = min(tj0, j); ti1 = max(ti1, i); tj1 = max(tj1, j); }
  }

  // Adds everything held to dst (window cells, L0 x L1; global or shared).
  // Lane k walks the 32 lanes' copies of entry k, starting at its own, so that
  // the lanes of a warp stay on different banks: 32 loads in flight at once and
  // one atomic instruction, about 0.3 us, where a warp-wide sum per entry took
  // 2.3 - 4.5 us a flush and made the CTAs that cross a slice boundary (20 - 30
  // flushes) end half as late again as the others.
  template <bool SHARED>
  __device__ __forceinline__ void flush(unsigned long long *dst, int L0, int L1) {
    if (!live) return;
    const int lane = threadIdx.x & 31;
    __syncwarp();
    unsigned long long sum = 0ull;
    if (lane < kSize) {
      const unsigned long long *w = tile - lane + lane * kPushThreads;
#pragma unroll
      for (int t = 0; t < 32; ++t) sum += w[(t + lane) & 31];
    }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < kSize; ++k) tile[k * kPushThreads] = 0ull;
    if (sum) {
      const int i = bi - OX + lane % TW, j = bj - OY + lane / TW;
      if (i >= 0 && j >= 0 && i < L0 && j < L1) {
        atomicAdd(&dst[j * L0 + i], sum);
        touch<SHARED>(i, j);
      }
    }
    __syncwarp();
    live = false;
  }

  // Re-bases the warp's tile on the start cell of a middle lane of those that
  // have a particle (has) in this pass: they are sorted along x, so the tile
  // then reaches as far to either side.
  template <bool SHARED>
  __device__ __forceinline__ void rebase(bool has, int ci, int cj, unsigned long long *dst, int L0, int L1) {
    const unsigned m = __ballot_sync(0xffffffffu, has);
    if (!m) return;
    const int src = (m >> 16) & 1 ? 16 : __ffs(m) - 1;
    const int nbi = __shfl_sync(0xffffffffu, ci, src), nbj = __shfl_sync(0xffffffffu, cj, src);
    if (nbi != bi || nbj != bj) {
      flush<SHARED>(dst, L0, L1);
      bi = nbi; bj = nbj;
    }
    live = true;
  }

  template <bool SHARED>
  __device__ __forceinline__ void add(int i, int j, long long v, unsigned long long *dst, int L0, int L1) {
    const int a = i - (bi - OX), b = j - (bj - OY);
    if ((unsigned)a < (unsigned)TW && (unsigned)b < (unsigned)TH) {
      tile[(b * TW + a) * kPushThreads] += (unsigned long long)v;
    } else if (i >= 0 && j >= 0 && i < L0 && j < L1) {
      atomicAdd(&dst[j * L0 + i], (unsigned long long)v);
      touch<SHARED>(i, j);
    }
  }
};

// Adds one particle's deposit to its warp's tile.  A box of contributions is
// checked against the tile once (open_box); inside it every entry is a load, an
// add and a store at a compile-time offset from one address.  Boxes that do not
// fit go to the tile or the window accumulator entry by entry.  (wi, wj): the
// window cell that the deposit's indices are relative to.
template <class Tile>
struct TileSink {
  unsigned long long *tile;  // this lane's tile
  int bi, bj;                // its first window cell
  int wi, wj;                // the particle's old cell (window cells)
  unsigned long long *acc;
  int L0, L1;
  unsigned long long *p;
  int i0, j0;
  bool in;
  __device__ __forceinline__ TileSink(const Tile &t, int wi_, int wj_, unsigned long long *acc_, int L0_, int L1_)
      : tile(t.tile), bi(t.bi - Tile::kOX), bj(t.bj - Tile::kOY), wi(wi_), wj(wj_), acc(acc_), L0(L0_), L1(L1_) {}
  template <int NX, int NY>
  __device__ __forceinline__ void box(int i, int j) {
    const int a = wi + i - bi, b = wj + j - bj;
    // a box larger than the tile (the cubic shape's general form) never fits
    in = NX <= Tile::kTW && NY <= Tile::kTH && a >= 0 && a <= Tile::kTW - NX && b >= 0 && b <= Tile::kTH - NY;
    p = tile + (b * Tile::kTW + a) * kPushThreads;
    i0 = i; j0 = j;
  }
  template <int N>
  __device__ __forceinline__ void row(int i, int j, const long long (&v)[N]) {
    if (in) {
#pragma unroll
      for (int c = 0; c < N; ++c) p[((j - j0) * Tile::kTW + c) * kPushThreads] += (unsigned long long)v[c];
    } else {
#pragma unroll
      for (int c = 0; c < N; ++c)
        if (v[c] != 0) put(tile, wi + i + c - bi, wj + j - bj, acc, wi + i + c, wj + j, L0, L1, v[c]);
    }
  }
  __device__ __forceinline__ void one(int i, int j, long long v) {
    if (in) p[((j - j0) * Tile::kTW + (i - i0)) * kPushThreads] += (unsigned long long)v;
    else if (v != 0) put(tile, wi + i - bi, wj + j - bj, acc, wi + i, wj + j, L0, L1, v);
  }
  // one entry at (a, b) of the tile, window cell (i, j)
  static __device__ __forceinline__ void put(unsigned long long *tile, int a, int b, unsigned long long *acc, int i, int j,
                                          int L0, int L1, long long v) {
    if ((unsigned)a < (unsigned)Tile::kTW && (unsigned)b < (unsigned)Tile::kTH)
      tile[(b * Tile::kTW + a) * kPushThreads] += (unsigned long long)v;
    else if (i >= 0 && j >= 0 && i < L0 && j < L1)
      atomicAdd(&acc[j * L0 + i], (unsigned long long)v);
  }
};

// Tile shape per shape order: relative to the start cell of the particle the
// deposit of a move of less than half a cell along x and a little along y (CFL
// <= 0.5) lies in i in [-1, 2], j in [-1, 2] for CIC and TSC, i in [-1, 3] for the
// cubic shape, for both current components; one more column on each side lets
// the lanes of a warp start one cell before or after the warp's base cell.
// (Eight columns for CIC and TSC: 413 against 380 us per step, 8192 x 1024
// mesh, 4e6 TSC particles, FP32: 64 KB a CTA leave the field tiles no room beside it.)
template <int ORDER>
struct TileFor;
template <>
struct TileFor<0> { using T = TileAcc<6, 4, 2, 1>; };
template <>
struct TileFor<1> { using T = TileAcc<6, 4, 2, 1>; };
template <>
struct TileFor<2> { using T = TileAcc<7, 4, 2, 1>; };

}  // namespace csrst
