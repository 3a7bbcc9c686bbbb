// FP32-mode current deposit with exact charge conservation.
//
// The reference deposits the current of every straight move old -> new as
// the path integral of its shape function (Zeroth/First/SecondOrderShape-
// Function: the segments between cell or dual-cell crossings, closed forms in
// the segment fraction tau).  That current is charge conserving: with the
// matching vertex charge shape S, rho(new) - rho(old) + dt div J = 0 holds
// per particle in exact arithmetic.  Evaluated in FP32 the identity would
// only hold to ~1e-7.  This file keeps it exact, in 64-bit integers, while the
// path integral itself runs in FP32:
//
//  1. charge: the 1D charge weights of both end points come from their exact
//     representation (integer cell + FP32 offset) in FP64 and are quantised
//     to the fixed-point unit as running sums, rows first: C(j) = round(K
//     sum_{j' <= j} Sy(j')), the last one K itself, R(j) = C(j) - C(j - 1);
//     then Q(i, j) = round(R(j) sum_{i' <= i} Sx(i')), the last one R(j),
//     rho(i, j) = Q(i, j) - Q(i - 1, j).  K = q * scale.  Every particle
//     carries exactly K, and no entry has to be set apart from the others.
//  2. Fy: the reference's y-current path integral in FP32 (flux units,
//     Fy = Jy dt hx / q) as running sums over the columns of a face row,
//     G(c, r), the last one the integer flux that the row charges force, Y(r) =
//     C_old(r) - C_new(r), and the ones right of the start vertex's column taken
//     down from it; Fy(c, r) = G(c, r) - G(c - 1, r).
//  3. Fx: continuity summed from the left edge of the stencil box,
//     Fx(c, r) = Q_old(c, r) - Q_new(c, r) - G(c, r) + G(c, r - 1):
//     three subtractions of sums that are there already.  On the box's right
//     edge it is R_old - R_new - Y(r) + Y(r - 1) = 0.
//
// The sums rather than the entries are rounded because the fluxes are
// differences of sums: entry-wise rounding needs the sums again, one entry per
// row corrected to the row's total, and its column found by selects.  For |K| <
// 2^50 a rounding is one FP64 FMA onto 1.5 * 2^52, whose low mantissa bits are
// then the integer; differences of two such numbers need no subtraction of
// the constant.
//
// So rho_new - rho_old + div F = 0 holds exactly in integers for the charge
// the particle carries, which is the FP64 charge shape to one fixed-point
// unit per weight.  In exact arithmetic step 3 reproduces the reference's
// path-integral Fx exactly (continuity determines Fx from Fy and rho), so the
// FP32 rounding of Fy moves Fx only by ~1e-7 of |Fy|, which is small against
// |Fx| for bunches moving along x.  A push deposits one component (TE/TM
// split): comp 0 emits Fx, comp 1 the corrected Fy; both run steps 1-2
// identically, so the two components of one move are consistent.
//
// Stencil box: the union of both end points' charge stencils, (S + 1) x
// (S + 1) vertices for a move of at most one cell per axis (S = 2, 3, 4 for
// shape orders 0, 1, 2).  Indices below are relative to the particle's old
// cell (ci, cj); a sink receives (i, j, value) in those coordinates: Fx at the
// x-face between vertices i and i + 1 of row j, Fy at the y-face between rows
// j and j + 1 of column i (the reference's Jx(i, j), Jy(i, j) elements).
#pragma once

// Plain arithmetic only (no CUDA runtime types), so that the host can compile
// this header too (the CPU test of the construction defines __device__,
// __forceinline__ and the two rounding conversions).
#include <math.h>
#include <stdlib.h>

#include "sinkbox.cuh"

namespace csrst {

template <int ORDER>
struct Flux32Shape;
// S: charge stencil width; OFF: first stencil vertex relative to the base
// index; DUAL: the path integral splits at dual-cell (half-integer) borders.
template <>
struct Flux32Shape<0> { static constexpr int S = 2, OFF = 0; static constexpr bool DUAL = false; };
template <>
struct Flux32Shape<1> { static constexpr int S = 3, OFF = -1; static constexpr bool DUAL = true; };
template <>
struct Flux32Shape<2> { static constexpr int S = 4, OFF = -1; static constexpr bool DUAL = false; };

// Arithmetic with one rounding per operation, whatever contraction the
// including file is compiled with: the compact and the general form of the
// deposit, and the stand-alone flux, must give the same integers.
#ifdef __CUDA_ARCH__
__device__ __forceinline__ float f_mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float f_add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float f_sub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float f_fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double d_mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double d_add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double d_sub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double d_fma(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ long long d_bits(double v) { return __double_as_longlong(v); }
#else
inline float f_mul(float a, float b) { return a * b; }
inline float f_add(float a, float b) { return a + b; }
inline float f_sub(float a, float b) { return a - b; }
inline float f_fma(float a, float b, float c) { return fmaf(a, b, c); }
inline double d_mul(double a, double b) { return a * b; }
inline double d_add(double a, double b) { return a + b; }
inline double d_sub(double a, double b) { return a - b; }
inline double d_fma(double a, double b, double c) { return fma(a, b, c); }
inline long long d_bits(double v) {
  long long b;
  __builtin_memcpy(&b, &v, sizeof b);
  return b;
}
#endif

// |T| below which round(T w), 0 <= w <= 1, is the low mantissa bits of
// fma(T, w, kRound): the sum stays in [2^52, 2^53), where the spacing is 1.
constexpr double kRoundMax = 1125899906842624.0;  // 2^50
constexpr double kRound = 6755399441055744.0;     // 1.5 * 2^52
constexpr long long kRoundBits = 0x4338000000000000ll;

__device__ __forceinline__ long long round_product(double T, double w) {
  if (fabs(T) < kRoundMax) return d_bits(d_fma(T, w, kRound)) - kRoundBits;
  return __double2ll_rn(d_mul(T, w));
}

// Base index of the offset o relative to its cell: floor(o), or floor(o + 1/2)
// for the quadratic shape, exactly.  (o + 0.5f rounds 0.5 - 2^-25 up to 1: a form
// chosen by that sum put such an end point's charge one row or column off.)
template <int ORDER>
__device__ __forceinline__ int base_index(float o) {
  const float f = floorf(o);
  return (int)f + (ORDER == 1 && f_sub(o, f) >= 0.5f ? 1 : 0);
}

// Whether a move of charge K takes the compact form of the deposit
// (flux_compact): it keeps its y base index, advances its x base index by 0 or 1,
// and |K| < kRoundMax.  The general form gives the same integers for it.
template <int ORDER>
__device__ __forceinline__ bool compact_form(float a0, float a1, int dc0, int dc1, float b0, float b1, double K) {
  return (unsigned)(dc0 + base_index<ORDER>(b0) - base_index<ORDER>(a0)) <= 1u &&
         dc1 + base_index<ORDER>(b1) == base_index<ORDER>(a1) && fabs(K) < kRoundMax;
}

// Base index (relative to the cell of the offset) and 1D charge weights of
// the offset o (cells): ZerothOrderShapeFunction.cpp:355-366 (CIC),
// FirstOrderShapeFunction.cpp:391-416 (quadratic), SecondOrderShapeFunction
// .cpp:408-441 (cubic), in FP64 on the exact offset.
template <int ORDER>
__device__ __forceinline__ int charge_weights(float o, double *w) {
  const int f = base_index<ORDER>(o);
  const double a = d_sub((double)o, (double)(float)f);
  if (ORDER == 0) {
    w[0] = d_sub(1.0, a); w[1] = a;
  } else if (ORDER == 1) {
    const double m = d_sub(0.5, a), p = d_add(0.5, a);
    w[0] = d_mul(d_mul(0.5, m), m);
    w[2] = d_mul(d_mul(0.5, p), p);
    w[1] = d_sub(d_sub(1.0, w[0]), w[2]);
  } else {
    const double b = d_sub(1.0, a), s6 = 1.0 / 6.0;
    w[0] = d_mul(s6, d_mul(d_mul(b, b), b));
    w[1] = d_mul(s6, d_sub(4.0, d_mul(d_mul(3.0, d_mul(a, a)), d_sub(2.0, a))));
    w[2] = d_mul(s6, d_sub(4.0, d_mul(d_mul(3.0, d_mul(b, b)), d_add(1.0, a))));
    w[3] = d_mul(s6, d_mul(d_mul(a, a), a));
  }
  return f;
}

// Running sums of the weights, all but the last (which is 1).
template <int ORDER>
__device__ __forceinline__ void running_sums(const double *w, double (&c)[Flux32Shape<ORDER>::S - 1]) {
  constexpr int S = Flux32Shape<ORDER>::S;
  c[0] = w[0];
  if constexpr (S == 4) c[1] = d_add(w[0], w[1]);
  if constexpr (S >= 3) c[S - 2] = d_sub(1.0, w[S - 1]);
}

// Quantised weights: differences of the rounded running sums, summing to Tint.
template <int ORDER>
__device__ __forceinline__ void quantise(const double *w, double T, long long Tint, long long *out) {
  constexpr int S = Flux32Shape<ORDER>::S;
  double c[S - 1];
  running_sums<ORDER>(w, c);
  long long prev = 0;
#pragma unroll
  for (int k = 0; k < S - 1; ++k) {
    const long long q = round_product(T, c[k]);
    out[k] = q - prev;
    prev = q;
  }
  out[S - 1] = Tint - prev;
}

// FP32 y-current path integral of one segment p -> e (cells, old-cell
// relative) with vertex (I, J) and segment fraction tau of a move of total
// displacement (d0, d1), in flux units Fy = Jy dt hx / q:
// ZerothOrderShapeFunction.cpp:279-290, FirstOrderShapeFunction.cpp:629-683
// (getCurrentY), SecondOrderShapeFunction.cpp:583-826 (Y branch).
// v[t][k]: the contribution to the face of column I - 1 + t (CIC: I + t) and
// face row J - 1 + k (CIC: J), t < S across, k < S - 1 along; only the columns
// whose bit is set in COLS are evaluated, the others are left unset.
template <int ORDER, int COLS>
__device__ __forceinline__ void fy_segment(float p0, float p1, float e0, float e1, int I, int J, float tau, float d0,
                                           float d1, float (&v)[Flux32Shape<ORDER>::S][Flux32Shape<ORDER>::S - 1]) {
  if constexpr (ORDER == 0) {
    const float c0 = f_mul(0.5f, f_add(p0, e0));
    const float D = f_mul(tau, d1);  // e1 - p1 without the cancellation of two O(1) coordinates
    if (COLS & 1) v[0][0] = f_mul(D, f_sub((float)(I + 1), c0));
    if (COLS & 2) v[1][0] = f_mul(D, f_sub(c0, (float)I));
  } else if constexpr (ORDER == 1) {
    const float third = 1.0f / 3.0f;
    const float a = f_sub(f_add((float)J, 0.5f), p1);  // along y: start to the face J + 1/2
    const float b = f_sub((float)I, p0);               // across x: vertex minus start
    const float tp2 = f_mul(f_mul(tau, tau), 0.5f), tp3 = f_mul(f_mul(tp2, tau), 2.0f * third);
    const float B = f_mul(d1, tau);                    // along y: B0 = -Bm
    const float um = f_sub(a, B), u0 = f_add(f_sub(1.0f, a), B);
    const float Cq = f_mul(f_mul(f_mul(0.5f, d0), d0), tp3), D2 = f_mul(d0, tp2);
    const float bl = f_add(0.5f, b), br = f_sub(0.5f, b);
#pragma unroll
    for (int t = 0; t < 3; ++t) {
      if (!(COLS >> t & 1)) continue;
      // terms of tau, tau^2 and tau^3 across
      const float A2 = t == 0   ? f_mul(f_mul(f_mul(0.5f, bl), bl), tau)
                       : t == 1 ? f_mul(f_fma(-b, b, 0.75f), tau)
                                : f_mul(f_mul(f_mul(0.5f, br), br), tau);
      const float B2 = t == 0 ? -f_mul(bl, D2) : t == 1 ? f_mul(f_mul(2.0f, b), D2) : f_mul(br, D2);
      const float C2 = t == 1 ? f_mul(-2.0f, Cq) : Cq;
      const float sm = f_add(f_add(A2, B2), C2);
      const float Bm = f_mul(B, f_fma(0.5f, A2, f_fma(third, B2, f_mul(0.25f, C2))));
      v[t][0] = f_mul(d1, f_fma(um, sm, Bm));
      v[t][1] = f_mul(d1, f_fma(u0, sm, -Bm));
    }
  } else {
    const float half = 0.5f, third = 1.0f / 3.0f, quarter = 0.25f, fifth = 0.2f, sixth = 1.0f / 6.0f;
    const float tp2 = f_mul(f_mul(tau, tau), half), tp3 = f_mul(f_mul(tp2, tau), 2.0f * third), tp4 = f_mul(tp2, tp2);
    const float a = f_sub(f_add((float)J, half), p1), b = f_sub((float)I, p0);
    const float dl = d1, dl2 = f_mul(d1, d1), de = d0, de2 = f_mul(d0, d0), de3 = f_mul(de2, de);
    const float ap = f_add(half, a), am = f_sub(half, a), dlt = f_mul(dl, tau), dlq = f_mul(dl2, tp2);
    const float sA[3] = {f_mul(f_mul(ap, ap), half), f_fma(-a, a, 0.75f), f_mul(f_mul(am, am), half)};
    const float sB[3] = {-f_mul(ap, dlt), f_mul(f_mul(2.0f, a), dlt), f_mul(am, dlt)};
    const float sC[3] = {f_mul(half, dlq), -dlq, f_mul(half, dlq)};
    const float bb = f_add(1.0f, b), b2 = f_mul(b, b), bb2 = f_mul(bb, bb);
    const float h2 = f_mul(half, f_mul(de, tp2)), h3 = f_mul(half, f_mul(de2, tp3)), s4 = f_mul(de3, tp4);
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      if (!(COLS >> t & 1)) continue;
      // terms of tau .. tau^4 across
      const float tA = t == 0   ? f_mul(f_mul(f_mul(bb2, bb), sixth), tau)
                       : t == 1 ? f_mul(f_mul(f_fma(f_mul(-3.0f, b2), f_add(2.0f, b), 4.0f), sixth), tau)
                       : t == 2 ? f_mul(f_mul(f_fma(f_mul(-3.0f, bb2), f_sub(1.0f, b), 4.0f), sixth), tau)
                                : -f_mul(f_mul(f_mul(b2, b), sixth), tau);
      const float tB = t == 0   ? -f_mul(bb2, h2)
                       : t == 1 ? f_mul(f_mul(b, f_fma(3.0f, b, 4.0f)), h2)
                       : t == 2 ? f_mul(f_fma(f_mul(-3.0f, b), b, f_fma(-2.0f, b, 1.0f)), h2)
                                : f_mul(b2, h2);
      const float tC = t == 0   ? f_mul(bb, h3)
                       : t == 1 ? -f_mul(f_fma(3.0f, b, 2.0f), h3)
                       : t == 2 ? f_mul(f_fma(3.0f, b, 1.0f), h3)
                                : -f_mul(b, h3);
      const float tD = f_mul(s4, t == 0 ? -sixth : t == 1 ? half : t == 2 ? -half : sixth);
      const float st = f_add(f_add(f_add(tD, tC), tB), tA), da = f_sub(tD, tA);
#pragma unroll
      for (int u = 0; u < 3; ++u) {
        float x = f_mul(f_add(f_add(sA[u], sB[u]), sC[u]), st);
        x = f_fma(f_fma(sC[u], da, -f_mul(sB[u], tB)), third, x);
        x = f_fma(f_fma(sC[u], tC, -f_mul(sB[u], tD)), fifth, x);
        x = f_fma(-f_mul(sB[u], tC), quarter, x);
        x = f_fma(-f_mul(sB[u], tA), half, x);
        v[t][u] = f_mul(dl, x);
      }
    }
  }
}

// Rounded running sums of Fy over a face row's columns 0 .. S - 1 of the box,
// from its columns in FP32 and its exact total Y: the columns left of the
// start vertex's sum up from the left edge, the ones right of it down from Y,
// so that the FP32 rounding of the row's total falls into the start vertex's
// column v.
template <int ORDER>
__device__ __forceinline__ void fy_sums(const float (&e)[Flux32Shape<ORDER>::S + 1], float Kf, long long Y, int v,
                                        long long (&G)[Flux32Shape<ORDER>::S]) {
  constexpr int S = Flux32Shape<ORDER>::S;
  long long left = 0, right = Y;
#pragma unroll
  for (int c = 0; c < S; ++c) {
    left += __float2ll_rn(f_mul(Kf, e[c]));
    if (c < v) G[c] = left;
  }
#pragma unroll
  for (int c = S; c > 0; --c) {
    right -= __float2ll_rn(f_mul(Kf, e[c]));
    if (c > v) G[c - 1] = right;
  }
}

// Border between base indices k and k + 1 of a path-integral split:
// k + 1 for cell borders, k + 1/2 for dual-cell borders.
template <bool DUAL>
__device__ __forceinline__ float split_border(int k) { return DUAL ? (float)k + 0.5f : (float)(k + 1); }

// Fraction of the move a + f d at coordinate X, clamped to [0, 1] (0 when
// the move has no extent along the axis).
__device__ __forceinline__ float cross_fraction(float X, float a, float d) {
  if (d == 0.0f) return 0.0f;
  return fminf(fmaxf(f_sub(X, a) / d, 0.0f), 1.0f);
}

// A row of a box's contributions at (i0 .. i0 + N - 1, j) to a sink: as one
// call if the sink takes rows, else entry by entry, zeros left out.
template <int N, class Sink>
__device__ __forceinline__ auto emit_row(Sink &s, int i0, int j, const long long (&v)[N], int)
    -> decltype(s.row(i0, j, v), void()) {
  s.row(i0, j, v);
}
template <int N, class Sink>
__device__ __forceinline__ void emit_row(Sink &s, int i0, int j, const long long (&v)[N], long) {
#pragma unroll
  for (int c = 0; c < N; ++c)
    if (v[c] != 0) s(i0 + c, j, v[c]);
}
// The displacement of a move, from its exact end points in FP64 (a difference
// of O(1) FP32 coordinates would carry an absolute error of their ulp).
__device__ __forceinline__ float displacement(int dc, float b, float a) {
  return (float)d_add((double)dc, d_sub((double)b, (double)a));
}

// The compact form of the deposit below, for the moves of compact_form (a bunch
// moving along +x at CFL <= 1, nearly every particle): the stencil box has
// S + 1 columns and S rows, start weights unshifted, and every index is a
// compile-time constant.  The second segment (from the x crossing on) is
// evaluated whether there is one or not, with tau = 0 if not: without
// branches the two segments' chains run side by side.
template <int ORDER, int COMP, class Sink>
__device__ __forceinline__ void flux_compact(float a0, float a1, int dc0, int dc1, float b0, float b1, double K,
                                             Sink &&sink) {
  using SH = Flux32Shape<ORDER>;
  constexpr int S = SH::S, BX = S + 1;
  const int IA = base_index<ORDER>(a0), JA = base_index<ORDER>(a1), IB = dc0 + base_index<ORDER>(b0);
  const bool wide = IB != IA;
  open_box<COMP == 0 ? BX - 1 : BX, COMP == 0 ? S : S - 1>(sink, IA + SH::OFF, JA + SH::OFF, 0);
  const double tK = d_add(K, kRound);
  double tA[S], tB[S];  // rounded running row charges of both end points, on kRound
  {
    double w[S], c[S - 1];
    charge_weights<ORDER>(a1, w);
    running_sums<ORDER>(w, c);
#pragma unroll
    for (int r = 0; r < S - 1; ++r) tA[r] = d_fma(K, c[r], kRound);
    charge_weights<ORDER>(b1, w);
    running_sums<ORDER>(w, c);
#pragma unroll
    for (int r = 0; r < S - 1; ++r) tB[r] = d_fma(K, c[r], kRound);
    tA[S - 1] = tB[S - 1] = tK;
  }
  // rounded running sums of Fy per face row
  long long G[S - 1][BX - 1], Y[S - 1];
  {
    const float d0 = displacement(dc0, b0, a0), d1 = displacement(dc1, b1, a1);
    const float te = wide ? cross_fraction(split_border<SH::DUAL>(IA), a0, d0) : 1.0f;
    const float m0 = f_fma(te, d0, a0), m1 = f_fma(te, d1, a1), n0 = f_add(a0, d0), n1 = f_add(a1, d1);
    // the columns fy_sums needs (all but the start vertex's): of the first
    // segment (box columns 0 .. S - 1) and of the second (1 .. S)
    constexpr int C1 = ORDER == 0 ? 0x2 : ORDER == 1 ? 0x5 : 0xd, C2 = ORDER == 0 ? 0x3 : ORDER == 1 ? 0x6 : 0xe;
    float v1[S][S - 1], v2[S][S - 1];
    fy_segment<ORDER, C1>(a0, a1, m0, m1, IA, JA, te, d0, d1, v1);
    fy_segment<ORDER, C2>(m0, m1, n0, n1, IB, JA, f_sub(1.0f, te), d0, d1, v2);
    const float Kf = (float)K;
#pragma unroll
    for (int r = 0; r < S - 1; ++r) {
      Y[r] = d_bits(tA[r]) - d_bits(tB[r]);
      float e[BX];
#pragma unroll
      for (int c = 0; c < BX; ++c) {
        const bool p = c < S && (C1 >> c & 1), q = c > 0 && (C2 >> (c > 0 ? c - 1 : 0) & 1);
        e[c] = p && q ? f_add(v1[c < S ? c : 0][r], v2[c > 0 ? c - 1 : 0][r])
               : p    ? v1[c < S ? c : 0][r]
               : q    ? v2[c > 0 ? c - 1 : 0][r]
                      : 0.0f;
      }
      fy_sums<ORDER>(e, Kf, Y[r], -SH::OFF, G[r]);
    }
  }
  if constexpr (COMP == 1) {
#pragma unroll
    for (int r = 0; r < S - 1; ++r) {
      long long f[BX];
      f[0] = G[r][0];
#pragma unroll
      for (int c = 1; c < BX - 1; ++c) f[c] = G[r][c] - G[r][c - 1];
      f[BX - 1] = Y[r] - G[r][BX - 2];
      emit_row<BX>(sink, IA + SH::OFF, JA + SH::OFF + r, f, 0);
    }
  } else {
    double ca[S - 1], cb[S];  // running x weights in the box frame
    {
      double w[S];
      charge_weights<ORDER>(a0, w);
      running_sums<ORDER>(w, ca);
      double c[S - 1];
      charge_weights<ORDER>(b0, w);
      running_sums<ORDER>(w, c);
#pragma unroll
      for (int k = 0; k < S; ++k) cb[k] = wide ? (k > 0 ? c[k - 1] : 0.0) : (k < S - 1 ? c[k] : 1.0);
    }
#pragma unroll
    for (int r = 0; r < S; ++r) {
      // this row's charges as exact doubles
      const double RA = d_sub(tA[r], r > 0 ? tA[r - 1] : kRound), RB = d_sub(tB[r], r > 0 ? tB[r - 1] : kRound);
      long long f[BX - 1];
#pragma unroll
      for (int c = 0; c < BX - 1; ++c) {
        const long long q = c < S - 1 ? d_bits(d_fma(RA, ca[c], kRound)) : d_bits(d_add(RA, kRound));
        f[c] = q - d_bits(d_fma(RB, cb[c], kRound));
        if (r < S - 1) f[c] -= G[r][c];
        if (r > 0) f[c] += G[r - 1][c];
      }
      emit_row<BX - 1>(sink, IA + SH::OFF, JA + SH::OFF + r, f, 0);
    }
  }
}

// The charge-conserving deposit of one move (see the top of the file).
// (a0, a1): start offset in cells from the old cell (ci, cj), any value;
// (dc0, dc1) = new cell - old cell, (b0, b1): end offset in the new cell;
// K = q * scale, Kint = its integer value.  COMP selects the emitted
// component; sink(i, j, v) gets old-cell-relative Jx / Jy indices.
// FAST: moves that allow the compact form take it.
// Returns false when the move spans more than one base index on an axis
// (more than one cell for CFL <= 1); nothing is emitted then.
template <int ORDER, int COMP, bool FAST, class Sink>
__device__ __forceinline__ bool flux_particle(float a0, float a1, int dc0, int dc1, float b0, float b1, double K,
                                              long long Kint, Sink &&sink) {
  using SH = Flux32Shape<ORDER>;
  if constexpr (FAST) {
    if (!compact_form<ORDER>(a0, a1, dc0, dc1, b0, b1, K))
      return flux_particle<ORDER, COMP, false>(a0, a1, dc0, dc1, b0, b1, K, Kint, sink);
    flux_compact<ORDER, COMP>(a0, a1, dc0, dc1, b0, b1, K, sink);
    return true;
  } else {
    constexpr int S = SH::S, OFF = SH::OFF, BX = S + 1, BY = S + 1;
    // 1. charge weights of both end points and their base indices (old-cell
    //    relative); the box starts at the lower base index of each axis
    double wAy[S], wBy[S], wAx[S], wBx[S];
    const int JA = charge_weights<ORDER>(a1, wAy), JB = dc1 + charge_weights<ORDER>(b1, wBy);
    const int IA = charge_weights<ORDER>(a0, wAx), IB = dc0 + charge_weights<ORDER>(b0, wBx);
    if (abs(JB - JA) > 1 || abs(IB - IA) > 1) return false;
    const int jmin = JA < JB ? JA : JB, imin = IA < IB ? IA : IB;
    const bool syA = JA != jmin, syB = JB != jmin, sxA = IA != imin, sxB = IB != imin;
    open_box<COMP == 0 ? BX - 1 : BX, COMP == 0 ? BY : BY - 1>(sink, imin + OFF, jmin + OFF, 0);
    long long RA[BY], RB[BY], Y[BY - 1];  // row charges and face-row fluxes in the box frame
    {
      long long q[S];
      quantise<ORDER>(wAy, K, Kint, q);
#pragma unroll
      for (int r = 0; r < BY; ++r) RA[r] = syA ? (r > 0 ? q[r - 1] : 0) : (r < S ? q[r] : 0);
      quantise<ORDER>(wBy, K, Kint, q);
#pragma unroll
      for (int r = 0; r < BY; ++r) RB[r] = syB ? (r > 0 ? q[r - 1] : 0) : (r < S ? q[r] : 0);
      long long y = 0;
#pragma unroll
      for (int r = 0; r < BY - 1; ++r) { y += RA[r] - RB[r]; Y[r] = y; }
    }

    // 2. running sums of the y-current path integral in FP32 over the segments
    //    between crossings, each moved into the box frame by its vertex's
    //    offset from the lower base index
    const float d0 = displacement(dc0, b0, a0), d1 = displacement(dc1, b1, a1);
    float fy[BY - 1][BX];
#pragma unroll
    for (int r = 0; r < BY - 1; ++r)
#pragma unroll
      for (int c = 0; c < BX; ++c) fy[r][c] = 0.0f;
    {
      const bool hx = IB != IA, hy = JB != JA;
      const float fx = hx ? cross_fraction(split_border<SH::DUAL>(imin), a0, d0) : 2.0f;
      const float fyc = hy ? cross_fraction(split_border<SH::DUAL>(jmin), a1, d1) : 2.0f;
      // up to three segments in order of the crossing fractions; the vertex of
      // the path switches from A's to B's index at each crossing
      const float f1 = fminf(fx, fyc), f2 = fmaxf(fx, fyc);
      const bool xfirst = fx <= fyc;
      float ts = 0.0f, p0 = a0, p1 = a1;
      int I = IA, J = JA;
#pragma unroll
      for (int sg = 0; sg < 3; ++sg) {
        const float te = sg == 2 ? 1.0f : sg == 0 ? fminf(f1, 1.0f) : fminf(f2, 1.0f);
        const float tau = f_sub(te, ts);
        const float e0 = te < 1.0f ? f_fma(te, d0, a0) : f_add(a0, d0);
        const float e1 = te < 1.0f ? f_fma(te, d1, a1) : f_add(a1, d1);
        if (tau > 0.0f) {
          float v[S][S - 1];
          fy_segment<ORDER, 0xf>(p0, p1, e0, e1, I, J, tau, d0, d1, v);
          const bool cx = I != imin, ry = J != jmin;
#pragma unroll
          for (int r = 0; r < BY - 1; ++r)
#pragma unroll
            for (int c = 0; c < BX; ++c) {
              const auto at = [&](int cc, int rr) { return cc >= 0 && cc < S && rr >= 0 && rr < S - 1 ? v[cc][rr] : 0.0f; };
              fy[r][c] = f_add(fy[r][c], cx ? (ry ? at(c - 1, r - 1) : at(c - 1, r)) : (ry ? at(c, r - 1) : at(c, r)));
            }
        }
        if (sg == 0 && f1 <= 1.0f) { if (xfirst) I = IB; else J = JB; }
        if (sg == 1 && f2 <= 1.0f) { if (xfirst) J = JB; else I = IB; }
        ts = te; p0 = e0; p1 = e1;
      }
    }

    // 3. the rounded sums' differences
    const float Kf = (float)K;
    long long prev[BX - 1];  // G of the face row below
#pragma unroll
    for (int c = 0; c < BX - 1; ++c) prev[c] = 0;
#pragma unroll
    for (int r = 0; r < BY; ++r) {
      long long G[BX - 1];
#pragma unroll
      for (int c = 0; c < BX - 1; ++c) G[c] = 0;
      if (r < BY - 1) fy_sums<ORDER>(fy[r < BY - 1 ? r : 0], Kf, Y[r < BY - 1 ? r : 0], IA - imin - OFF, G);
      if constexpr (COMP == 1) {
        if (r < BY - 1) {
          long long f[BX];
          f[0] = G[0];
#pragma unroll
          for (int c = 1; c < BX - 1; ++c) f[c] = G[c] - G[c - 1];
          f[BX - 1] = Y[r < BY - 1 ? r : 0] - G[BX - 2];
          emit_row<BX>(sink, imin + OFF, jmin + OFF + r, f, 0);
        }
      } else {
        long long qA[S], qB[S], f[BX - 1], sum = 0;
        quantise<ORDER>(wAx, (double)RA[r], RA[r], qA);
        quantise<ORDER>(wBx, (double)RB[r], RB[r], qB);
#pragma unroll
        for (int c = 0; c < BX - 1; ++c) {
          sum += (sxA ? (c > 0 ? qA[c - 1] : 0) : qA[c]) - (sxB ? (c > 0 ? qB[c - 1] : 0) : qB[c]);
          f[c] = sum - G[c] + prev[c];
        }
        emit_row<BX - 1>(sink, imin + OFF, jmin + OFF + r, f, 0);
      }
#pragma unroll
      for (int c = 0; c < BX - 1; ++c) prev[c] = G[c];
    }
    return true;
  }
}

}  // namespace csrst
