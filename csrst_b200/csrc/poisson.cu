// Initial fields of the bunch: the three boosted electrostatic solves of
// PoissonSolver::computeField (PoissonSolver.cpp:85-201) on the GPU.
//
// The matrix is the reference's (cutoffStencil, PoissonSolver.cpp:678-766): the
// 5-point Laplacian with spacings (gamma hx, hy) on the vertices that are
// inside the pipe or on a cut cell of area > 0.5 and lie before the bend
// (i < L_before / hx, Bend::getLengthStraightSection); every other row is an
// identity row.  Identity rows fix phi = b there, which moves their couplings
// to the right-hand side of the rows next to them; what remains is symmetric
// positive definite and is solved by CG preconditioned with one multigrid
// V-cycle:
//   - x-semicoarsening: the boosted x-spacing is gamma times the y-spacing,
//     so the operator couples along y about gamma^2 times more strongly and
//     only x is coarsened (columns are merged in pairs);
//   - Galerkin coarse operators R A P with P piecewise constant over a pair
//     of columns and R = P^T / 2; they keep the 5-point shape;
//   - zebra y-line Gauss-Seidel smoothing: a column is one tridiagonal system,
//     solved exactly by one warp from factors computed once per level.  The
//     pre-smoother (even columns, odd columns) and the post-smoother (odd, even)
//     mirror each other, so the V-cycle is a symmetric preconditioner.
// All arithmetic is FP64.  Vectors are stored column-major (i * ny + j), so a
// y-line is contiguous.  Dot products are two-pass block trees with a fixed
// grid, so a solve gives the same bits on every run.
//
// The lines' exactness takes most of a V-cycle's other passes away:
//   - the correction starts at zero, so the even columns' first solve reads
//     only their right-hand side, and after it and the odd columns' solve the
//     residual is zero on the odd columns and -(W u_west + E u_east) on the even
//     ones: the restricted residual is half of that, formed by the coarse
//     level's first solves as they load it;
//   - the post-smoother's odd solve overwrites the odd columns and reads the
//     even ones only as u + (coarse correction), and its even solve overwrites
//     those: the correction is added as it is read and never stored.
// So a level is four line launches, and the levels of at most kTailColumns
// columns, whose solves are latency, run as one launch of one CTA.
//
// 2048 x 512 mesh, 2e5 particles (8 V-cycles, with the bunch's upload): 7.4 ms,
// 37.3 with a solver that solved each line by cyclic reduction in a CTA (9.7 - 38
// us a launch, two divisions per row and pass), kept residual, restriction and
// prolongation passes, and allocated its 120 arrays one by one.  A line is 4 - 8
// us of latency now; the tail's 36 solves at 32 columns and more in one CTA
// (64 registers a thread) took 745 us a V-cycle, at 16 columns 146.
#include <algorithm>
#include <cmath>
#include <string>
#include <vector>

#include "kernels.cuh"
#include "shapes.cuh"

namespace csrst {
namespace {

// The stencil is symmetric (E of a column is W of the next, N of a row S of the
// next) and 0 towards inactive cells.  D and S of a coarse level are gone once
// its factors and the next level are there.
struct Level {
  int nx, ny;
  double *D, *W, *S;
  double d0;                  // the finest level's D on its active rows (D is nullptr there, 1 on the others)
  uint8_t *act;
  double *u, *f;              // correction, right-hand side
  double *fac;                // line factors (LineFactors)
};

constexpr int kDotBlocks = 1184, kPsumBlocks = 296;
constexpr int kMaxLineLen = 4096;  // y-line length the shared-memory solver takes

__device__ __forceinline__ long long gtid() { return blockIdx.x * (long long)blockDim.x + threadIdx.x; }

// Row classes: good = inside or a cut cell with area > 0.5; active = good and
// before the bend.  Column-major output.
__global__ void k_classes(const uint8_t *mask, const int *cutidx, const CutCellDev *cells, int Nx, int Ny,
                          long long maxX, uint8_t *good, uint8_t *act) {
  const long long k = gtid();
  if (k >= (long long)Nx * Ny) return;
  const int i = (int)(k / Ny), j = (int)(k % Ny);
  const size_t rm = (size_t)j * Nx + i;
  const int c = cutidx[rm];
  const bool g = mask[rm] || (c >= 0 && cells[c].area > 0.5);
  good[k] = g;
  act[k] = g && i < maxX;
}

__global__ void k_coeff0(Level L, double EW, double NS) {
  const long long k = gtid();
  if (k >= (long long)L.nx * L.ny) return;
  const int i = (int)(k / L.ny), j = (int)(k % L.ny);
  if (!L.act[k]) {
    L.W[k] = L.S[k] = 0.0;
    return;
  }
  L.W[k] = (i > 0 && L.act[k - L.ny]) ? EW : 0.0;
  L.S[k] = (j > 0 && L.act[k - 1]) ? NS : 0.0;
}

// Galerkin coarse stencil of a pair of columns (2I, 2I+1).
__global__ void k_coarsen(Level F, Level C) {
  const long long k = gtid();
  if (k >= (long long)C.nx * C.ny) return;
  const int I = (int)(k / C.ny), j = (int)(k % C.ny);
  const size_t a = (size_t)(2 * I) * F.ny + j, b = a + F.ny;
  const bool ha = F.act[a], hb = 2 * I + 1 < F.nx && F.act[b];
  if (!ha && !hb) {
    C.act[k] = 0;
    C.D[k] = 1.0; C.W[k] = C.S[k] = 0.0;
    return;
  }
  double D = 0.0, W = 0.0, S = 0.0;
  const double E = 2 * I + 1 < F.nx ? F.W[b] : 0.0;  // between the two
  if (ha) { D += (F.D ? F.D[a] : F.d0) + E; W += F.W[a]; S += F.S[a]; }
  if (hb) { D += (F.D ? F.D[b] : F.d0) + E; S += F.S[b]; }
  C.act[k] = 1;
  C.D[k] = 0.5 * D; C.W[k] = 0.5 * W; C.S[k] = 0.5 * S;
}

// A u at an active row of the finest level.
__device__ __forceinline__ double apply_at(const Level &L, const double *u, long long k) {
  const int i = (int)(k / L.ny), j = (int)(k % L.ny);
  double v = L.d0 * u[k];
  if (i > 0) v += L.W[k] * u[k - L.ny];
  if (i + 1 < L.nx) v += L.W[k + L.ny] * u[k + L.ny];
  if (j > 0) v += L.S[k] * u[k - 1];
  if (j + 1 < L.ny) v += L.S[k + 1] * u[k + 1];
  return v;
}

// --- y-line solves ------------------------------------------------------------
//
// One warp solves one column.  Lane i owns rows i m .. i m + m - 1 (m =
// ceil(ny / 32); rows past ny are identity rows): its last row is a separator
// with unknown X_i, the others, its interior, are eliminated: x = u + v X_{i-1}
// + w X_i with u from the lane's right-hand side by a Thomas sweep and v, w fixed
// by the matrix.  The separators' tridiagonal system is solved over the lanes by
// five cyclic-reduction steps.  Everything but u and the separators' right-hand
// side is computed once per level: per interior row l, g, h, v, w (forward
// multiplier, inverse pivot, back-substitution factor) and per lane the couplings
// of its separator, the ten reduction multipliers and the last inverse pivot.
constexpr int kRowFactors = 5, kLaneFactors = 13;

__host__ __device__ inline int line_rows(int ny) { return (ny + 31) / 32; }
__host__ __device__ inline size_t line_factors(int ny) {
  return (size_t)32 * (kRowFactors * line_rows(ny) + kLaneFactors);
}
// Shared memory of one warp's column, lane blocks an odd number of doubles apart.
__host__ __device__ inline int line_stride(int ny) { return line_rows(ny) | 1; }
__host__ __device__ inline size_t line_smem(int ny) { return (size_t)32 * line_stride(ny) * sizeof(double); }

// The factors of one level, one warp per column.
__global__ void __launch_bounds__(128) k_factor(Level L) {
  const int col = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (col >= L.nx) return;
  const int ny = L.ny, m = line_rows(ny), j0 = lane * m;
  const size_t base = (size_t)col * ny;
  double *F = L.fac + (size_t)col * line_factors(ny) + lane;
  auto row = [&](int j, double &a, double &b, double &c) {
    const bool in = j < ny;
    a = in ? L.S[base + j] : 0.0;
    b = !in ? 1.0 : L.D ? L.D[base + j] : L.act[base + j] ? L.d0 : 1.0;
    c = j + 1 < ny ? L.S[base + j + 1] : 0.0;
  };
  auto at = [&](int q, int k) -> double & { return F[(size_t)(k * kRowFactors + q) * 32]; };
  // interior rows k = 0 .. m - 2: pivots, v's forward sweep
  double den = 1.0, cp = 0.0, y = 0.0, a, b, c;
  for (int k = 0; k < m - 1; ++k) {
    row(j0 + k, a, b, c);
    const double l = k > 0 ? a / den : 0.0;
    den = b - l * cp;
    y = k > 0 ? -l * y : -a;
    cp = c;
    at(0, k) = l; at(1, k) = 1.0 / den; at(2, k) = c / den; at(3, k) = y;
  }
  double v = 0.0, w = 0.0;  // back substitution; w enters with -c of the last interior row
  for (int k = m - 2; k >= 0; --k) {
    const double g = at(1, k), h = at(2, k);
    v = k == m - 2 ? at(3, k) * g : at(3, k) * g - h * v;
    w = k == m - 2 ? -h : -h * w;
    at(3, k) = v; at(4, k) = w;
  }
  const double v0 = v, w0 = w;  // of the first interior row
  const double vl = m > 1 ? at(3, m - 2) : 0.0, wl = m > 1 ? at(4, m - 2) : 0.0;
  row(j0 + m - 1, a, b, c);
  const double vn = __shfl_down_sync(0xffffffffu, v0, 1), wn = __shfl_down_sync(0xffffffffu, w0, 1);
  if (lane == 31) c = 0.0;
  // the separators' system A X_{i-1} + B X_i + C X_{i+1} = D
  double A, B, C;
  if (m > 1) { A = a * vl; B = b + a * wl + c * vn; C = c * wn; }
  else { A = a; B = b; C = c; }
  double *G = F + (size_t)m * kRowFactors * 32;
  G[0] = m > 1 ? a : 0.0;
  G[32] = m > 1 ? c : 0.0;
#pragma unroll
  for (int t = 0; t < 5; ++t) {
    const int s = 1 << t;
    const double Au = __shfl_up_sync(0xffffffffu, A, s), Bu = __shfl_up_sync(0xffffffffu, B, s);
    const double Cu = __shfl_up_sync(0xffffffffu, C, s);
    const double Ad = __shfl_down_sync(0xffffffffu, A, s), Bd = __shfl_down_sync(0xffffffffu, B, s);
    const double Cd = __shfl_down_sync(0xffffffffu, C, s);
    const double al = lane >= s ? -A / Bu : 0.0, ga = lane + s < 32 ? -C / Bd : 0.0;
    A = lane >= s ? al * Au : 0.0;
    C = lane + s < 32 ? ga * Cd : 0.0;
    B = B + (lane >= s ? al * Cu : 0.0) + (lane + s < 32 ? ga * Ad : 0.0);
    G[(size_t)(2 + 2 * t) * 32] = al;
    G[(size_t)(3 + 2 * t) * 32] = ga;
  }
  G[(size_t)12 * 32] = 1.0 / B;
}

// What a line solve's right-hand side is made of (see the top of the file).
enum LineMode : int {
  kDown0,  // even column, zero start: f
  kDown1,  // odd column after them: f - W u_west - E u_east
  kUp1,    // odd column, the even ones corrected by the coarse level's u
  kPlain   // f - W u_west - E u_east
};

// Solves column `col` of level L; sm: this warp's shared memory.  In the down
// modes of a coarse level (fine != nullptr) f comes from the finer level and is
// stored; coarse: the next level, for kUp1.  The loads of a batch of rows are
// issued together, ahead of the stores and of the chains that use them (a line
// is latency: about 17 us with the loads inside the chains, 4 - 6 with these).
constexpr int kBatch = 8, kSweep = 16;

template <int MODE>
__device__ __forceinline__ void line_column(const Level &L, const Level *fine, const Level *coarse, int col,
                                            double *sm) {
  const int lane = threadIdx.x & 31, ny = L.ny, m = line_rows(ny), mp = m | 1;
  const unsigned inv = ((1u << 20) + m - 1) / m;  // j / m by a multiply for j < 32 m
  const size_t base = (size_t)col * ny;
  const bool restricted = (MODE == kDown0 || MODE == kDown1) && fine;
  const bool west = MODE != kDown0 && col > 0, east = MODE != kDown0 && col + 1 < L.nx;
  const size_t fb = (size_t)(2 * col) * ny;
  const bool fwest = restricted && col > 0, feast = restricted && 2 * col + 1 < fine->nx;
  const double *F = L.fac + (size_t)col * line_factors(ny) + lane;
  auto at = [&](int q, int k) { return __ldg(F + (size_t)(k * kRowFactors + q) * 32); };
  for (int t0 = 0; t0 < m; t0 += kBatch) {
    double d[kBatch], uw[kBatch], ue[kBatch], cw[kBatch], ce[kBatch], ew[kBatch], ee[kBatch];
    double fw[kBatch], fe[kBatch];
#pragma unroll
    for (int t = 0; t < kBatch; ++t) {
      const int j = lane + 32 * (t0 + t);
      const bool in = t0 + t < m && j < ny;
      const size_t k = base + j;
      d[t] = uw[t] = ue[t] = cw[t] = ce[t] = ew[t] = ee[t] = fw[t] = fe[t] = 0.0;
      if (!in) continue;
      if (restricted) {  // (fw, ew) and (fe, ee): the finer level's even column
        if (fwest) { fw[t] = __ldg(fine->W + fb + j); ew[t] = fine->u[fb + j - ny]; }
        if (feast) { fe[t] = __ldg(fine->W + fb + j + ny); ee[t] = fine->u[fb + j + ny]; }
      } else {
        d[t] = L.f[k];
      }
      if (west) { cw[t] = __ldg(L.W + k); uw[t] = L.u[k - ny]; }
      if (east) { ce[t] = __ldg(L.W + k + ny); ue[t] = L.u[k + ny]; }
      if (MODE == kUp1) {
        if (west) ew[t] = coarse->u[(size_t)((col - 1) / 2) * ny + j];
        if (east) ee[t] = coarse->u[(size_t)((col + 1) / 2) * ny + j];
      }
    }
#pragma unroll
    for (int t = 0; t < kBatch; ++t) {
      const unsigned j = lane + 32 * (t0 + t), q = (j * inv) >> 20;
      if (restricted) {
        d[t] = -0.5 * (fw[t] * ew[t] + fe[t] * ee[t]);
        ew[t] = ee[t] = 0.0;
        if (t0 + t < m && (int)j < ny) L.f[base + j] = d[t];
      }
      const double v = d[t] - cw[t] * (uw[t] + ew[t]) - ce[t] * (ue[t] + ee[t]);
      if (t0 + t < m) sm[q * mp + (j - q * m)] = v;
    }
  }
  double *x = sm + lane * mp;
  const double *G = F + (size_t)m * kRowFactors * 32;
  auto lf = [&](int q) { return __ldg(G + (size_t)q * 32); };
  double y = 0.0, u = 0.0, X;
  auto separators = [&]() {
    double al[5], ga[5];
#pragma unroll
    for (int t = 0; t < 5; ++t) { al[t] = lf(2 + 2 * t); ga[t] = lf(3 + 2 * t); }
    const double un = __shfl_down_sync(0xffffffffu, u, 1);
    double D = x[m - 1];
    if (m > 1) D = D - lf(0) * x[m - 2] - lf(1) * un;
#pragma unroll
    for (int t = 0; t < 5; ++t) {
      const double up = __shfl_up_sync(0xffffffffu, D, 1 << t), dn = __shfl_down_sync(0xffffffffu, D, 1 << t);
      D = D + al[t] * up + ga[t] * dn;
    }
    X = D * lf(12);
  };
  if (m - 1 <= kSweep) {  // (up to 544 rows) every factor in registers
    double f0[kSweep], f1[kSweep], f2[kSweep];
#pragma unroll
    for (int k = 0; k < kSweep; ++k) {
      const bool in = k < m - 1;
      f0[k] = in ? at(0, k) : 0.0; f1[k] = in ? at(1, k) : 0.0; f2[k] = in ? at(2, k) : 0.0;
    }
    __syncwarp();
    double v[kSweep];
#pragma unroll
    for (int k = 0; k < kSweep; ++k) {  // (row 0's l is 0)
      const double r = k < m - 1 ? x[k] : 0.0;
      y = r - f0[k] * y;
      v[k] = y;
    }
#pragma unroll
    for (int k = kSweep - 1; k >= 0; --k) {  // (past the interior: factors 0, u 0)
      u = v[k] * f1[k] - f2[k] * u;
      v[k] = u;
    }
#pragma unroll
    for (int k = 0; k < kSweep; ++k) {
      const bool in = k < m - 1;
      f0[k] = in ? at(3, k) : 0.0; f1[k] = in ? at(4, k) : 0.0;
      if (k == m - 2) x[k] = v[k];
    }
    separators();
    double XL = __shfl_up_sync(0xffffffffu, X, 1);
    if (lane == 0) XL = 0.0;
    x[m - 1] = X;
#pragma unroll
    for (int k = 0; k < kSweep; ++k)
      if (k < m - 1) x[k] = v[k] + (f0[k] * XL + f1[k] * X);
  } else {
    __syncwarp();
    for (int k0 = 0; k0 < m - 1; k0 += kSweep) {
      double f0[kSweep];
#pragma unroll
      for (int t = 0; t < kSweep; ++t) f0[t] = k0 + t < m - 1 ? at(0, k0 + t) : 0.0;
#pragma unroll
      for (int t = 0; t < kSweep; ++t)
        if (k0 + t < m - 1) {
          y = x[k0 + t] - f0[t] * y;
          x[k0 + t] = y;
        }
    }
    for (int k0 = (m - 2) / kSweep * kSweep; k0 >= 0; k0 -= kSweep) {
      double f1[kSweep], f2[kSweep];
#pragma unroll
      for (int t = 0; t < kSweep; ++t) {
        const bool in = k0 + t < m - 1;
        f1[t] = in ? at(1, k0 + t) : 0.0; f2[t] = in ? at(2, k0 + t) : 0.0;
      }
#pragma unroll
      for (int t = kSweep - 1; t >= 0; --t)
        if (k0 + t < m - 1) {
          u = x[k0 + t] * f1[t] - f2[t] * u;
          x[k0 + t] = u;
        }
    }
    separators();
    double XL = __shfl_up_sync(0xffffffffu, X, 1);
    if (lane == 0) XL = 0.0;
    x[m - 1] = X;
    for (int k0 = 0; k0 < m - 1; k0 += kSweep) {
      double f3[kSweep], f4[kSweep];
#pragma unroll
      for (int t = 0; t < kSweep; ++t) {
        const bool in = k0 + t < m - 1;
        f3[t] = in ? at(3, k0 + t) : 0.0; f4[t] = in ? at(4, k0 + t) : 0.0;
      }
#pragma unroll
      for (int t = 0; t < kSweep; ++t)
        if (k0 + t < m - 1) x[k0 + t] += f3[t] * XL + f4[t] * X;
    }
  }
  __syncwarp();
#pragma unroll 4
  for (int j = lane; j < ny; j += 32) {
    const unsigned q = ((unsigned)j * inv) >> 20;
    L.u[base + j] = sm[q * mp + (j - q * m)];
  }
  __syncwarp();
}

// One colour of one level: a warp per column.
template <int MODE>
__global__ void __launch_bounds__(128) k_line(const __grid_constant__ Level L, const __grid_constant__ Level other,
                                              int has_other, int colour) {
  extern __shared__ double line_sm[];
  const int w = threadIdx.x >> 5, col = 2 * (int)(blockIdx.x * (blockDim.x >> 5) + w) + colour;
  if (col >= L.nx) return;
  const Level *o = has_other ? &other : nullptr;
  line_column<MODE>(L, MODE == kUp1 ? nullptr : o, MODE == kUp1 ? o : nullptr, col,
                    line_sm + (size_t)w * 32 * line_stride(L.ny));
}

// The coarse levels [lt, nl) of a V-cycle, down and up again, in one CTA: lv
// points at level lt (with the finer level before it when has_fine).
constexpr int kTailColumns = 16;  // 8 warps: a line keeps some 150 registers a thread
constexpr int kMaxLevels = 24;
struct TailLevels {
  Level lv[kMaxLevels];
  int n, has_fine;  // lv[0 .. n): with the finer level first when has_fine
};

__global__ void __launch_bounds__(kTailColumns / 2 * 32, 1) k_tail(const __grid_constant__ TailLevels t) {
  extern __shared__ double line_sm[];
  const int w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const Level &first = t.lv[t.has_fine];
  double *sm = line_sm + (size_t)w * 32 * line_stride(first.ny);
  const int last = t.n - 1;
  for (int l = t.has_fine; l <= last; ++l) {
    const Level &L = t.lv[l];
    const Level *fine = l > 0 ? &t.lv[l - 1] : nullptr;
    for (int c = 2 * w; c < L.nx; c += 2 * nw) line_column<kDown0>(L, fine, nullptr, c, sm);
    __syncthreads();
    for (int c = 2 * w + 1; c < L.nx; c += 2 * nw) line_column<kDown1>(L, fine, nullptr, c, sm);
    __syncthreads();
  }
  for (int k = 0; k < 7; ++k) {  // the coarsest level: even, odd, ... nine solves in all, the last one even
    const Level &L = t.lv[last];
    for (int c = 2 * w + (k & 1); c < L.nx; c += 2 * nw) line_column<kPlain>(L, nullptr, nullptr, c, sm);
    __syncthreads();
  }
  for (int l = last - 1; l >= t.has_fine; --l) {
    const Level &L = t.lv[l];
    for (int c = 2 * w + 1; c < L.nx; c += 2 * nw) line_column<kUp1>(L, nullptr, &t.lv[l + 1], c, sm);
    __syncthreads();
    for (int c = 2 * w; c < L.nx; c += 2 * nw) line_column<kPlain>(L, nullptr, nullptr, c, sm);
    __syncthreads();
  }
}

// --- CG vector kernels -------------------------------------------------------

// Scalars of a solve on the device: the iteration's alpha and beta never
// wait for the host, which reads one residual norm per iteration.
struct Scalars {
  double *part;    // kDotBlocks partial sums
  double *v;       // results
  unsigned *done;  // blocks that ended
};
enum : int { kSBn2, kSRr, kSDq, kSRz0, kSRz1, kSCount };

// Ends a reduction kernel of kDotBlocks blocks of 256 threads: each thread's
// sum s, tree over the block, then the last block's tree over the blocks' sums
// into v[slot].  The order of the additions is fixed.
__device__ __forceinline__ void reduce_to(const Scalars &S, double s, int slot) {
  __shared__ double sh[256];
  __shared__ bool last;
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w) sh[threadIdx.x] += sh[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    S.part[blockIdx.x] = sh[0];
    __threadfence();
    last = atomicAdd(S.done, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  const volatile double *part = S.part;
  s = 0.0;
  for (int k = threadIdx.x; k < (int)gridDim.x; k += 256) s += part[k];
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w) sh[threadIdx.x] += sh[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    S.v[slot] = sh[0];
    *S.done = 0u;
  }
}

__global__ void __launch_bounds__(256) k_dot(const double *a, const double *b, long long n, Scalars S, int slot) {
  double s = 0.0;
  for (long long k = blockIdx.x * 256ll + threadIdx.x; k < n; k += (long long)gridDim.x * 256) s += a[k] * b[k];
  reduce_to(S, s, slot);
}

// q = A d and d . q
__global__ void __launch_bounds__(256) k_apply_dot(const __grid_constant__ Level L, const double *d, double *q,
                                                   Scalars S) {
  const long long n = (long long)L.nx * L.ny;
  double s = 0.0;
  for (long long k = blockIdx.x * 256ll + threadIdx.x; k < n; k += (long long)gridDim.x * 256) {
    const double v = L.act[k] ? apply_at(L, d, k) : 0.0;
    q[k] = v;
    s += d[k] * v;
  }
  reduce_to(S, s, kSDq);
}

// u += alpha d, r -= alpha q with alpha = rz / dq, and r . r
__global__ void __launch_bounds__(256) k_axpy_dot(double *u, double *r, const double *d, const double *q, long long n,
                                                  Scalars S, int rz) {
  const double alpha = S.v[rz] / S.v[kSDq];
  double s = 0.0;
  for (long long k = blockIdx.x * 256ll + threadIdx.x; k < n; k += (long long)gridDim.x * 256) {
    u[k] += alpha * d[k];
    const double v = r[k] - alpha * q[k];
    r[k] = v;
    s += v * v;
  }
  reduce_to(S, s, kSRr);
}

// r = f - A x and r . r
__global__ void __launch_bounds__(256) k_residual_dot(const __grid_constant__ Level L, const double *f, const double *x,
                                                      double *r, Scalars S) {
  const long long n = (long long)L.nx * L.ny;
  double s = 0.0;
  for (long long k = blockIdx.x * 256ll + threadIdx.x; k < n; k += (long long)gridDim.x * 256) {
    const double v = f[k] - (L.act[k] ? apply_at(L, x, k) : 0.0);
    r[k] = v;
    s += v * v;
  }
  reduce_to(S, s, kSRr);
}

// d = z + beta d with beta = rz_new / rz_old (first: d = z)
__global__ void k_direction(double *d, const double *z, long long n, Scalars S, int rz_new, int rz_old, int first) {
  const long long k = gtid();
  if (k >= n) return;
  d[k] = first ? z[k] : z[k] + (S.v[rz_new] / S.v[rz_old]) * d[k];
}

__global__ void k_sum_parts(const double *part, int np, double *out) {
  __shared__ double sh[512];
  sh[threadIdx.x] = threadIdx.x < np ? part[threadIdx.x] : 0.0;
  __syncthreads();
  for (int w = 256; w > 0; w >>= 1) {
    if (threadIdx.x < w) sh[threadIdx.x] += sh[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = sh[0];
}

// --- right-hand side, shifts and fields ----------------------------------------

__global__ void k_psum(const double *px, const double *py, const double *q, long long n, double *part) {
  __shared__ double sh[3][256];
  double a = 0.0, b = 0.0, c = 0.0;
  for (long long k = blockIdx.x * 256ll + threadIdx.x; k < n; k += (long long)gridDim.x * 256) {
    a += px[k]; b += py[k]; c += fabs(q[k]);
  }
  sh[0][threadIdx.x] = a; sh[1][threadIdx.x] = b; sh[2][threadIdx.x] = c;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w)
      for (int t = 0; t < 3; ++t) sh[t][threadIdx.x] += sh[t][threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0)
    for (int t = 0; t < 3; ++t) part[t * kPsumBlocks + blockIdx.x] = sh[t][0];
}

// Charge of the bunch at the positions of one solve (mode 0: R + dt/2 drift;
// 1: that, drifted back and moved by -hx/2 in x; 2: R), accumulated in 64-bit
// fixed point on the row-major Nx x Ny vertices, the lanes of a warp that hit
// the same vertex together (the bunch is sorted by cell: one atomic per vertex
// and particle took 101 us a solve for 2e5 particles).
template <int ORDER>
__global__ void k_rho(const double *x, const double *y, const double *px, const double *py, const double *q,
                      long long n, int mode, double full, double back, double mv, double org0, double org1,
                      double h0, double h1, int Nx, int Ny, unsigned long long *acc, double scale) {
  for (long long k = gtid(); k < n; k += (long long)gridDim.x * blockDim.x) {
    double X = x[k], Y = y[k];
    if (mode < 2) {
      const double p0 = px[k], p1 = py[k];
      const double r = inv_gamma(p0, p1);
      X = X + full * p0 * r; Y = Y + full * p1 * r;
      if (mode == 1) { X = (X + back * p0 * r) + mv; Y = (Y + back * p1 * r) + 0.0; }
    }
    charge_shape<ORDER>(X, Y, q[k], org0, org1, h0, h1, [&](int i, int j, double v) {
      const bool in = i >= 0 && j >= 0 && i < Nx && j < Ny;
      warp_add(acc, in ? j * Nx + i : -1, __double2ll_rn(v * scale));
    });
  }
}

// b = rho / (eps0 gamma), column-major; rho = (fixed-point sum) / (hx hy).
__global__ void k_rhs(const unsigned long long *acc, double inv, double area, double cc, int Nx, int Ny,
                      double *b) {
  const long long k = gtid();
  if (k >= (long long)Nx * Ny) return;
  const int i = (int)(k / Ny), j = (int)(k % Ny);
  b[k] = ((double)(long long)acc[(size_t)j * Nx + i] * inv / area) * cc;
}

// Right-hand side of the active rows: b minus the couplings to identity rows.
__global__ void k_rhs_eff(Level L, const uint8_t *good, const double *b, double EW, double NS, double *f) {
  const long long k = gtid();
  if (k >= (long long)L.nx * L.ny) return;
  if (!L.act[k]) { f[k] = 0.0; return; }
  const int i = (int)(k / L.ny), j = (int)(k % L.ny);
  double v = b[k];
  if (j > 0 && good[k - 1] && !L.act[k - 1]) v -= NS * b[k - 1];
  if (i > 0 && good[k - L.ny] && !L.act[k - L.ny]) v -= EW * b[k - L.ny];
  if (i + 1 < L.nx && good[k + L.ny] && !L.act[k + L.ny]) v -= EW * b[k + L.ny];
  if (j + 1 < L.ny && good[k + 1] && !L.act[k + 1]) v -= NS * b[k + 1];
  f[k] = v;
}

// Initial guess from the previous solution (shiftLHS, PoissonSolver.cpp:270-303):
// tau = +1 takes the right neighbour, tau = -1/2 mixes in the left one.
__global__ void k_shift(const double *phi, const uint8_t *act, double *out, double tau, int Nx, int Ny) {
  const long long k = gtid();
  if (k >= (long long)Nx * Ny) return;
  if (!act[k]) { out[k] = 0.0; return; }
  const int i = (int)(k / Ny);
  if (tau > 0) {
    const double nb = i + 1 < Nx ? phi[k + Ny] : 0.0;
    out[k] = phi[k] + (tau * nb - tau * phi[k]);
  } else {
    const double t = -tau;
    const double nb = i > 0 ? phi[k - Ny] : 0.0;
    out[k] = phi[k] + (t * nb - t * phi[k]);
  }
}

__global__ void k_finish(const uint8_t *act, const double *u, const double *b, double *phi, long long n) {
  const long long k = gtid();
  if (k < n) phi[k] = act[k] ? u[k] : b[k];
}

// PoissonSolver::fillFields (PoissonSolver.cpp:441-507): Ey from the first
// potential, Hz (both split halves) from the second, Ex from the third; the
// guard beyond the last row / column holds zero.
__global__ void k_fields(const double *phi1, const double *phi2, const double *phi3, int Nx, int Ny,
                         double gamma, double hr0, double hr1, double bg, double hden, Plane Ex, Plane Ey,
                         Plane Hx, Plane Hy) {
  const long long t = gtid();
  if (t >= (long long)Nx * Ny) return;
  const int i = (int)(t % Nx), j = (int)(t / Nx);
  const size_t k = (size_t)i * Ny + j;
  const double ey0 = gamma * phi1[k] / hr1;
  const double ey1 = j + 1 < Ny ? gamma * phi1[k + 1] / hr1 : 0.0;
  Ey.at(i, j) = ey0 - ey1;
  const double h0v = bg * phi2[k] / hden;
  const double h1v = j + 1 < Ny ? bg * phi2[k + 1] / hden : 0.0;
  Hx.at(i, j) = h0v - h1v;
  Hy.at(i, j) = h0v - h1v;
  const double ex0 = phi3[k] / hr0;
  const double ex1 = i + 1 < Nx ? phi3[k + Ny] / hr0 : 0.0;
  Ex.at(i, j) = ex0 - ex1;
}

inline unsigned blocks_for(long long n, int bs = 256) { return (unsigned)((n + bs - 1) / bs); }

// Device memory of one call, carved from one allocation: sized first (base ==
// nullptr), then handed out in the same order.
struct Arena {
  char *base = nullptr;
  size_t used = 0;
  template <class T>
  T *get(size_t count) {
    used = (used + 255) / 256 * 256;
    T *p = base ? reinterpret_cast<T *>(base + used) : nullptr;
    used += (count > 0 ? count : 1) * sizeof(T);
    return p;
  }
};

struct Work {
  double *part, *scal;
  unsigned *done;
  std::vector<Level> lv;
  uint8_t *good;
  double *b, *r, *d, *q, *phi[3];
  double *f;                // the right-hand side, until the first search direction takes its place (d)
  unsigned long long *acc;  // the charge, until the first A d does (q)
  void carve(Arena &A, int Nx, int Ny) {
    const size_t m = (size_t)Nx * Ny;
    part = A.get<double>(std::max(kDotBlocks, 3 * kPsumBlocks)); scal = A.get<double>(8); done = A.get<unsigned>(1);
    good = A.get<uint8_t>(m);
    for (double **p : {&b, &r, &d, &q, &phi[0], &phi[1], &phi[2]}) *p = A.get<double>(m);
    f = d;
    static_assert(sizeof(unsigned long long) == sizeof(double), "acc shares q's place");
    acc = reinterpret_cast<unsigned long long *>(q);
    lv.clear();
    // D and S of the coarse levels, in turns: a level's are read by its factors and the next level only
    const size_t c1 = (size_t)((Nx + 1) / 2) * Ny, c2 = (size_t)((Nx + 3) / 4) * Ny;
    double *D[2] = {A.get<double>(c1), A.get<double>(c2)}, *S[2] = {A.get<double>(c1), A.get<double>(c2)};
    for (int nx = Nx;; nx = (nx + 1) / 2) {
      Level L{};
      L.nx = nx; L.ny = Ny;
      const size_t c = (size_t)nx * Ny;
      for (double **p : {&L.W, &L.u}) *p = A.get<double>(c);
      if (lv.empty()) L.S = A.get<double>(c);
      else { L.D = D[(lv.size() - 1) & 1]; L.S = S[(lv.size() - 1) & 1]; }
      L.act = A.get<uint8_t>(c);
      L.f = lv.empty() ? r : A.get<double>(c);  // the finest level's right-hand side is CG's residual
      L.fac = A.get<double>((size_t)nx * line_factors(Ny));
      lv.push_back(L);
      if (nx <= 2) break;
    }
  }
};

class Solver {
 public:
  Solver(const std::vector<Level> &lv, cudaStream_t s) : lv_(lv), s_(s) {
    const int nl = (int)lv.size(), ny = lv[0].ny;
    lt_ = 0;
    while (lt_ + 1 < nl && lv[lt_].nx > kTailColumns) ++lt_;
    tail_.has_fine = lt_ > 0 ? 1 : 0;
    tail_.n = nl - lt_ + tail_.has_fine;
    for (int k = 0; k < tail_.n; ++k) tail_.lv[k] = lv[lt_ - tail_.has_fine + k];
    smem_ = line_smem(ny);
    // a warp for every column of the tail's widest colour, as many as shared memory takes
    const size_t fit = kSmemMax / smem_, want = (size_t)(lv[lt_].nx + 1) / 2;
    tail_warps_ = (int)std::max<size_t>(1, std::min<size_t>({fit, want, kTailColumns / 2}));
    line_warps_ = (int)std::max<size_t>(1, std::min<size_t>(fit, 4));
  }

  cudaError_t opt_in() {
    cudaError_t e = cudaSuccess;
    auto one = [&](auto *k, size_t b) {
      if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)b);
    };
    one(k_line<kDown0>, kSmemMax); one(k_line<kDown1>, kSmemMax);
    one(k_line<kUp1>, kSmemMax); one(k_line<kPlain>, kSmemMax);
    one(k_tail, kSmemMax);
    return e;
  }

  // lv[0].u = V-cycle(lv[0].f), zero initial correction.
  void vcycle() {
    for (int l = 0; l < lt_; ++l) {
      line<kDown0>(l, l - 1, 0);
      line<kDown1>(l, l - 1, 1);
    }
    k_tail<<<1, 32 * tail_warps_, tail_warps_ * smem_, s_>>>(tail_);
    for (int l = lt_ - 1; l >= 0; --l) {
      line<kUp1>(l, l + 1, 1);
      line<kPlain>(l, -1, 0);
    }
  }

 private:
  template <int MODE>
  void line(int l, int other, int colour) {
    const int ncol = (lv_[l].nx - colour + 1) / 2;
    if (ncol <= 0) return;
    k_line<MODE><<<(ncol + line_warps_ - 1) / line_warps_, 32 * line_warps_, line_warps_ * smem_, s_>>>(
        lv_[l], lv_[other >= 0 ? other : l], other >= 0, colour);
  }

  static constexpr size_t kSmemMax = 200 * 1024;
  const std::vector<Level> &lv_;
  TailLevels tail_;
  int lt_ = 0, tail_warps_ = 1, line_warps_ = 1;
  size_t smem_ = 0;
  cudaStream_t s_;
};

}  // namespace

int poisson_initial_fields(const PoissonInput &in, PoissonReport *rep, cudaStream_t s, std::string *msg) {
  const int Nx = in.b.Nx, Ny = in.b.Ny;
  const long long m = (long long)Nx * Ny;
  auto fail = [&](const char *what, cudaError_t e) {
    if (msg) *msg = std::string(what) + (e != cudaSuccess ? std::string(": ") + cudaGetErrorString(e) : "");
    return e != cudaSuccess ? kErrCuda : kErrArg;
  };
  if (in.n <= 0) return fail("no particles", cudaSuccess);
  if (Ny > kMaxLineLen) return fail("the multigrid line solver takes at most 4096 rows", cudaSuccess);
  cudaError_t e;
  Work w;
  Arena arena;
  w.carve(arena, Nx, Ny);
  ScratchBuffer mem(s);
  if ((e = mem.alloc(arena.used)) != cudaSuccess) return fail("cudaMalloc (multigrid hierarchy)", e);
  arena.base = static_cast<char *>(mem.p);
  arena.used = 0;
  w.carve(arena, Nx, Ny);
  const std::vector<Level> &lv = w.lv;
  double *part = w.part, *scal = w.scal;
  // mean momentum and total |q| (Distribution::get_pmean)
  k_psum<<<kPsumBlocks, 256, 0, s>>>(in.px, in.py, in.q, in.n, part);
  for (int t = 0; t < 3; ++t) k_sum_parts<<<1, 512, 0, s>>>(part + t * kPsumBlocks, kPsumBlocks, scal + t);
  double sums[3];
  e = cudaMemcpyAsync(sums, scal, sizeof(sums), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(w.done, 0, sizeof(unsigned), s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return fail("momentum sum", e);
  const double pm0 = sums[0] / (double)in.n, pm1 = sums[1] / (double)in.n;
  const double gamma = std::sqrt((pm0 * pm0 + pm1 * pm1) + 1);
  const double hr0 = in.b.hr0 * gamma, hr1 = in.b.hr1;
  const double EW = -1 / (hr0 * hr0), NS = -1 / (hr1 * hr1), Dc = -2 * (EW + NS);
  const long long maxX = (long long)(size_t)(in.b.Lb / in.b.hr0);

  k_classes<<<blocks_for(m), 256, 0, s>>>(in.mask, in.cutidx, in.cells, Nx, Ny, maxX, w.good, lv[0].act);
  w.lv[0].d0 = Dc;
  k_coeff0<<<blocks_for(m), 256, 0, s>>>(lv[0], EW, NS);
  for (size_t l = 0; l < lv.size(); ++l) {
    if (l > 0) k_coarsen<<<blocks_for((long long)lv[l].nx * Ny), 256, 0, s>>>(lv[l - 1], lv[l]);
    k_factor<<<(lv[l].nx + 3) / 4, 128, 0, s>>>(lv[l]);
  }
  Solver sv(lv, s);
  if ((e = sv.opt_in()) != cudaSuccess) return fail("line solver shared memory", e);
  const Scalars S{part, scal, w.done};
  auto read = [&](int slot, double *out) {
    cudaError_t c = cudaMemcpyAsync(out, scal + slot, sizeof(double), cudaMemcpyDeviceToHost, s);
    return c == cudaSuccess ? cudaStreamSynchronize(s) : c;
  };
  const double area = in.b.hr0 * in.b.hr1, cc = 1 / (kEps0 * gamma);
  const double qsum = sums[2] > 0 ? sums[2] : 1e-300;
  const double scale = std::ldexp(1.0, (int)std::floor(std::log2(std::ldexp(1.0, 62) / qsum)));
  const double full = (in.dt / 2) * kC, back = (-in.dt / 2) * kC, mv = -0.5 * hr0 / gamma;
  const unsigned pg = blocks_for(in.n) < 4096 ? blocks_for(in.n) : 4096;
  const double tols[3] = {in.tol_first, in.tol_rest, in.tol_rest};
  double *r = w.r, *z = lv[0].u;
  for (int sol = 0; sol < 3; ++sol) {
    double *x = w.phi[sol];
    // right-hand side of this solve
    cudaMemsetAsync(w.acc, 0, m * sizeof(unsigned long long), s);
    const int mode = sol;  // 0: R + dt/2 drift, 1: shifted by -hx/2, 2: R
    if (in.order == 0)
      k_rho<0><<<pg, 256, 0, s>>>(in.x, in.y, in.px, in.py, in.q, in.n, mode, full, back, mv, in.b.org0,
                                  in.b.org1, in.b.hr0, in.b.hr1, Nx, Ny, w.acc, scale);
    else if (in.order == 1)
      k_rho<1><<<pg, 256, 0, s>>>(in.x, in.y, in.px, in.py, in.q, in.n, mode, full, back, mv, in.b.org0,
                                  in.b.org1, in.b.hr0, in.b.hr1, Nx, Ny, w.acc, scale);
    else
      k_rho<2><<<pg, 256, 0, s>>>(in.x, in.y, in.px, in.py, in.q, in.n, mode, full, back, mv, in.b.org0,
                                  in.b.org1, in.b.hr0, in.b.hr1, Nx, Ny, w.acc, scale);
    k_rhs<<<blocks_for(m), 256, 0, s>>>(w.acc, 1.0 / scale, area, cc, Nx, Ny, w.b);
    k_rhs_eff<<<blocks_for(m), 256, 0, s>>>(lv[0], w.good, w.b, EW, NS, w.f);
    // initial guess: 0, then the shifted previous potential
    if (sol == 0) cudaMemsetAsync(x, 0, m * sizeof(double), s);
    else k_shift<<<blocks_for(m), 256, 0, s>>>(w.phi[sol - 1], lv[0].act, x, sol == 1 ? 1.0 : -0.5, Nx, Ny);
    // preconditioned CG
    k_dot<<<kDotBlocks, 256, 0, s>>>(w.f, w.f, m, S, kSBn2);
    k_residual_dot<<<kDotBlocks, 256, 0, s>>>(lv[0], w.f, x, r, S);
    double n2[2];  // |f|^2, |r|^2
    e = cudaMemcpyAsync(n2, scal + kSBn2, sizeof(n2), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return fail("dot", e);
    const double bn = std::sqrt(n2[0]);
    double rn = std::sqrt(n2[1]);
    int it = 0;
    if (bn == 0.0) {
      cudaMemsetAsync(x, 0, m * sizeof(double), s);
      rn = 0.0;
    } else {
      int rz = kSRz0;
      while (rn / bn > tols[sol] && it < in.maxit) {
        sv.vcycle();
        const int next = it == 0 ? kSRz0 : kSRz0 + kSRz1 - rz;
        k_dot<<<kDotBlocks, 256, 0, s>>>(r, z, m, S, next);
        k_direction<<<blocks_for(m), 256, 0, s>>>(w.d, z, m, S, next, rz, it == 0);
        rz = next;
        k_apply_dot<<<kDotBlocks, 256, 0, s>>>(lv[0], w.d, w.q, S);
        k_axpy_dot<<<kDotBlocks, 256, 0, s>>>(x, r, w.d, w.q, m, S, rz);
        ++it;
        double rn2 = 0;
        if ((e = read(kSRr, &rn2)) != cudaSuccess) return fail("dot", e);
        rn = std::sqrt(rn2);
      }
    }
    k_finish<<<blocks_for(m), 256, 0, s>>>(lv[0].act, x, w.b, w.phi[sol], m);
    if (rep) { rep->iters[sol] = it; rep->relres[sol] = bn == 0.0 ? 0.0 : rn / bn; }
  }
  const double bg = std::sqrt(gamma * gamma - 1), hden = 2 * kC * kMu0 * hr1;
  k_fields<<<blocks_for(m), 256, 0, s>>>(w.phi[0], w.phi[1], w.phi[2], Nx, Ny, gamma, hr0, hr1, bg, hden, in.Ex, in.Ey,
                                         in.Hx, in.Hy);
  e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return fail("initial-field kernels", e);
  if (rep) { rep->gamma = gamma; rep->levels = (int)lv.size(); }
  return kOk;
}

}  // namespace csrst
