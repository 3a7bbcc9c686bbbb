// Launch sequences of the wake surrogate: the network's forward pass, its
// backward pass and the refresh of its BF16 weight copies as one host call
// each, over the GEMM (gemm.cu) and the element-wise kernels (nn.cu).
//
// A forward pass is 22 launches and a training step about 90, of 3 to 30 us each at
// small batches, so a host that takes longer than that per launch is what
// bounds them: from Python, at 23 us a launch (argument structures, views,
// foreign calls), the wake of 37 bunches took 426 us and a 64-member training
// step 1677 us, where the same launches replayed as a graph took 141 and 972 us.  From
// here a launch costs its tensor maps and the launch itself: 163 and 1155 us with
// the kernels as they were then.  Nothing is kept between calls: every pointer comes in with the call.
#include <cuda_runtime.h>
#include <stdint.h>

#include <initializer_list>

#include "../../include/csrst.h"
#include "nn.h"

namespace {

constexpr int kBins = 256, kFeat = 64;
constexpr int kSplit = 256;  // K-columns per partial product of a weight gradient

// Output map index = z sb + (m / md) sm0 + (m % md) sm1 + (n / nd) sn0 + (n % nd) sn1.
struct Map {
  int md, nd;
  long long sm0, sm1, sn0, sn1;
};
Map rows_of(long long ld) { return {1, 1, ld, 0, 1, 0}; }
Map columns_of(long long ld) { return {1, 1, 1, 0, ld, 0}; }

csrst_gemm_epilogue epilogue(const Map &m, long long sb = 0) {
  csrst_gemm_epilogue e{};
  e.alpha = 1.0f;
  e.md = m.md;
  e.nd = m.nd;
  e.sb = sb;
  e.sm0 = m.sm0;
  e.sm1 = m.sm1;
  e.sn0 = m.sn0;
  e.sn1 = m.sn1;
  return e;
}

// The network with the offsets of its parameters in the flat buffer, and the
// first error of the sequence (later launches are then left out).
//
// A training step's weight gradients, bias sums and the transposes they need lie off
// the chain of activations and gradients, and most launches fill a part of the chip
// only, so they go to the side stream: aside(f) runs f's launches there after
// what the main stream holds so far, rejoin() makes the main stream wait for all
// of them.  A buffer that work aside reads is written again only after a rejoin, and
// the calls end with one, whatever happened in between.  (`part` and `cpart` are
// used aside, or after the last rejoin.)  64 members: 556 us a step, 630 on one
// stream.
struct Seq {
  const csrst_fno &f;
  int *err;
  void *s;
  int rc = CSRST_OK;
  long long w, m, R, B;
  cudaStream_t main, side;
  cudaEvent_t out = nullptr, back = nullptr;

  Seq(const csrst_fno &net, int *e, void *stream, bool two)
      : f(net), err(e), s(stream), w(net.width), m(net.modes), R((long long)net.batch * kBins), B(net.batch),
        main(static_cast<cudaStream_t>(stream)), side(two ? static_cast<cudaStream_t>(net.side) : nullptr) {
    if (side && (cudaEventCreateWithFlags(&out, cudaEventDisableTiming) != cudaSuccess ||
                 cudaEventCreateWithFlags(&back, cudaEventDisableTiming) != cudaSuccess))
      rc = CSRST_E_CUDA;
  }
  ~Seq() {
    if (out) cudaEventDestroy(out);
    if (back) cudaEventDestroy(back);
  }
  Seq(const Seq &) = delete;

  void cuda(cudaError_t e) { ck(e == cudaSuccess ? CSRST_OK : CSRST_E_CUDA); }
  template <class F>
  void aside(F launches) {
    if (!ok()) return;
    if (side) {
      cuda(cudaEventRecord(out, main));
      cuda(cudaStreamWaitEvent(side, out, 0));
      s = side;
    }
    launches();
    s = main;
  }
  void rejoin() {  // also after an error
    if (!side || !out || !back) return;
    cuda(cudaEventRecord(back, side));
    cuda(cudaStreamWaitEvent(main, back, 0));
  }

  void ck(int r) {
    if (rc == CSRST_OK) rc = r;
  }
  bool ok() const { return rc == CSRST_OK; }

  // offsets: P, p, then per layer W, b, Wr, Wi, then Q1, q1, Q2, q2
  long long oP() const { return 0; }
  long long op() const { return w * kFeat; }
  long long oW(int l) const { return op() + w + l * (w * w + w + 2 * m * w * w); }
  long long ob(int l) const { return oW(l) + w * w; }
  long long oWr(int l) const { return ob(l) + w; }
  long long oWi(int l) const { return oWr(l) + m * w * w; }
  long long oQ1() const { return oW(f.layers); }
  long long oq1() const { return oQ1() + w * w; }
  long long oQ2() const { return oq1() + w; }
  long long oq2() const { return oQ2() + f.nout * w; }
  const float *p32(long long o) const { return f.w + o; }
  float *g32(long long o) const { return f.g + o; }
  void *p16(long long o) const { return static_cast<uint16_t *>(f.w16) + o; }

  // M-row, N-column, K-deep product of row-major operands
  void gemm(const void *A, const void *Bm, long long M, long long N, long long K, const csrst_gemm_epilogue &ep) {
    if (ok()) ck(csrst_gemm_bf16(A, K, 0, Bm, K, 0, (int)M, (int)N, (int)K, 1, &ep, err, s));
  }
  void gemm_batched(const void *A, long long lda, long long sa, const void *Bm, long long ldb, long long sb,
                    long long M, long long N, long long K, long long batch, const csrst_gemm_epilogue &ep) {
    if (ok()) ck(csrst_gemm_bf16(A, lda, sa, Bm, ldb, sb, (int)M, (int)N, (int)K, (int)batch, &ep, err, s));
  }
  void transpose16(const void *src, void *dst, long long batch, long long rows, long long cols, long long ldd) {
    if (ok()) ck(csrst_nn_transpose_bf16(src, dst, (int)batch, (int)rows, (int)cols, (int)ldd, s));
  }
  void transpose32(const void *src, void *dst, long long rows, long long cols) {
    if (ok()) ck(csrst_nn_transpose_b32(src, dst, 1, (int)rows, (int)cols, (int)rows, s));
  }
  void cast(const float *x, void *y, long long n) {
    if (ok()) ck(csrst_nn_cast_bf16(x, y, n, s));
  }
  void colsum(const float *x, long long rows, long long cols, float *out) {
    if (ok()) ck(csrst_nn_colsum(x, (int)rows, (int)cols, f.cpart, out, 0, s));
  }
  // dy through the activation (pre NULL: none) as dx32, dH16 and dHt16
  void activation_bwd(const float *dy, const float *pre, float *dx32) {
    if (ok()) ck(csrst::nn_backward_rows(dy, pre, dx32, f.dH16, f.dHt16, (int)R, (int)w, s));
  }
  // grad[M][N] = At[M][R] Bt[N][R]^T as kSplit-column partial products summed in order
  void wgrad(const void *At, const void *Bt, long long M, long long N, float *out) {
    const long long S = R / kSplit;
    csrst_gemm_epilogue ep = epilogue(rows_of(N), M * N);
    ep.out32 = f.part;
    gemm_batched(At, R, kSplit, Bt, R, kSplit, M, N, kSplit, S, ep);
    colsum(f.part, S, M * N, out);
  }
};

// A call is refused before its first launch when a size is one that a kernel of
// the sequence does not take, or a buffer it reads or writes is missing or, where
// its kernels read it 16 bytes at a time or as a product's operand, not 16-byte aligned.
bool there(std::initializer_list<const void *> ps) {
  for (const void *p : ps)
    if (!p) return false;
  return true;
}
bool aligned(std::initializer_list<const void *> ps) {
  for (const void *p : ps)
    if (!p || ((uintptr_t)p & 15)) return false;
  return true;
}
bool aligned(const void *const *table, int n) {
  if (!table) return n <= 0;
  for (int k = 0; k < n; ++k)
    if (!aligned({table[k]})) return false;
  return true;
}

// The network itself (any sequence).
bool valid(const csrst_fno *f) {
  constexpr long long most = 0x7fffffffll;
  if (!f || f->width <= 0 || f->width % 64 || f->modes <= 0 || f->modes % 32 || f->layers < 1 || f->nout < 16 ||
      f->nout > 64 || f->nout % 16 || f->batch <= 0)
    return false;
  // (rows, columns and output counts go to the kernels as ints; the modes are a batch)
  return (long long)f->batch * kBins <= most && (long long)f->batch * f->width <= most &&
         (long long)f->width * f->width <= most && f->modes <= 65535 && f->w && aligned({f->w16});
}

bool can_forward(const csrst_fno *f) {
  if (!valid(f)) return false;
  const int L = f->layers;
  if (!aligned({f->F16, f->G16, f->U16, f->Zp16, f->A1_16}) || !f->Z16 || !aligned(f->Mk16, L) || !f->Mk16 || !f->V16 ||
      !aligned(f->V16, f->train ? L + 1 : 2))
    return false;
  if (!f->train) return true;
  // weight gradients are products over batch columns; R rows go to the transposes 32 to a block
  return f->batch % 64 == 0 && f->batch * (kBins / 32) <= 65535 && aligned({f->A1pre, f->A1t16}) && f->Vg16 && f->Ut16 &&
         aligned(f->Vg16, L + 1) && aligned(f->Ut16, L) && aligned((const void *const *)f->Hfull, L - 1);
}

bool can_backward(const csrst_fno *f) {
  return can_forward(f) && f->train && f->g && f->WT16 && f->MkT16 && aligned(f->WT16, f->layers) &&
         aligned(f->MkT16, f->layers) &&
         aligned({f->Q1T16, f->Q2T16, f->FT16, f->GT16, f->Xt16, f->dOut, f->dOut16, f->dOutT16, f->dA1, f->dH, f->dH16,
                  f->dHt16, f->dV, f->dVn, f->dZ16, f->dZt16, f->dS16}) &&
         there({f->out, f->dSk16, f->dMk, f->part, f->cpart, f->lpart, f->loss});
}

void forward(Seq &q, const void *X16, float *out) {
  const csrst_fno &f = q.f;
  const long long w = q.w, m = q.m, R = q.R, B = q.B;
  const bool tr = f.train != 0;
  csrst_gemm_epilogue ep = epilogue(rows_of(w));
  ep.bias = q.p32(q.op());
  ep.out16 = f.V16[0];
  q.gemm(X16, q.p16(q.oP()), R, w, kFeat, ep);  // lift
  for (int l = 0; l < f.layers; ++l) {
    const int i = tr ? l : l & 1, o = tr ? l + 1 : (l + 1) & 1;
    const bool act = l < f.layers - 1;
    if (tr) q.aside([&] { q.transpose16(f.V16[i], f.Vg16[i], 1, R, w, R); });
    // forward DFT over the bins, per member b: rows c of V[b] read MN-major -> U[k][b][2c + ri]
    ep = epilogue({1, 2, 2, 0, 2 * w * B, 1}, 2 * w);
    ep.out16 = f.U16;
    if (q.ok())
      q.ck(csrst_gemm_bf16_ex(f.V16[i], w, kBins * w, 1, f.F16, kBins, 0, (int)w, (int)(2 * m), kBins, (int)B, &ep,
                              q.err, q.s));
    if (tr) q.aside([&] { q.transpose16(f.U16, f.Ut16[l], m, B, 2 * w, B); });
    // mode mixing: per mode k, Z[b][2o + p] = sum U[b][2c + q] Mk[2o + p][2c + q]
    ep = epilogue(rows_of(2 * w), 2 * w * B);
    ep.out16 = f.Z16;
    q.gemm_batched(f.U16, 2 * w, 2 * w * B, f.Mk16[l], 2 * w, 4 * w * w, B, 2 * w, 2 * w, m, ep);
    q.transpose32(f.Z16, f.Zp16, m, B * w);  // Zp[(b, o)][2k + p]
    // per member: truncated inverse DFT and pointwise product in one accumulator, bias, activation
    ep = epilogue(columns_of(w), kBins * w);
    ep.bias_m = q.p32(q.ob(l));
    ep.pre = tr && act ? f.Hfull[l] : nullptr;
    ep.act = act ? 1 : 0;
    ep.out16 = f.V16[o];
    if (q.ok())
      q.ck(csrst_gemm_bf16_dual(f.Zp16, 2 * m, 2 * m * w, f.G16, 2 * m, 0, (int)(2 * m), q.p16(q.oW(l)), w, 0,
                                f.V16[i], w, kBins * w, (int)w, (int)w, kBins, (int)B, &ep, q.err, q.s));
    if (tr) q.rejoin();  // U16 is written again in the next layer
  }
  void *V = f.V16[tr ? f.layers : f.layers & 1];
  if (tr) q.aside([&] { q.transpose16(V, f.Vg16[f.layers], 1, R, w, R); });
  ep = epilogue(rows_of(w));
  ep.bias = q.p32(q.oq1());
  ep.act = 1;
  ep.out16 = f.A1_16;
  if (tr) {
    ep.pre = f.A1pre;
    ep.out16t = f.A1t16;
    ep.tmd = ep.tnd = 1;
    ep.tm0 = 1;
    ep.tn0 = R;
  }
  q.gemm(V, q.p16(q.oQ1()), R, w, w, ep);
  ep = epilogue(rows_of(f.nout));
  ep.bias = q.p32(q.oq2());
  ep.out32 = out;
  q.gemm(f.A1_16, q.p16(q.oQ2()), R, f.nout, w, ep);
  if (tr) q.rejoin();
}

void backward(Seq &q, const void *X16, const float *T, const float *Wt) {
  const csrst_fno &f = q.f;
  const long long w = q.w, m = q.m, R = q.R, B = q.B, nout = f.nout;
  csrst_gemm_epilogue ep;
  // loss and dLoss/dout into the first nout columns of a 64-column buffer
  if (q.ok())
    q.ck(csrst_nn_mse(f.out, T, Wt, R * nout, f.dOut, (int)nout, 64, 1, f.lpart, f.loss, q.s));
  if (q.ok()) q.ck(csrst::nn_backward_rows(f.dOut, nullptr, nullptr, f.dOut16, f.dOutT16, (int)R, 64, q.s));
  q.aside([&] {
    q.wgrad(f.dOutT16, f.A1t16, nout, w, q.g32(q.oQ2()));
    q.colsum(f.dOut, R, 64, q.g32(q.oq2()));  // q2 and the padding after it
    q.transpose16(X16, f.Xt16, 1, R, kFeat, R);
  });
  ep = epilogue(rows_of(w));
  ep.out32 = f.dA1;
  q.gemm(f.dOut16, f.Q2T16, R, w, 64, ep);
  q.activation_bwd(f.dA1, f.A1pre, f.dH);
  q.aside([&] {
    q.wgrad(f.dHt16, f.Vg16[f.layers], w, w, q.g32(q.oQ1()));
    q.colsum(f.dH, R, w, q.g32(q.oq1()));
  });
  ep.out32 = f.dV;
  q.gemm(f.dH16, f.Q1T16, R, w, w, ep);
  float *dV = f.dV, *dVn = f.dVn;
  for (int l = f.layers - 1; l >= 0; --l) {
    const bool act = l < f.layers - 1;
    const float *dH = act ? f.dH : dV;
    q.rejoin();  // dH, dH16, dHt16, dZt16 and the gradient before last are free
    q.activation_bwd(dV, act ? f.Hfull[l] : nullptr, act ? f.dH : nullptr);
    q.aside([&] {
      q.wgrad(f.dHt16, f.Vg16[l], w, w, q.g32(q.oW(l)));
      q.colsum(dH, R, w, q.g32(q.ob(l)));
    });
    // adjoint of the inverse DFT: dZ[k][(o, ri)][b] = sum_n dH[b][n][o] G[n][2k + ri] (rows (o, b) of dH^T)
    ep = epilogue({(int)B, 2, 2 * B, 1, 2 * w * B, B});
    ep.out16 = f.dZt16;
    q.gemm(f.dHt16, f.GT16, w * B, 2 * m, kBins, ep);
    q.transpose16(f.dZt16, f.dZ16, m, 2 * w, B, 2 * w);
    // mode-mixing weights: dMk[k] = dZ_k^T U_k, then back to (dWr, dWi)
    q.aside([&] {
      csrst_gemm_epilogue e = epilogue(rows_of(2 * w), 4 * w * w);
      e.out32 = f.dMk;
      q.gemm_batched(f.dZt16, B, 2 * w * B, f.Ut16[l], B, 2 * w * B, 2 * w, 2 * w, B, m, e);
      if (q.ok())
        q.ck(csrst_nn_spectral_unpack(f.dMk, (int)m, (int)w, q.g32(q.oWr(l)), q.g32(q.oWi(l)), q.s));
    });
    // dU_k = dZ_k Mk -> dSk[k][b][2c + q] -> dS[(b, c)][2k + q]
    ep = epilogue(rows_of(2 * w), 2 * w * B);
    ep.out16 = f.dSk16;
    q.gemm_batched(f.dZ16, 2 * w, 2 * w * B, f.MkT16[l], 2 * w, 4 * w * w, B, 2 * w, 2 * w, m, ep);
    q.transpose32(f.dSk16, f.dS16, m, B * w);
    // input gradient: pointwise part, then the adjoint of the forward DFT added on
    ep = epilogue(rows_of(w));
    ep.out32 = dVn;
    q.gemm(f.dH16, f.WT16[l], R, w, w, ep);
    ep = epilogue({(int)w, 1, kBins * w, 1, w, 0});
    ep.out32 = dVn;
    ep.accumulate = 1;
    q.gemm(f.dS16, f.FT16, B * w, kBins, 2 * m, ep);
    float *t = dV;
    dV = dVn;
    dVn = t;
  }
  q.rejoin();
  q.activation_bwd(dV, nullptr, nullptr);
  q.wgrad(f.dHt16, f.Xt16, w, kFeat, q.g32(q.oP()));
  q.colsum(dV, R, w, q.g32(q.op()));
}

}  // namespace

extern "C" {

int csrst_fno_forward(const csrst_fno *f, const void *X16, float *out, int *err, void *stream) {
  if (!can_forward(f) || !err || !aligned({X16}) || !out) return CSRST_E_ARG;
  Seq q(*f, err, stream, f->train);
  if (q.ok()) forward(q, X16, out);
  return q.rc;
}

int csrst_fno_backward(const csrst_fno *f, const void *X16, const float *T, const float *Wt, int *err, void *stream) {
  if (!can_backward(f) || !err || !aligned({X16}) || !T) return CSRST_E_ARG;
  Seq q(*f, err, stream, true);
  if (q.ok()) backward(q, X16, T, Wt);
  return q.rc;
}

int csrst_fno_refresh(const csrst_fno *f, long long n, void *stream) {
  int none = 0;
  if (!valid(f) || !there({f->WT16, f->Mk16, f->MkT16, f->Q1T16, f->Q2T16}) || !aligned(f->WT16, f->layers) ||
      !aligned(f->Mk16, f->layers) || !aligned(f->MkT16, f->layers))
    return CSRST_E_ARG;
  Seq q(*f, &none, stream, false);
  const long long w = q.w;
  if (n < q.oq2() + f->nout) return CSRST_E_ARG;  // w16 is read up to there
  q.cast(f->w, f->w16, n);
  for (int l = 0; l < f->layers; ++l) {
    q.transpose16(q.p16(q.oW(l)), f->WT16[l], 1, w, w, w);
    if (q.ok())
      q.ck(csrst_nn_spectral_pack(q.p32(q.oWr(l)), q.p32(q.oWi(l)), (int)q.m, (int)w, f->Mk16[l], f->MkT16[l],
                                  stream));
  }
  q.transpose16(q.p16(q.oQ1()), f->Q1T16, 1, w, w, w);
  q.transpose16(q.p16(q.oQ2()), f->Q2T16, 1, f->nout, w, 64);
  return q.rc;
}

}  // extern "C"
