"""Wake surrogate: a 1D Fourier neural operator (Li et al. 2021) that maps a
bunch's line-charge profile on 256 bins plus the bend parameters (gamma, R,
sigma_s, pipe width) to the longitudinal wake E_s on the same bins at 32
stations along the bend.

Training and inference run on the GPU through the library alone: every product
is the BF16 tensor-core GEMM (tcgen05, FP32 accumulation, csrst_gemm_bf16) and
every other step an element-wise or reduction kernel of nn.cu; torch holds
the device memory and supplies the stream.

Network (width w = 128, 32 Fourier modes, 4 layers, 32 outputs per bin):
  V0      = X P^T + p                          X: 64 features per bin (6 used)
  H_l     = V_l W_l^T + b_l + irfft(rfft(V_l)[:32] . (Wr_l + i Wi_l))
  V_{l+1} = gelu(H_l) (l < 3), V_4 = H_3
  out     = gelu(V_4 Q1^T + q1) Q2^T + q2
The spectral product is three GEMMs per layer: the forward DFT as a product
with a [64 x 256] matrix of cosines and sines (per member, its channels as
rows, reading V's rows of bins as an MN-major operand; output written
mode-major), the mode mixing as a batch of 32 real [2w x 2w] block matrices
(one per mode: [[Wr, -Wi], [Wi, Wr]] interleaved), and, per member, the
truncated inverse DFT with the layer's pointwise product as a second K
segment of the same accumulator, and bias, activation and the BF16 copy
fused into its epilogue.

Activations are BF16 between products (FP32 accumulation inside them); the
loss, gradients of biases and the Adam state are FP32.  Reductions are in a
fixed order, so a training run repeats bit for bit.
"""
import ctypes as C
import math
import threading

import numpy as np
import torch

from ._lib import CsrstError, lib
from .tensor import _err, check_errors

NBINS, NFEAT = 256, 64
KSPLIT = 256          # K-columns per partial product of a weight gradient


def layout(width=128, modes=32, layers=4, nout=32):
    """(name, shape) of every parameter in the order of the flat FP32 buffer."""
    out = [("P", (width, NFEAT)), ("p", (width,))]
    for l in range(layers):
        out += [("W%d" % l, (width, width)), ("b%d" % l, (width,)), ("Wr%d" % l, (modes, width, width)),
                ("Wi%d" % l, (modes, width, width))]
    out += [("Q1", (width, width)), ("q1", (width,)), ("Q2", (nout, width)), ("q2", (nout,)), ("pad", (64 - nout,))]
    return out


def init_params(seed=0, width=128, modes=32, layers=4, nout=32):
    """Uniform initialisation: pointwise weights U(+-1/sqrt(fan_in)), spectral
    weights U(+-0.5/sqrt(width)), biases zero (numpy FP64, by name)."""
    g = np.random.Generator(np.random.Philox(seed))
    d = {}
    for name, shape in layout(width, modes, layers, nout):
        if name.startswith(("Wr", "Wi")):
            d[name] = g.uniform(-0.5, 0.5, shape) / np.sqrt(width)
        elif len(shape) == 2:
            d[name] = g.uniform(-1.0, 1.0, shape) / np.sqrt(shape[1])
        else:
            d[name] = np.zeros(shape)
    return d


def _p(t):
    return None if t is None else C.c_void_p(t.data_ptr())


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def _ck(rc, what):
    if rc:
        raise CsrstError(rc, what)


class _Net(C.Structure):
    """csrst_fno (include/csrst.h): one network's device pointers and one batch size's buffers."""
    _fields_ = ([(k, C.c_int) for k in ("width", "modes", "layers", "nout", "batch", "train")] +
                [(k, C.c_void_p) for k in (
                    "w", "g", "w16", "WT16", "Mk16", "MkT16", "Q1T16", "Q2T16", "F16", "FT16", "G16", "GT16", "V16",
                    "U16", "Z16", "Zp16", "A1_16", "out", "Vg16", "Ut16", "Hfull", "A1pre", "A1t16", "Xt16", "dOut",
                    "dOut16", "dOutT16", "dA1", "dH", "dH16", "dHt16", "dV", "dVn", "dZ16", "dZt16", "dSk16", "dS16",
                    "dMk", "part", "cpart", "lpart", "loss", "side")])


def _ptrs(ts):
    return (C.c_void_p * max(len(ts), 1))(*[t.data_ptr() for t in ts])


class _Buffers:
    """Activations and scratch of one batch size, or of any up to it in
    inference, where a pass uses the front of each (training keeps every
    layer's input for the backward pass; inference ping-pongs two).

    Layouts (b member, n bin, c channel, k mode, ri real/imaginary):
      V16  [b][n][c]      rows of the pointwise products; per member, the forward
                          DFT's operand read MN-major (its 256 bins are the K rows)
      Vg16 [c][b][n]      every bin of a channel in one row: weight gradients
      U16  [k][b][2c+ri]  spectra, the mode mixing's operand
      Z16  [k][b][2o+p]   mixed spectra; Zp16 [b][o][2k+p] the inverse DFT's operand
    The pointwise product rides in the inverse DFT's accumulator as a second
    K segment, so the layer's FP32 pre-activation sum never goes to memory
    (it is kept only for training, for the activation's backward pass).
    Every product writes its large outputs in a layout its epilogue can store
    contiguously; the others come from transposes."""

    def __init__(self, net, B, train):
        w, m, L, dev = net.width, net.modes, net.layers, net.device
        R = B * NBINS
        bf, f32 = dict(dtype=torch.bfloat16, device=dev), dict(dtype=torch.float32, device=dev)
        nkeep = L + 1 if train else 2
        self.V16 = [torch.empty(R, w, **bf) for _ in range(nkeep)]
        self.U16 = torch.empty(m, B, 2 * w, **bf)
        self.Z16 = torch.empty(m, B, 2 * w, **bf)
        self.Zp16 = torch.empty(B * w, 2 * m, **bf)
        self.A1_16 = torch.empty(R, w, **bf)
        self.train = train
        self.lock = threading.Lock()  # held while a pass's launches go out
        if not train:
            return
        self.out = torch.empty(R, net.nout, **f32)
        self.Vg16 = [torch.empty(w, R, **bf) for _ in range(L + 1)]
        self.Ut16 = [torch.empty(m, 2 * w, B, **bf) for _ in range(L)]
        self.Hfull = [torch.empty(R, w, **f32) for _ in range(L - 1)]
        self.A1pre = torch.empty(R, w, **f32)
        self.A1t16 = torch.empty(w, R, **bf)
        self.Xt16 = torch.empty(NFEAT, R, **bf)
        self.dOut = torch.zeros(R, 64, **f32)
        self.dOut16 = torch.empty(R, 64, **bf)
        self.dOutT16 = torch.empty(64, R, **bf)
        self.dA1 = torch.empty(R, w, **f32)
        self.dH = torch.empty(R, w, **f32)
        self.dH16 = torch.empty(R, w, **bf)
        self.dHt16 = torch.empty(w, R, **bf)
        self.dV = torch.empty(R, w, **f32)
        self.dVn = torch.empty(R, w, **f32)
        self.dZ16 = torch.empty(m, B, 2 * w, **bf)
        self.dZt16 = torch.empty(m, 2 * w, B, **bf)
        self.dSk16 = torch.empty(m, B, 2 * w, **bf)
        self.dS16 = torch.empty(B * w, 2 * m, **bf)
        self.dMk = torch.empty(m, 2 * w, 2 * w, **f32)
        self.part = torch.empty(max(R // KSPLIT, 1) * max(w * w, w * NFEAT), **f32)
        # column-sum scratch: ceil(rows / 256) * cols floats for every column sum of the backward pass
        self.cpart = torch.empty(max(B * max(w, 64), ((R // KSPLIT + 255) // 256) * w * max(w, NFEAT)), **f32)
        self.lpart = torch.empty(256, dtype=torch.float64, device=dev)
        self.loss = torch.zeros(1, dtype=torch.float64, device=dev)

    # the training step's second stream, joined to the caller's within each call; made by
    # the first step, so that a network can be unpickled where there is no GPU
    side = None

    def side_stream(self):
        if self.side is None:
            self.side = torch.cuda.Stream(self.loss.device)
        return self.side.cuda_stream

    def __getstate__(self):   # a copy gets a side stream and a lock of its own
        return {k: v for k, v in vars(self).items() if k not in ("side", "lock")}

    def __setstate__(self, d):
        vars(self).update(d, lock=threading.Lock())


class FNO:
    """The surrogate network on one GPU.  Parameters live in one flat FP32
    buffer (order: layout()) with its gradient and Adam moments beside it;
    BF16 copies of the weights (and transposed and block-packed copies) are
    refreshed after every update."""

    def __init__(self, width=128, modes=32, layers=4, nout=32, seed=0, params=None, device="cuda"):
        if width % 64 or modes % 32 or nout % 16 or not 16 <= nout <= 64 or layers < 1:
            raise ValueError("width must be a multiple of 64, modes of 32, nout of 16 (<= 64)")
        self.width, self.modes, self.layers, self.nout = width, modes, layers, nout
        self.device = torch.device(device)
        self.lay = layout(width, modes, layers, nout)
        sizes = [int(np.prod(s)) for _, s in self.lay]
        self.n = sum(sizes)
        f32 = dict(dtype=torch.float32, device=self.device)
        self.w = torch.zeros(self.n, **f32)
        self.g = torch.zeros(self.n, **f32)
        self.m1 = torch.zeros(self.n, **f32)
        self.m2 = torch.zeros(self.n, **f32)
        self.w16 = torch.zeros(self.n, dtype=torch.bfloat16, device=self.device)
        self.off = {}
        o = 0
        for (name, shape), sz in zip(self.lay, sizes):
            self.off[name] = (o, shape)
            o += sz
        self.set_params(params if params is not None else init_params(seed, width, modes, layers, nout))
        bf = dict(dtype=torch.bfloat16, device=self.device)
        self.WT16 = [torch.empty(width, width, **bf) for _ in range(layers)]
        self.Mk16 = [torch.empty(modes, 2 * width, 2 * width, **bf) for _ in range(layers)]
        self.MkT16 = [torch.empty(modes, 2 * width, 2 * width, **bf) for _ in range(layers)]
        self.Q1T16 = torch.empty(width, width, **bf)
        self.Q2T16 = torch.zeros(width, 64, **bf)
        F, G = _dft_matrices(modes)
        self.F16 = torch.from_numpy(F).to(**bf)
        self.FT16 = torch.from_numpy(np.ascontiguousarray(F.T)).to(**bf)
        self.G16 = torch.from_numpy(G).to(**bf)
        self.GT16 = torch.from_numpy(np.ascontiguousarray(G.T)).to(**bf)
        self.t = torch.zeros(1, dtype=torch.int32, device=self.device)
        self.coef = torch.zeros(3, **f32)
        self._bufs = {}
        self.refresh()

    # ---- parameters ----
    def view(self, name, buf=None):
        o, shape = self.off[name]
        return (self.w if buf is None else buf)[o:o + int(np.prod(shape))].view(shape)

    def set_params(self, d):
        flat = np.concatenate([np.asarray(d.get(n, np.zeros(s)), dtype=np.float32).reshape(-1) for n, s in self.lay])
        self.w.copy_(torch.from_numpy(flat))
        if hasattr(self, "WT16"):
            self.refresh()

    def params(self):
        flat = self.w.cpu().numpy().astype(np.float64)
        return {n: flat[self.off[n][0]:self.off[n][0] + int(np.prod(s))].reshape(s) for n, s in self.lay}

    def grads(self):
        flat = self.g.cpu().numpy().astype(np.float64)
        return {n: flat[self.off[n][0]:self.off[n][0] + int(np.prod(s))].reshape(s) for n, s in self.lay}

    def refresh(self):
        """BF16 copies of the weights: one cast of the flat buffer, then the
        transposed pointwise weights and the block-packed spectral weights."""
        _ck(lib().csrst_fno_refresh(C.byref(self._net()), self.n, _stream()), "refresh")

    def _net(self, bf=None, B=1):
        """The C structure of this network and of the buffers of a batch of B members, for one call."""
        n = _Net(self.width, self.modes, self.layers, self.nout, B, 1 if bf is not None and bf.train else 0)
        for k in ("w", "g", "w16", "Q1T16", "Q2T16", "F16", "FT16", "G16", "GT16"):
            setattr(n, k, getattr(self, k).data_ptr())
        n.keep = [_ptrs(v) for v in (self.WT16, self.Mk16, self.MkT16)]
        n.WT16, n.Mk16, n.MkT16 = map(C.addressof, n.keep)
        if bf is not None:
            for k, v in vars(bf).items():
                if isinstance(v, list):
                    v = _ptrs(v)
                    n.keep.append(v)
                    setattr(n, k, C.addressof(v))
                elif torch.is_tensor(v):
                    setattr(n, k, v.data_ptr())
            if bf.train:
                n.side = bf.side_stream()
        return n

    def _buf(self, B, train):
        """Buffers for a batch of B members.  Inference has sets per stream, so that passes on
        two streams run beside each other, each for the next power of two of members (above
        4096 the next multiple of it), so that any number of different batch sizes keeps a few
        sets (they stay: a captured pass may use them).  A training pass writes the network's
        gradient, so two of them are not for running at a time anyway: one set per batch size."""
        size = B if train else 1 << (B - 1).bit_length() if B <= 4096 else -(-B // 4096) * 4096
        key = (B, True) if train else (size, False, _stream().value)
        if key not in self._bufs:
            self._bufs.setdefault(key, _Buffers(self, size, train))
        return self._bufs[key]

    # ---- forward ----
    def _forward(self, net, X16, out):
        assert X16.dtype == torch.bfloat16
        _ck(lib().csrst_fno_forward(C.byref(net), _p(X16), _p(out), _p(_err(self.device)), _stream()), "forward")

    def predict(self, X, chunk=4096):
        """X: [N][256][64] BF16 (device) -> wake [N][256][nout] FP32 (device), in chunks of members."""
        N = X.shape[0]
        out = torch.empty(N, NBINS, self.nout, dtype=torch.float32, device=self.device)
        for a in range(0, N, chunk):
            B = min(chunk, N - a)
            bf = self._buf(B, False)
            with bf.lock:  # threads on one stream: one pass's launches after another's
                self._forward(self._net(bf, B), X[a:a + B].reshape(B * NBINS, NFEAT), out[a:a + B])
        return out

    # ---- backward ----
    def loss_and_grad(self, X, T, weight=None):
        """X: [B][256][64] BF16, T: [B][256][nout] FP32 (device, B a multiple
        of 64), weight: optional FP32 per-output weights of the squared error
        (0 leaves an output out).  Fills the gradient buffer; returns the loss
        as a device scalar."""
        B = X.shape[0]
        if B % 64:
            raise ValueError("training batches must be a multiple of 64 members")
        bf = self._buf(B, True)
        X16 = X.reshape(B * NBINS, NFEAT)
        T = T.reshape(B * NBINS, self.nout)
        Wt = None if weight is None else weight.reshape(B * NBINS, self.nout)
        net = self._net(bf, B)
        self._forward(net, X16, bf.out)
        _ck(lib().csrst_fno_backward(C.byref(net), _p(X16), _p(T), _p(Wt), _p(_err(self.device)), _stream()),
            "backward")
        return bf.loss

    def adam(self, lr0=1e-3, lr_min=1e-5, total=10000, b1=0.9, b2=0.999, eps=1e-8):
        s = _stream()
        _ck(lib().csrst_nn_adam_tick(_p(self.t), _p(self.coef), lr0, lr_min, total, b1, b2, s), "adam")
        _ck(lib().csrst_nn_adam(_p(self.w), _p(self.g), _p(self.m1), _p(self.m2), self.n, _p(self.coef), b1, b2, eps,
                                s), "adam")
        self.refresh()

    def check(self):
        check_errors(self.device)


def _dft_matrices(modes, n=NBINS):
    """F[2k + ri][t] (forward DFT, real and imaginary rows) and G[t][2k + ri]
    (the real inverse truncated to `modes` modes: weight 1/n for k = 0, 2/n
    for the others)."""
    k = np.arange(modes)[:, None]
    t = np.arange(n)[None, :]
    th = 2.0 * np.pi * k * t / n
    F = np.empty((2 * modes, n), dtype=np.float32)
    F[0::2], F[1::2] = np.cos(th), -np.sin(th)
    wk = np.where(np.arange(modes) == 0, 1.0 / n, 2.0 / n)[:, None]
    G = np.empty((2 * modes, n), dtype=np.float32)
    G[0::2], G[1::2] = wk * np.cos(th), -wk * np.sin(th)
    return F, np.ascontiguousarray(G.T)
