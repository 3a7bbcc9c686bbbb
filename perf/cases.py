"""Performance cases: the work a user of this framework has it do, each one
pass through the public entry points (the Simulation / Ensemble classes and
the C ABI's host-buffer read-backs, and the wake surrogate's FNO and GEMM).

Kinds of case
  scan      a short run from a fresh start, as a parameter scan makes many of:
            zero static fields, bunch upload, a block of steps, everything read
            back (bunch, window, static mesh, beam moments);
  loop      a block of steps of a long run, with the beam moments every `stat`
            steps (the reference's statistics modulus), then the read-back at
            the block's end; the run goes on from pass to pass;
  poisson   the initial fields of a freshly loaded bunch (three solves);
  ensemble  a block of steps of many independent bunches stepped together,
            then every member's bunch and wake;
  predict   wake surrogate, forward: profiles -> wakes;
  train     one training step: loss, gradients, Adam update;
  layer     one network layer through the tensor-core GEMM: product, bias,
            GELU, BF16 activations and the FP32 pre-activation.

Results of FP32 mode are kept as FP32 (the mode's own precision; the C ABI
hands host arrays out as doubles), those of the FP64 path as FP64.
"""
import ctypes as C
import math

import numpy as np
import torch

from csrst_b200 import Simulation
from csrst_b200._lib import CsrstError, check, lib, ptr
from csrst_b200.pic import Ensemble
from csrst_b200.surrogate import FNO, NBINS, NFEAT, layout
from csrst_b200.tensor import gemm
from csrst_b200.workloads import BunchSpec, bend_config_fit, make_bunch, workload

NOUT = 32


def listed():
    return [
        # the smallest runs of the tests' 512 x 104 bend: launches and latency count
        dict(name="scan-small-fp64-cic", kind="scan", Nx=512, Ny=104, n=4000, order=0, fp32=False, steps=100),
        # odd sizes, the cubic shape, FP32 mode
        dict(name="scan-odd-fp32-cubic", kind="scan", Nx=1531, Ny=203, n=150_001, order=2, fp32=True, steps=100),
        # the 2048 x 512 CIC configuration, 2e5 particles
        dict(name="scan-c1-fp64-cic", kind="scan", Nx=2048, Ny=512, n=200_000, order=0, fp32=False, steps=200),
        # the headline configuration: 8192 x 1024, 4e6 TSC particles, both precisions
        dict(name="loop-c2-fp32-tsc", kind="loop", Nx=8192, Ny=1024, n=4_000_000, order=1, fp32=True, steps=160,
             stat=20),
        dict(name="loop-c2-fp64-tsc", kind="loop", Nx=8192, Ny=1024, n=4_000_000, order=1, fp32=False, steps=80,
             stat=20),
        # initial fields on the 2048 x 512 mesh
        dict(name="poisson-c1-fp64", kind="poisson", Nx=2048, Ny=512, n=200_000, order=0, fp32=False),
        # many small members (the bench's small ensemble, on meshes long enough to go on stepping)
        dict(name="ensemble-256-small-fp32", kind="ensemble", members=256, Nx=2048, Ny=104, n=4000, fp32=True,
             steps=40),
        # wake-data-sized members: 5e4 particles each, uneven meshes
        dict(name="ensemble-48-wake-fp32", kind="ensemble", members=48, Nx=1301, Ny=701, n=50_000, fp32=True,
             steps=40),
        # a handful of profiles, and a screen of many
        dict(name="predict-37", kind="predict", n=37),
        dict(name="predict-50000", kind="predict", n=50_000),
        # the training batch of the surrogate study
        dict(name="train-64", kind="train", batch=64),
        # one pointwise layer over an odd number of rows
        dict(name="layer-100003x128x128", kind="layer", M=100_003, N=128, K=128),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["scan", "scan", "loop", "poisson", "ensemble", "predict", "predict", "train", "layer"])
    fp32 = rng.random() < 0.5
    if kind == "scan":
        Nx = _log(rng, 500, 3000)
        return dict(kind=kind, Nx=Nx, Ny=_log(rng, 104, Nx // 3), n=_log(rng, 2000, 600_000),
                    order=rng.randrange(3), fp32=fp32, steps=rng.choice([50, 100, 150]))
    if kind == "loop":
        return dict(kind=kind, Nx=rng.randrange(6000, 8193), Ny=_log(rng, 256, 1024), n=_log(rng, 1_000_000, 4_000_000),
                    order=rng.randrange(3) if fp32 else rng.randrange(2), fp32=fp32, steps=40, stat=rng.choice([10, 20]))
    if kind == "poisson":
        Nx = _log(rng, 500, 2048)
        return dict(kind=kind, Nx=Nx, Ny=_log(rng, 104, Nx // 3), n=_log(rng, 4000, 200_000),
                    order=rng.randrange(2), fp32=fp32)
    if kind == "ensemble":
        m = _log(rng, 32, 256)  # meshes long enough for a few thousand steps
        return dict(kind=kind, members=m, Nx=rng.randrange(3600, 4200), Ny=_log(rng, 104, 300),
                    n=_log(rng, 800_000 // m, 2_500_000 // m), fp32=fp32, steps=rng.choice([10, 20]))
    if kind == "predict":
        return dict(kind=kind, n=_log(rng, 1, 50_000))
    if kind == "train":
        return dict(kind=kind, batch=64 * rng.choice([1, 1, 2, 3, 4]))
    return dict(kind=kind, M=_log(rng, 200, 300_000), N=16 * rng.randrange(2, 17), K=64 * rng.randrange(1, 9))


# ---- runs of the PIC loop -----------------------------------------------------

def _configs(case, h, order, R=1.0, sigma_cells=10.0):
    """Bends on the case's mesh with the bunch's rms sizes and start, from
    cells of h to coarser ones (the bunch keeps its size in cells); the 8192 x
    1024 and 2048 x 512 meshes are the named workloads."""
    for name in ("c1", "c2"):
        if (case["Nx"], case["Ny"]) == {"c1": (2048, 512), "c2": (8192, 1024)}[name]:
            cfg, spec = workload(name)
            cfg.shape_order = order
            yield cfg, spec.sigma_s, spec.sigma_x, spec.x0
    for k in range(48):
        hk = h * 1.25 ** (k % 24)
        s = sigma_cells * hk
        x0 = 40 * hk + 6 * s
        try:
            yield bend_config_fit(case["Nx"], case["Ny"], hk, R if k < 24 else 0.1 * R, 0.6 * (case["Ny"] - 2) * hk,
                                  1000.0, x0 + 8 * s, shape_order=order), s, 0.5 * s, x0
        except ValueError:
            continue


def _bunch(cfg, n, sigma_s, sigma_x, x0, seed):
    return make_bunch(BunchSpec(n=n, gamma=1000.0, sigma_s=sigma_s, sigma_x=sigma_x, energy_spread=1e-4,
                                charge=-1e-9, x0=x0, y0=0.5 * cfg.width, seed=seed))


def _pinned(shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=True)


def _keep(t, fp32):
    return t.float() if fp32 else t


def _open(case, fp32, **where):
    """The simulation of a case (empty) with its bunch's sizes: the first of
    _configs whose bend the reference's geometry rules accept."""
    for cfg, ss, sx, x0 in _configs(case, **where):
        try:
            return Simulation(cfg, fp32=fp32), cfg, ss, sx, x0
        except CsrstError:
            continue
    raise ValueError("no bend fits this mesh")


class _Run:
    """A loaded simulation and the pinned host buffers a program keeps for it."""

    def __init__(self, case, seed):
        self.case, self.fp32 = case, case["fp32"]
        small = case["n"] < 50_000
        # 3 cells per sigma for small bunches (the tests' 4000-particle one), 5 for larger
        self.sim, cfg, ss, sx, x0 = _open(case, self.fp32, h=20e-6 if small else 10e-6, order=case["order"],
                                          sigma_cells=3.0 if small else 5.0)
        self.bunch = [torch.from_numpy(a).pin_memory().numpy() for a in
                      _bunch(cfg, case["n"], ss, sx, x0, seed)]
        self.sim.load(*self.bunch)
        self.parts = _pinned((4, case["n"]))
        # room for the window of any bunch of this size (its extent is the draw's)
        h = self.sim.info()
        self.win = torch.zeros(6, int((13 * ss / h["hx"] + 16) * (13 * sx / h["hy"] + 16)), dtype=torch.float64).pin_memory()
        self.line = torch.zeros(2 * int(13 * ss / h["hx"] + 16), 7, dtype=torch.float64)
        self.mesh = None
        if case["kind"] != "loop" or not self.fp32:
            self.mesh = _pinned((4, cfg.Ny, cfg.Nx))
        if case["kind"] == "scan":
            self.zero = torch.zeros(cfg.Ny, cfg.Nx, dtype=torch.float64).pin_memory().numpy()

    def read(self):
        s, L = self.sim, lib()
        check(L.csrst_get_particles(s.h, *[ptr(a) for a in self.parts.numpy()]), s.h)
        for k in range(6):
            check(L.csrst_get_window_field(s.h, k, ptr(self.win[k].numpy())), s.h)
        out = dict(bunch=_keep(self.parts, self.fp32), window=_keep(self.win, self.fp32))
        out.update(self.read_mesh())
        return out

    def read_mesh(self):
        if self.mesh is None:
            return {}
        check(lib().csrst_get_static_fields(self.sim.h, *[ptr(a) for a in self.mesh.numpy()]), self.sim.h)
        return dict(mesh=_keep(self.mesh, self.fp32))


def _run_scan(st):
    s = st.sim
    s.set_static(st.zero, st.zero, st.zero, st.zero)
    s.load(*st.bunch)
    s.step(st.case["steps"])
    m = torch.from_numpy(s.moments())
    return dict(st.read(), moments=_keep(m, st.fp32))


def _run_loop(st):
    s, c = st.sim, st.case
    rows = []
    for _ in range(c["steps"] // c["stat"]):
        s.step(c["stat"])
        rows.append(s.moments())
    line = s.line_fields()
    st.line[:len(line)] = torch.from_numpy(line)
    return dict(st.read(), moments=_keep(torch.from_numpy(np.stack(rows)), st.fp32), line=_keep(st.line, st.fp32))


def _run_poisson(st):
    s = st.sim
    s.load(*st.bunch)
    s.initial_fields()
    return st.read_mesh()


class _Batch:
    def __init__(self, case, seed):
        self.case, self.fp32 = case, case["fp32"]
        small = case["n"] < 20_000
        self.sims = []
        self.wlen = []
        for k in range(case["members"]):  # uneven members: meshes, bend radii and bunch sizes
            c = dict(case, Nx=case["Nx"] + 37 * k % 64, Ny=case["Ny"] + 11 * k % 17)
            s, cfg, ss, sx, x0 = _open(c, self.fp32, h=10e-6, order=k % 2, R=0.5 + 0.37 * k % 4.5,
                                       sigma_cells=3.0 if small else 8.0)
            n = case["n"] + 29 * k % 101
            self.wlen.append(int(13 * ss / s.info()["hx"]) + 16)
            s.load(*_bunch(cfg, n, ss, sx, x0, seed * 1009 + k))
            self.sims.append(s)
        self.ens = Ensemble(self.sims)
        self.ens.sync()
        self.total = sum(s.n for s in self.sims)
        self.parts = _pinned(4 * self.total)
        self.wn = [s.window()[0][2] - 4 for s in self.sims]
        self.wake = torch.zeros(sum(self.wlen), dtype=torch.float64, device="cuda")
        self.meta = torch.zeros(4 * len(self.sims), dtype=torch.float64, device="cuda")


def _run_ensemble(st):
    st.ens.step(st.case["steps"])
    st.ens.sync()
    L, o, w = lib(), 0, 0
    flat = st.parts.numpy()
    for k, s in enumerate(st.sims):
        check(L.csrst_diag_wake_async(s.h, C.c_void_p(st.wake.data_ptr() + 8 * w), st.wn[k],
                                      C.c_void_p(st.meta.data_ptr() + 32 * k)), s.h)
        check(L.csrst_get_particles(s.h, *[ptr(flat[o + j * s.n:o + (j + 1) * s.n]) for j in range(4)]), s.h)
        o += 4 * s.n
        w += st.wlen[k]
    return dict(bunch=_keep(st.parts, st.fp32), wake=_keep(st.wake, st.fp32))


# ---- the wake surrogate ---------------------------------------------------------

def _params(seed, width=128):
    """Parameters of a trained network's sizes: uniform weights, small biases."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    d = {}
    for name, shape in layout(width):
        u = torch.rand(shape, generator=g, device="cuda") * 2 - 1
        if name.startswith(("Wr", "Wi")):
            u *= 0.5 / math.sqrt(width)
        elif len(shape) == 2:
            u *= 1.0 / math.sqrt(shape[1])
        else:
            u *= 0.0 if name == "pad" else 0.1
        d[name] = u
    return d


def _profiles(n, seed):
    """Input features: 6 smooth columns per bin (density, slope, position,
    run parameters), the rest padding zeros."""
    g = torch.Generator(device="cuda").manual_seed(seed + 1)
    X = torch.zeros(n, NBINS, NFEAT, dtype=torch.bfloat16, device="cuda")
    s = torch.linspace(-4, 4, NBINS, device="cuda")
    a, b, c = (torch.rand(n, 1, generator=g, device="cuda") for _ in range(3))
    z = (s - (a - 0.5)) / (0.5 + b)
    d = torch.exp(-0.5 * z * z) * (1 + 0.5 * c * torch.sin(6 * s))
    X[..., 0] = d.to(torch.bfloat16)
    X[..., 1] = (-z * d).to(torch.bfloat16)
    X[..., 2] = (s / 4).expand(n, NBINS).to(torch.bfloat16)
    for k in range(3, 6):
        X[..., k] = (torch.rand(n, 1, generator=g, device="cuda") * 2 - 1).to(torch.bfloat16)
    return X


def _targets(n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed + 2)
    return torch.randn(n, NBINS, NOUT, generator=g, device="cuda")


class _Net:
    def __init__(self, case, seed):
        self.net = FNO(params={k: v.cpu().numpy() for k, v in _params(seed).items()})
        n = case["n"] if case["kind"] == "predict" else case["batch"]
        self.X = _profiles(n, seed)
        if case["kind"] == "train":
            self.T = _targets(n, seed)


def _layer_inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    A = torch.randn(case["M"], case["K"], generator=g, device="cuda").to(torch.bfloat16)
    B = (torch.randn(case["N"], case["K"], generator=g, device="cuda") / math.sqrt(case["K"])).to(torch.bfloat16)
    bias = torch.randn(case["N"], generator=g, device="cuda") * 0.1
    return A, B, bias


class _Layer:
    def __init__(self, case, seed):
        self.A, self.B, self.bias = _layer_inputs(case, seed)
        M, N = case["M"], case["N"]
        self.pre = torch.empty(M, N, device="cuda")
        self.act = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("scan", "loop", "poisson"):
        st = _Run(case, seed)
    elif kind == "ensemble":
        st = _Batch(case, seed)
    elif kind in ("predict", "train"):
        st = _Net(case, seed)
    else:
        st = _Layer(case, seed)
    st.kind = kind
    st.case = case
    return st


def run(st):
    if st.kind == "scan":
        return _run_scan(st)
    if st.kind == "loop":
        return _run_loop(st)
    if st.kind == "poisson":
        return _run_poisson(st)
    if st.kind == "ensemble":
        return _run_ensemble(st)
    if st.kind == "predict":
        return st.net.predict(st.X)
    if st.kind == "train":
        loss = st.net.loss_and_grad(st.X, st.T)
        st.net.adam()
        return dict(loss=loss, grad=st.net.g, weights=st.net.w)
    c = st.case
    gemm(st.A, st.B, c["M"], c["N"], c["K"], bias=st.bias, act=1, pre=st.pre, out16=st.act)
    return dict(pre=st.pre, act=st.act)


def work(case):
    kind = case["kind"]
    if kind in ("scan", "loop", "poisson", "ensemble"):
        size = 4 if case["fp32"] else 8
        cells, n = case["Nx"] * case["Ny"], case["n"]
        planes = 4 * cells * size
        if kind == "poisson":  # the bunch read, four planes written
            return dict(bytes=5.0 * 8 * n + planes, flops=0.0)
        # per step: the four field planes read and written once and one byte per
        # cell, two pushes reading and writing positions and momenta and reading charges
        step = 2 * planes + cells + 2 * n * (9 * size)
        if kind == "ensemble":
            return dict(bytes=float(case["members"]) * (case["steps"] * step + 32 * n), flops=0.0)
        back = 32 * n + (8 * 4 * cells if kind == "scan" or not case["fp32"] else 0)
        up = 40 * n + 32 * cells if kind == "scan" else 0
        return dict(bytes=float(case["steps"]) * step + back + up, flops=0.0)
    if kind == "layer":
        M, N, K = case["M"], case["N"], case["K"]
        return dict(bytes=2.0 * (M * K + N * K) + 6.0 * M * N + 4 * N, flops=2.0 * M * N * K)
    n = case["n"] if kind == "predict" else case["batch"]
    w, m, layers = 128, 32, 4
    params = sum(int(np.prod(s)) for _, s in layout())
    per = 2.0 * NBINS * (NFEAT * w + w * w + w * NOUT)  # lift and head
    per += layers * (2.0 * NBINS * w * w + 2 * 2.0 * NBINS * w * 2 * m + 2.0 * m * (2 * w) ** 2)
    if kind == "predict":
        return dict(bytes=n * (2.0 * NBINS * NFEAT + 4.0 * NBINS * NOUT) + 2.0 * params, flops=n * per)
    return dict(bytes=n * (2.0 * NBINS * NFEAT + 4.0 * NBINS * NOUT) + 28.0 * params, flops=3 * n * per)


# ---- the same results in 64 bits, by plain torch ---------------------------------

def _forward64(p, X):
    w, m, layers = 128, 32, 4
    V = X @ p["P"].T + p["p"]
    for l in range(layers):
        U = torch.fft.rfft(V, dim=1)[:, :m]
        Z = torch.einsum("bkc,kco->bko", U, torch.complex(p["Wr%d" % l], p["Wi%d" % l]))
        S = torch.fft.irfft(torch.nn.functional.pad(Z, (0, 0, 0, NBINS // 2 + 1 - m)), n=NBINS, dim=1)
        H = V @ p["W%d" % l].T + p["b%d" % l] + S
        V = torch.nn.functional.gelu(H) if l < layers - 1 else H
    A = torch.nn.functional.gelu(V @ p["Q1"].T + p["q1"])
    return A @ p["Q2"].T + p["q2"]


def exact(case, seed):
    kind = case["kind"]
    if kind == "layer":
        A, B, bias = _layer_inputs(case, seed)
        pre = A.double() @ B.double().T + bias.double()
        return dict(pre=pre, act=torch.nn.functional.gelu(pre))
    if kind == "predict":
        p = {k: v.double() for k, v in _params(seed).items()}
        X = _profiles(case["n"], seed)
        return torch.cat([_forward64(p, X[a:a + 2000].double()) for a in range(0, case["n"], 2000)])
    if kind == "train":
        p = {k: v.double().requires_grad_() for k, v in _params(seed).items()}
        X, T = _profiles(case["batch"], seed).double(), _targets(case["batch"], seed).double()
        loss = ((_forward64(p, X) - T) ** 2).mean()
        loss.backward()
        g = torch.cat([(torch.zeros_like(v) if v.grad is None else v.grad).reshape(-1) for v in p.values()])
        return dict(loss=loss.detach().reshape(1), grad=g, weights=None)
    return None
