"""FP32 mode's deposit at offsets where o + 0.5 rounds up in FP32 (0.5 - 2^-25,
and its neighbours and the other borders of a base index) on the CPU: the
compact form is taken for exactly the moves whose base indices allow it, gives the general form's integers,
and continuity holds (tests/cpp/flux32_host.cpp, tests/cpp/flux32_rule_host.cpp)."""
import ctypes as C
import itertools
import subprocess
from fractions import Fraction
from math import floor

import numpy as np
import pytest

from test_flux32 import ROOT, flux, host  # noqa: F401

HALF = np.float32(0.5)
BORDERS = [np.float32(0.0), np.nextafter(HALF, np.float32(0)), HALF, np.nextafter(HALF, np.float32(1)),
           np.nextafter(np.float32(1), np.float32(0))]
INSIDE = [np.float32(0.26), np.float32(0.51), np.float32(0.74)]


def border_moves():
    """Every move between two offsets of which one lies at a border, along each
    axis and in both directions, the ends in the same or the next cell."""
    pts = [(o, c) for o in BORDERS + INSIDE for c in (0, 1)]
    ends = [(p, q) for p, q in itertools.product(pts, pts)
            if (p[0] in BORDERS or q[0] in BORDERS) and abs(float(q[0]) + q[1] - float(p[0]) - p[1]) <= 1.0]
    rows = []
    for (a, ca), (b, cb) in ends:
        # along y with a step in x, and along x with a step in y (a start offset may lie
        # outside the start cell: the start's cell is 20, its offset a + ca)
        if ca == 0:
            rows.append((0.3, a, 0, cb, 0.35, b))
            rows.append((a, 0.3, cb, 0, b, 0.35))
            rows.append((a, b if cb == 0 else a, cb, 0, b, a))
    r = np.array(rows, dtype=np.float64)
    n = len(r)
    ci = np.full(n, 20)
    f32 = lambda k: r[:, k].astype(np.float32)
    dc0, dc1 = r[:, 2].astype(int), r[:, 3].astype(int)
    pack = lambda i, j: (i | (j << 16)).astype(np.int32)
    q = np.full(n, -1.5e-15, dtype=np.float32)
    return (pack(ci, ci), f32(0), f32(1), pack(ci + dc0, ci + dc1), f32(4), f32(5), q,
            (ci, ci, ci + dc0, ci + dc1))


def one(mv, k):
    """Move k of a set, alone."""
    return tuple(x[k:k + 1] for x in mv[:7]) + (tuple(x[k:k + 1] for x in mv[7]),)


@pytest.mark.parametrize("order", [0, 1, 2])
def test_border_moves(host, order):  # noqa: F811
    mv = border_moves()
    scale = 2.0 ** 49 / 1.5e-15          # |K| below the compact form's 2^50
    for k in range(len(mv[0])):
        m = one(mv, k)
        f = []
        for comp in (0, 1):
            a, rho = flux(host, order, comp, m, scale, drho=True, fast=True)
            b, _ = flux(host, order, comp, m, scale, fast=False)
            assert np.array_equal(a, b), (order, comp, k, [x[0] for x in m[:6]])
            f.append(a)
        res = rho[1:, 1:] + (f[0][1:, 1:] - f[0][1:, :-1]) + (f[1][1:, 1:] - f[1][:-1, 1:])
        assert (res == 0).all(), (order, k)


@pytest.mark.parametrize("order", [0, 1, 2])
def test_rule_of_the_compact_form(tmp_path, order):
    """compact_form() against base indices in exact arithmetic."""
    so = tmp_path / "rule.so"
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-shared", "-fPIC",
                    str(ROOT / "tests/cpp/flux32_rule_host.cpp"), "-o", str(so)], check=True)
    L = C.CDLL(str(so))
    L.compact_form_host.argtypes = [C.c_int, C.c_float, C.c_float, C.c_int, C.c_int, C.c_float, C.c_float, C.c_double]
    base = lambda o: floor(Fraction(float(o)) + (Fraction(1, 2) if order == 1 else 0))
    c0, a0, a1, c1, b0, b1, _, (ci, cj, ni, nj) = border_moves()
    taken = 0
    for k in range(len(c0)):
        d0, d1 = int(ni[k] - ci[k]), int(nj[k] - cj[k])
        want = d0 + base(b0[k]) - base(a0[k]) in (0, 1) and d1 + base(b1[k]) == base(a1[k])
        for K, ok in ((2.0 ** 49, want), (-2.0 ** 49, want), (2.0 ** 50, False), (float("nan"), False)):
            assert bool(L.compact_form_host(order, a0[k], a1[k], d0, d1, b0[k], b1[k], K)) == ok, (k, K)
        taken += want
    assert 0 < taken < len(c0)
