"""How a push shares its bunch out over the grid (csrc/pushwork.cuh): every
particle is moved and deposited exactly once for bunches of one particle, of
one CTA round and around it, of two rounds per CTA, and large enough for a part
of the bunch to be handed out by a counter (8 rounds per CTA).  The check is
exact: the window current after a push is, integer for integer, the stand-alone
deposit of the moves the push made."""
import numpy as np
import pytest

from csrst_b200 import Simulation
from csrst_b200.pic import ShapeFunction
from csrst_b200.workloads import make_bunch, workload

pytestmark = pytest.mark.gpu


def loaded(order, n, fp32):
    cfg, spec = workload(f"small-{order}")
    spec.n = n
    s = Simulation(cfg, fp32=fp32, keep_old=True)
    s.load(*make_bunch(spec))
    return s


SIZES = [(0, 1), (1, 33), (2, 255), (1, 257), (2, 150_001), (1, 1_900_001)]


@pytest.mark.parametrize("order,n", SIZES)
def test_fp32_push_moves_every_particle_once(gpu_lib, order, n):
    s = loaded(order, n, True)
    s.step(2)
    info = s.info()
    sf = ShapeFunction(order)
    for comp in (0, 1):
        before = s.bunch32(0)
        s.push(comp)
        c1, b0, b1, _, _, q = s.bunch32(0)
        c0, a0, a1 = s.bunch32(1)
        assert np.array_equal(c0, before[0])  # every particle's move starts from its stored cell
        (P0, P1, L0, L1), _, _ = s.window()
        F = sf.flux32(comp, c0, a0, a1, c1, b0, b1, q, info["fixed_scale"], P0, P1, L0, L1)
        inv = 1.0 / (info["fixed_scale"] * info["dt"] * (info["hy"], info["hx"])[comp])
        assert comp == 1 or np.abs(F).max() > 0
        assert np.array_equal(s.window_field(4 + comp)[1:L1 + 1, 1:L0 + 1], F.astype(np.float64) * inv)
        s.update_e(comp)
        s.drift(-0.5 * info["dt"])
    s.close()


@pytest.mark.parametrize("order,n", SIZES)
def test_fp64_push_moves_every_particle_once(gpu_lib, order, n):
    """The FP64 push rounds each contribution by an FP64 add for bunches of
    1024 particles or more and by a conversion for smaller ones."""
    s = loaded(order, n, False)
    s.step(2)
    info = s.info()
    h, dt, scale = (info["hx"], info["hy"]), info["dt"], info["fixed_scale"]
    q = np.full(n, make_bunch(workload(f"small-{order}")[1])[4][0] * 4000 / n)  # equal charges, any order
    sf = ShapeFunction(order)
    for comp in (0, 1):
        s.push(comp)
        x, y, _, _ = s.particles()
        ox, oy = s.old_positions()
        (_, _, L0, L1), org, _ = s.window()
        J = sf.getCurrentDensityBase(comp, ox, oy, x, y, q, org, h, dt, 0, 0, L0, L1, scale)
        assert comp == 1 or np.abs(J).max() > 0
        assert np.array_equal(s.window_field(4 + comp)[1:L1 + 1, 1:L0 + 1], J)
        s.update_e(comp)
        s.drift(-0.5 * dt)
    s.close()
