"""FP32 mode's push deposits particles that start at y offsets next to the border
of a base index (0.5 - 2^-25, which + 0.5 rounds up in FP32) as the stand-alone
deposit does, bit for bit, whatever the other particles of their warp are."""
import numpy as np
import pytest

from csrst_b200 import ShapeFunction, Simulation
from csrst_b200.workloads import make_bunch, workload

pytestmark = pytest.mark.gpu

BELOW = float(np.nextafter(np.float32(0.5), np.float32(0)))


@pytest.mark.parametrize("order", [0, 1, 2])
@pytest.mark.parametrize("offsets", [(BELOW,), (BELOW, 0.5, 0.3, 0.7)])
def test_push_at_base_index_borders(gpu_lib, order, offsets):
    cfg, spec = workload(f"small-{order}")
    x, y, px, py, q = make_bunch(spec)
    s = Simulation(cfg, fp32=True, keep_old=True)
    s.load(x, y, px, py, q)
    info = s.info()
    _, org, _ = s.window()
    k = np.floor((y - org[1]) / info["hy"])
    y = org[1] + (k + np.resize(offsets, len(y))) * info["hy"]
    s.load(x, y, px, np.abs(py) + 1e-2 * px, q)          # every particle moves up by some 5e-3 cells
    sf = ShapeFunction(order)
    for comp in (0, 1):
        before = s.bunch32(0)
        s.push(comp)
        c1, b0, b1, _, _, q32 = s.bunch32(0)
        c0, a0, a1 = s.bunch32(1)
        if comp == 0:
            assert np.isin(np.float32(BELOW), before[2]) and np.array_equal(a1, before[2])
        (P0, P1, L0, L1), _, _ = s.window()
        F = sf.flux32(comp, c0, a0, a1, c1, b0, b1, q32, s.info()["fixed_scale"], P0, P1, L0, L1)
        inv = 1.0 / (s.info()["fixed_scale"] * info["dt"] * (info["hy"], info["hx"])[comp])
        assert np.abs(F).max() > 0
        assert np.array_equal(s.window_field(4 + comp)[1:L1 + 1, 1:L0 + 1], F.astype(np.float64) * inv)
        s.load(x, y, px, np.abs(py) + 1e-2 * px, q)
    s.close()
