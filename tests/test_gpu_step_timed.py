"""csrst_step_timed: the groups' times are of stretches of one stream that do not
overlap (so they add up to at most the step, with a move that takes time), and the
step is bit for bit csrst_step's, in any order with it."""
import numpy as np
import pytest

from csrst_b200 import Simulation
from csrst_b200.workloads import make_bunch, workload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,fp32", [("c1", False), ("c1", True), ("small-2", True)])
def test_groups_of_a_timed_step(gpu_lib, name, fp32):
    cfg, spec = workload(name)
    bunch = make_bunch(spec)
    a, b = Simulation(cfg, fp32=fp32), Simulation(cfg, fp32=fp32)
    a.load(*bunch)
    b.load(*bunch)
    a.step(12)
    b.step(3)
    rows = []
    for _ in range(4):
        rows.append(b.step_timed())
    b.step(1)
    rows.append(b.step_timed())
    b.step(3)
    # event times come in half microseconds: two per group, eight groups' ends
    for t in rows:
        assert t["push"] > 0 and t["fields"] > 0
        assert t["push"] + t["fields"] + t["move"] <= t["total"] + 0.004, t
    assert np.median([t["move"] for t in rows]) > 0.003, rows   # three launches, no empty stretch
    for x, y in zip(a.particles() + [a.window_field(k) for k in range(6)] + a.get_static(),
                    b.particles() + [b.window_field(k) for k in range(6)] + b.get_static()):
        assert np.array_equal(x, y)
    assert np.array_equal(a.window()[0], b.window()[0])
