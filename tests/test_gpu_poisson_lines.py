"""The Poisson solver's y-line solves at the edges of their forms: one row per
lane (up to 32 rows), rows past the last lane's block, all of a lane's factors in
registers (up to 544 rows) and in batches above that, and columns so long that
fewer warps share an SM (kMaxLineLen rows).  As in test_gpu_poisson: GPU and
oracle solve the same matrix to a relative residual of 1e-13 and the fields
agree to 1e-8 of their maximum."""
import numpy as np
import pytest

from csrst_b200 import Simulation
from csrst_b200.workloads import BunchSpec, RunConfig, make_bunch

pytestmark = pytest.mark.gpu


def straight(Nx, Ny, h=20e-6):
    """A straight pipe that fills the mesh, and a bunch of one cell rms in it."""
    cfg = RunConfig(Nx=Nx, Ny=Ny, length_before=(Nx - 12) * h, length_after=10 * h, width=(Ny - 2) * h, phi_deg=0.0,
                    ekin_mev=50.0, bz=0.0, shape_order=1, dt=0.5 * h / 299792458.0)
    gamma = 1.0 + 50.0 / 0.511
    spec = BunchSpec(n=500, gamma=gamma, sigma_s=h, sigma_x=0.5 * h, energy_spread=1e-4, charge=-1e-9,
                     x0=0.5 * Nx * h, y0=0.5 * cfg.width, seed=5)
    return cfg, make_bunch(spec)


@pytest.mark.parametrize("Nx,Ny", [(61, 30), (40, 32), (96, 33), (130, 544), (70, 545), (33, 1500), (40, 4096)])
def test_line_solves(gpu_lib, oracle, Nx, Ny):
    cfg, bunch = straight(Nx, Ny)
    g = Simulation(cfg)
    g.load(*bunch)
    rep = g.initial_fields(1e-13, 1e-13, 500)
    assert all(rr <= 1e-13 and it <= 30 for it, rr in rep["solves"])
    d = cfg.dict()
    d["order"] = cfg.shape_order
    o = oracle.Sim(d)
    o.load(*bunch)
    o.initial_fields(1e-13, 1e-13, 20000)
    for a, b in zip(g.get_static(), o.get_static()):
        assert np.abs(b).max() > 0
        assert np.abs(a - b.reshape(a.shape)).max() <= 1e-8 * np.abs(b).max()
    g.close()
