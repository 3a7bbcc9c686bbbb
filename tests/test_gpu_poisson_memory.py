"""The initial-field solve's device memory: at most 220 bytes a mesh cell on a
mesh of 512 rows (the pool's 32 MiB steps aside), kept in the library's pool for the
next call and given back by csrst_release_memory, also to other allocations of the process."""
import pytest

pytestmark = pytest.mark.gpu


def test_solve_memory(gpu_lib):
    import torch
    from csrst_b200 import Simulation
    from csrst_b200.workloads import make_bunch, workload
    cfg, spec = workload("c1")
    s = Simulation(cfg)
    s.load(*make_bunch(spec))
    s.initial_fields()                       # (kernels are loaded by their first launch)

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    gpu_lib.csrst_release_memory()
    before = free()
    s.initial_fields()
    kept = before - free()
    step = 32 << 20
    assert 0 < kept <= -(-220 * cfg.Nx * cfg.Ny // step) * step
    assert gpu_lib.csrst_release_memory() == 0
    assert free() == before
