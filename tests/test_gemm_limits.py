"""The GEMM's tile count: launches whose tiles its 32-bit index cannot walk are
refused before any device call (host only: without a device what passes the check
fails at the next call)."""
import ctypes as C

import pytest

from conftest import gpu_available

E_ARG = -1


@pytest.mark.skipif(gpu_available(), reason="host addresses stand in for device buffers")
@pytest.mark.parametrize("M,N,batch,refused", [
    (128, 32, 2 ** 31 - 1, True), (1, 16, 2 ** 31 - 1, True), (128, 32, 2 ** 31 - 65536, False),
    (128, 32, 2 ** 31 - 65535, True), (2 ** 31 - 1, 128, 127, False), (2 ** 31 - 1, 128, 128, True),
    (129, 256, 2 ** 29, True), (128, 256, 2 ** 29, False)])
def test_tile_count(gpu_lib, M, N, batch, refused):
    from csrst_b200.tensor import Epilogue
    mem = (C.c_char * 64)()
    at = (C.addressof(mem) + 15) & ~15
    ep = Epilogue(alpha=1.0, md=1, nd=1, sn0=1)
    ep.out32 = at
    rc = gpu_lib.csrst_gemm_bf16_ex(at, 64, 0, 0, at, 64, 0, M, N, 64, batch, C.byref(ep), at, None)
    assert (rc == E_ARG) == refused, rc
