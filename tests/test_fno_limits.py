"""Networks and buffers that the surrogate's kernels cannot take are refused
with CSRST_E_ARG at the C boundary, before any launch.  For hosts without a GPU
only: the addresses are the host's, and a structure that passes gets as far as the
launch, which fails for want of a device."""
import ctypes as C

import pytest

from conftest import gpu_available

pytestmark = pytest.mark.skipif(gpu_available(), reason="host addresses stand in for device buffers")

E_ARG = -1
TABLES = {"WT16": 3, "Mk16": 3, "MkT16": 3, "V16": 4, "Vg16": 4, "Ut16": 3, "Hfull": 2}
SCALARS = ("width", "modes", "layers", "nout", "batch", "train")


@pytest.fixture
def net(gpu_lib):
    """A training structure of three layers whose buffers all lie at one 16-byte aligned address."""
    from csrst_b200.surrogate import _Net
    mem = (C.c_char * 64)()
    at = (C.addressof(mem) + 15) & ~15
    f = _Net(128, 32, 3, 32, 64, 1)
    keep = [mem]
    for name, kind in _Net._fields_:
        if name in TABLES:
            t = (C.c_void_p * TABLES[name])(*[at] * TABLES[name])
            keep.append(t)
            setattr(f, name, C.addressof(t))
        elif name not in SCALARS and name != "side":
            setattr(f, name, at)
    f.keep, f.at = keep, at
    return f


def forward(L, f, X=None):
    return L.csrst_fno_forward(C.addressof(f), f.at if X is None else X, f.at, f.at, None)


def backward(L, f, X=None):
    return L.csrst_fno_backward(C.addressof(f), f.at if X is None else X, f.at, None, f.at, None)


def passes(L, f):
    return E_ARG not in (forward(L, f), backward(L, f))


def test_a_whole_structure_passes(gpu_lib, net):
    assert passes(gpu_lib, net)
    net.layers = 1
    net.Hfull = None                     # one layer has no kept pre-activations
    assert passes(gpu_lib, net)


@pytest.mark.parametrize("field,value", [
    ("nout", 80), ("nout", 8), ("nout", 24), ("nout", 0), ("width", 96), ("width", 0), ("width", 1 << 16),
    ("modes", 48), ("modes", 65536), ("layers", 0), ("batch", 37), ("batch", 96), ("batch", 8192), ("batch", 0),
    ("batch", 1 << 23)])
def test_sizes(gpu_lib, net, field, value):
    setattr(net, field, value)
    assert forward(gpu_lib, net) == backward(gpu_lib, net) == E_ARG
    if field in ("nout", "width", "modes", "layers"):
        assert gpu_lib.csrst_fno_refresh(C.addressof(net), 1 << 40, None) == E_ARG


FORWARD = ("w", "w16", "F16", "G16", "V16", "U16", "Z16", "Zp16", "A1_16", "Mk16", "Vg16", "Ut16", "Hfull", "A1pre",
           "A1t16")
BACKWARD = ("g", "WT16", "MkT16", "Q1T16", "Q2T16", "FT16", "GT16", "out", "Xt16", "dOut", "dOut16", "dOutT16", "dA1",
            "dH", "dH16", "dHt16", "dV", "dVn", "dZ16", "dZt16", "dSk16", "dS16", "dMk", "part", "cpart", "lpart",
            "loss")


@pytest.mark.parametrize("field", FORWARD + BACKWARD)
def test_missing_arrays(gpu_lib, net, field):
    setattr(net, field, None)
    assert backward(gpu_lib, net) == E_ARG
    assert (forward(gpu_lib, net) == E_ARG) == (field in FORWARD)


@pytest.mark.parametrize("field", sorted(TABLES))
def test_missing_table_entries(gpu_lib, net, field):
    t = (C.c_void_p * TABLES[field])(*[net.at] * TABLES[field])
    t[TABLES[field] - 1] = None
    setattr(net, field, C.addressof(t))
    assert backward(gpu_lib, net) == E_ARG


@pytest.mark.parametrize("field", ["w16", "F16", "U16", "A1_16", "A1pre", "dH", "dZt16", "FT16"])
def test_misaligned_arrays(gpu_lib, net, field):
    setattr(net, field, net.at + 8)
    assert backward(gpu_lib, net) == E_ARG
    setattr(net, field, net.at)
    assert forward(gpu_lib, net, net.at + 2) == backward(gpu_lib, net, net.at + 2) == E_ARG    # X16


def test_refresh(gpu_lib, net):
    n = 128 * 64 + 128 + 3 * (128 * 128 + 128 + 2 * 32 * 128 * 128) + 128 * 128 + 128 + 32 * 128 + 32
    p = C.addressof(net)
    assert gpu_lib.csrst_fno_refresh(p, n - 1, None) == E_ARG    # copies read w16 beyond what would be cast
    assert gpu_lib.csrst_fno_refresh(p, n, None) != E_ARG
    for field in ("WT16", "Mk16", "MkT16", "Q1T16", "Q2T16"):
        old = getattr(net, field)
        setattr(net, field, None)
        assert gpu_lib.csrst_fno_refresh(p, n, None) == E_ARG
        setattr(net, field, old)


def test_inference_needs_no_training_arrays(gpu_lib, net):
    for name in FORWARD[10:] + BACKWARD:
        setattr(net, name, None)
    net.train, net.batch = 0, 37                  # any batch
    assert forward(gpu_lib, net) != E_ARG
    assert backward(gpu_lib, net) == E_ARG
