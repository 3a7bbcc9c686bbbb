"""The surrogate's launch sequences at their C boundary (no GPU needed): the
ctypes mirror of csrst_fno has the header's layout, and calls that cannot run
are refused before any launch."""
import ctypes as C
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_struct_layout(tmp_path):
    from csrst_b200.surrogate import _Net
    names = [f[0] for f in _Net._fields_]
    src = tmp_path / "o.c"
    src.write_text('#include <stddef.h>\n#include <stdio.h>\n#include "%s/include/csrst.h"\nint main(void) {\n' % ROOT +
                   "".join('printf("%%zu ", offsetof(csrst_fno, %s));\n' % n for n in names) +
                   'printf("%zu", sizeof(csrst_fno));\nreturn 0;\n}\n')
    subprocess.run(["gcc", "-o", str(tmp_path / "o"), str(src)], check=True)
    got = [int(v) for v in subprocess.run([str(tmp_path / "o")], capture_output=True, text=True).stdout.split()]
    assert got == [getattr(_Net, n).offset for n in names] + [C.sizeof(_Net)]


def test_refusals(gpu_lib):
    from csrst_b200.surrogate import _Net
    a, err = (C.c_float * 4)(), C.c_int()
    p, e = C.addressof(a), C.addressof(err)
    net = _Net(128, 32, 4, 32, 0, 0)            # no members
    net.w = net.g = net.w16 = p
    assert gpu_lib.csrst_fno_forward(C.addressof(net), p, p, e, None) != 0
    net.batch = 1 << 24                         # 2^32 rows
    assert gpu_lib.csrst_fno_forward(C.addressof(net), p, p, e, None) != 0
    net.batch = 64
    assert gpu_lib.csrst_fno_forward(C.addressof(net), None, p, e, None) != 0
    assert gpu_lib.csrst_fno_forward(C.addressof(net), p, p, None, None) != 0
    assert gpu_lib.csrst_fno_backward(C.addressof(net), p, p, None, e, None) != 0   # not a training structure
    assert gpu_lib.csrst_fno_refresh(C.addressof(net), 0, None) != 0
