"""Device memory of a gradient run: its buffers, small and large, take little
more than their own bytes, and small ones few allocations."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

SRC = os.path.join(ROOT, "tests", "scratch_host.cu")
DEP = os.path.join(ROOT, "3dalm_b200", "csrc", "scratch.hpp")
LIB = os.path.join(ROOT, "tests", "_build", "libscratch_host.so")


def run(nbytes, n, every):
    if not os.path.exists(LIB) or os.path.getmtime(LIB) < max(os.path.getmtime(SRC), os.path.getmtime(DEP)):
        os.makedirs(os.path.dirname(LIB), exist_ok=True)
        subprocess.run(["nvcc", "-O2", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", SRC, "-o", LIB], check=True)
    lib = C.CDLL(LIB)
    lib.scratch_run.restype = C.c_longlong
    lib.scratch_run.argtypes = [C.c_longlong, C.c_int, C.c_int] + [C.POINTER(C.c_longlong)] * 3
    out, most, still = (C.c_longlong * n)(), C.c_longlong(), C.c_longlong()
    peak = lib.scratch_run(nbytes, n, every, out, C.byref(most), C.byref(still))
    return peak, np.array(out), most.value, still.value


# fields of 64x32x32, of 16 and 17 MiB, a little over a third and a half of a
# chunk, 512x256x128, and larger than a chunk; 90 of them with small buffers between
@pytest.mark.parametrize("field", [783360, 1 << 24, 17 << 20, 86 << 20, 129 << 20, 516 * 260 * 144 * 8, 300 << 20])
def test_bytes(field):
    n = 90
    peak, at, allocations, still = run(field, n, 7)
    assert peak >= n * field
    if field > 1 << 24:
        assert peak <= n * field + (2 << 20)
    else:
        # a chunk loses less than a field; the last one may be nearly empty
        assert peak <= n * field * 16 // 15 + (256 << 20)
        assert allocations <= n * field // ((256 - 16) << 20) + 1
    assert still == 0
    # aligned for any access, and apart
    assert not np.any(at % 256)
    assert np.all(np.diff(np.sort(at)) >= field)
