"""The sum of a molecule's displacements in units of 2^-40 A (cm_fixed.h): a
sum beyond 2^62 units is reported (the molecule then takes the FP64 chain)
before it can wrap around."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "complexmixtures.jl_gb300", "csrc")
SRC = r"""
#include "cm_fixed.h"
extern "C" int sum(int64_t d, int n, int64_t *out) {
    int64_t s = 0;
    bool ok = true;
    for (int i = 0; i < n; ++i) ok = cmgeom::fixed_add(s, d) && ok;
    *out = s;
    return ok;
}
"""


@pytest.mark.parametrize("d,n", [(2**51 - 1, 2047), (2**51 - 1, 2049), (2**51 - 1, 8191), (-(2**51 - 1), 2049), (150 * 2**40, 27961),
                                 (150 * 2**40, 27963), (150 * 2**40, 111849), (-150 * 2**40, 70000), (0, 100000), (1, 100000)])
def test_sum(tmp_path, d, n):
    (tmp_path / "s.cpp").write_text(SRC)
    so = tmp_path / "s.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-I{CSRC}", str(tmp_path / "s.cpp"), "-o", str(so)], check=True)
    lib = ctypes.CDLL(str(so))
    lib.sum.argtypes = [ctypes.c_int64, ctypes.c_int, ctypes.POINTER(ctypes.c_int64)]
    out = ctypes.c_int64(0)
    ok = lib.sum(d, n, ctypes.byref(out))
    assert ok == (abs(d) * n < 2**62)
    if ok:
        assert out.value == d * n
