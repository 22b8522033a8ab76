"""Error bounds of the FP32 search (cm_fixed.h), compiled for the host: a slot
placed in FP64 from its molecule's FP32 offsets lies farther from the FP64
placement than one rounding of the placed offset, by the offset's own rounding,
and the band of those slots counts it."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "complexmixtures.jl_gb300", "csrc")
SRC = r"""
#include "cm_fixed.h"
extern "C" double pair_units(double Q, double O, double rs, double rv, double c) { return cmgeom::fp32_pair_units(Q, O, rs, rv, c); }
extern "C" double slot_units(double Q, double r) { return cmgeom::fp32_slot_units(Q, r); }
extern "C" double offset_units(double r) { return cmgeom::fp32_offset_units(r); }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("band")
    (d / "b.cpp").write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-I{CSRC}", str(d / "b.cpp"), "-o", str(d / "b.so")], check=True)
    lib = ctypes.CDLL(str(d / "b.so"))
    for f, n in ((lib.pair_units, 5), (lib.slot_units, 2), (lib.offset_units, 1)):
        f.restype = ctypes.c_double
        f.argtypes = [ctypes.c_double] * n
    return lib


@pytest.mark.parametrize("r", [0.9, 3.7, 41.0])
def test_fp32_offsets_rotated_in_fp64(lib, r):
    rng = np.random.default_rng(5)
    u = 2.0**-24
    n = 200000
    w = rng.normal(size=(n, 3))
    w *= r / np.linalg.norm(w, axis=1, keepdims=True)
    q = rng.normal(size=(n, 4))
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    a, b, c, d = q.T
    A = np.array([[1 - 2 * (c * c + d * d), 2 * (b * c - a * d), 2 * (b * d + a * c)],
                  [2 * (b * c + a * d), 1 - 2 * (b * b + d * d), 2 * (c * d - a * b)],
                  [2 * (b * d - a * c), 2 * (c * d + a * b), 1 - 2 * (b * b + c * c)]]).transpose(2, 0, 1)
    exact = np.einsum("nij,nj->ni", A, w)
    rounded = np.einsum("nij,nj->ni", A, w.astype(np.float32).astype(np.float64)).astype(np.float32).astype(np.float64)
    worst = np.abs(rounded - exact).max() / u
    # one rounding of the placed offset (the pair bound's) and the offsets' own
    assert worst <= r + lib.offset_units(r)
    assert lib.offset_units(r) >= r


def test_pair_and_slot_bounds(lib):
    Q, OFF, rs, rv, cut = 21.0, 43.0, 4.1, 1.3, 10.0
    assert lib.pair_units(Q, OFF, rs, rv, cut) >= (5 * Q + 4 * OFF + 2 * rv + rs + cut + 1) * (1 + 2.0**-20)
    assert lib.slot_units(Q, rv) == 5 * Q + 44 * rv
