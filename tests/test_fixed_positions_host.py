"""The integer positions of the FP32 search's prep kernels (cm_fixed.h),
compiled for the host, against exact rational arithmetic: coordinates in and
out of the unit cell, orthorhombic and triclinic cells, FP32 and FP64 inputs,
and the values that must be left to the FP64 chain.

Bounds (u = 2^-24): a cell-relative position within (1 + 2^-19) u of its
bound's magnitude (the sum of the cell edges' components) plus the integer
error 3 (2^-40 + |x| 2^-64 |H|) + |H| 2^-62 + the FP64 rounding of H^-1 times
the coordinate; a displacement in FP32 within u of its magnitude plus 2^-40.
"""
import ctypes
import os
import subprocess
from fractions import Fraction as Fr

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "complexmixtures.jl_gb300", "csrc")

SRC = r"""
#include "cm_fixed.h"
using namespace cmgeom;
extern "C" int bin32(const FrameGeom *G, const float *x, int *c, float *q) {
    FixedGeom X; memset(&X, 0, sizeof X);
    for (int i = 0; i < 9; ++i) if (!fixed_geometry_entry(*G, X, i)) return 2;
    for (int k = 0; k < 3; ++k) X.n[k] = G->n[k];
    X.ortho = G->hortho;
    int64_t p[3]; bool ok = true;
    for (int k = 0; k < 3; ++k) ok = fixed_of(x[k], p[k]) && ok;
    if (!ok) return 1;
    bin_fixed(X, p[0], p[1], p[2], c, q);
    return 0;
}
extern "C" int bin64(const FrameGeom *G, const double *x, int *c, float *q) {
    FixedGeom X; memset(&X, 0, sizeof X);
    for (int i = 0; i < 9; ++i) if (!fixed_geometry_entry(*G, X, i)) return 2;
    for (int k = 0; k < 3; ++k) X.n[k] = G->n[k];
    X.ortho = G->hortho;
    int64_t p[3]; bool ok = true;
    for (int k = 0; k < 3; ++k) ok = fixed_of(x[k], p[k]) && ok;
    if (!ok) return 1;
    bin_fixed(X, p[0], p[1], p[2], c, q);
    return 0;
}
extern "C" int unwrap64(const FrameGeom *G, const double *a, const double *b, float *d) {
    FixedGeom X; memset(&X, 0, sizeof X);
    for (int i = 0; i < 9; ++i) fixed_geometry_entry(*G, X, i);
    int64_t p[3], q[3];
    for (int k = 0; k < 3; ++k) { fixed_of(a[k], p[k]); fixed_of(b[k], q[k]); p[k] -= q[k]; }
    if (!fixed_unwrap(X, p)) return 1;
    for (int k = 0; k < 3; ++k) d[k] = fixed_f32(p[k]);
    return 0;
}
extern "C" int64_t mean(int64_t s, int n) { return fixed_mean(s, n); }
extern "C" float bound(double x) { int64_t X; fixed_of(x, X); return fixed_abs(X); }
extern "C" int size() { return (int)sizeof(FrameGeom); }
"""


class FrameGeom(ctypes.Structure):
    _fields_ = [("H", ctypes.c_double * 9), ("Hi", ctypes.c_double * 9), ("Hn", ctypes.c_double * 9),
                ("det", ctypes.c_double), ("w", ctypes.c_double * 3), ("cw", ctypes.c_double * 3),
                ("weight", ctypes.c_double), ("hw", ctypes.c_double), ("frame_id", ctypes.c_int64),
                ("n", ctypes.c_int * 3), ("ncell", ctypes.c_int), ("sample_off", ctypes.c_int),
                ("nsamples", ctypes.c_int), ("ndistinct", ctypes.c_int), ("hortho", ctypes.c_int)]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("fixed")
    src, so = d / "f.cpp", d / "f.so"
    src.write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", f"-I{CSRC}", str(src), "-o", str(so)],
                   check=True)
    lib = ctypes.CDLL(str(so))
    lib.mean.restype = ctypes.c_int64
    lib.mean.argtypes = [ctypes.c_int64, ctypes.c_int]
    lib.bound.restype = ctypes.c_float
    lib.bound.argtypes = [ctypes.c_double]
    assert lib.size() == ctypes.sizeof(FrameGeom)
    return lib


def geom(H, n):
    g = FrameGeom()
    Hi = np.linalg.inv(H)
    g.H[:] = H.T.ravel()
    g.Hi[:] = Hi.ravel()
    g.Hn[:] = (H / np.asarray(n)[None, :]).T.ravel()
    g.n[:] = n
    g.ncell = int(np.prod(n))
    g.hortho = int(np.count_nonzero(H - np.diag(np.diag(H))) == 0)
    return g


TRI = np.array([[31.7, 15.85, -4.1], [0.0, 27.45, 6.3], [0.0, 0.0, 25.9]])
SMALL = np.diag([2.5, 900.0, 77.77])


@pytest.mark.parametrize("H,n", [(np.diag([60.0, 61.5, 59.25]), (5, 6, 1)), (TRI, (3, 2, 4)), (SMALL, (1, 90, 7))],
                         ids=["ortho", "triclinic", "narrow"])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_cells_and_positions(lib, H, n, dtype):
    rng = np.random.default_rng(3)
    g = geom(H, n)
    pts = np.concatenate([rng.random((600, 3)) @ H.T, (rng.random((300, 3)) * 40 - 20) @ H.T, rng.normal(size=(50, 3)) * 1e-4,
                          np.array([[0.0, 0.0, 0.0], [-1e-9, 1e-12, -0.0], [H[0, 0], 0.0, 0.0], [3e5, -3e5, 1e5]])])
    fn = lib.bin32 if dtype == np.float32 else lib.bin64
    ct = ctypes.c_float if dtype == np.float32 else ctypes.c_double
    Hi = [[Fr(float(v)) for v in row] for row in np.array(list(g.Hi)).reshape(3, 3)]
    Hn = [[Fr(float(v)) for v in row] for row in np.array(list(g.Hn)).reshape(3, 3)]  # [k][m]: edge k
    hmax = float(np.abs(H).max())
    for p in pts.astype(dtype):
        c, q = (ctypes.c_int * 3)(), (ctypes.c_float * 3)()
        assert fn(ctypes.byref(g), (ct * 3)(*[float(v) for v in p]), c, q) == 0
        x = [Fr(float(v)) for v in p]
        lost = 3 * (2.0**-40 + float(np.abs(p).max()) * 2.0**-64 * hmax) + hmax * 2.0**-62
        # c + g and the exact fractional coordinate times n agree modulo n
        pos = [Fr(0)] * 3
        for k in range(3):
            assert 0 <= c[k] < n[k]
            t = sum(Hi[k][j] * x[j] for j in range(3))
            f = (t - (t.numerator // t.denominator)) * n[k]
            gk = f - c[k]
            # a point on a cell face may fall on either side of it
            if not -1e-9 <= gk <= 1 + 1e-9:
                gk += n[k] if gk < 0 else -n[k]
            assert -1e-9 <= gk <= 1 + 1e-9
            for m in range(3):
                pos[m] += gk * Hn[k][m]
        for m in range(3):
            mag = float(sum(abs(Hn[k][m]) for k in range(3)))
            assert abs(float(Fr(float(q[m])) - pos[m])) <= mag * (1 + 2.0**-19) * 2.0**-24 + lost


@pytest.mark.parametrize("H", [np.diag([20.0, 21.0, 22.0]), TRI])
def test_displacements(lib, H):
    rng = np.random.default_rng(4)
    g = geom(H, (3, 3, 3))
    Hi = np.linalg.inv(H)
    left = 0
    for _ in range(1500):
        a = rng.random(3) @ H.T
        b = a + rng.normal(scale=1.5, size=3) + H @ rng.integers(-2, 3, 3)
        d = (ctypes.c_float * 3)()
        f = Hi @ (a - b)
        if lib.unwrap64(ctypes.byref(g), (ctypes.c_double * 3)(*a), (ctypes.c_double * 3)(*b), d):
            left += 1
            assert np.abs(f - np.rint(f)).max() > 0.498
            continue
        want = (a - b) - H @ np.rint(f)
        assert np.abs(np.array(list(d)) - want).max() <= 2.0**-24 * np.abs(want).max() + 8 * 2.0**-40 + 1e-12
    assert left < 100


def test_left_to_fp64(lib):
    g = geom(np.diag([20.0, 20.0, 20.0]), (3, 3, 3))
    c, q = (ctypes.c_int * 3)(), (ctypes.c_float * 3)()
    for v in (float("nan"), float("inf"), -float("inf"), 4194304.0, -1e30):
        assert lib.bin32(ctypes.byref(g), (ctypes.c_float * 3)(1.0, v, 2.0), c, q) == 1
        assert lib.bin64(ctypes.byref(g), (ctypes.c_double * 3)(1.0, v, 2.0), c, q) == 1
    assert lib.bin32(ctypes.byref(geom(np.diag([1.9, 20.0, 20.0]), (1, 3, 3))), (ctypes.c_float * 3)(1.0, 1.0, 2.0), c, q) == 2


def test_mean_and_bound(lib):
    rng = np.random.default_rng(5)
    for n in (1, 2, 3, 14, 31, 32, 1000):
        for s in list(rng.integers(-2**55, 2**55, 200)) + [0, 1, -1, n, -n]:
            assert abs(Fr(int(lib.mean(int(s), n))) - Fr(int(s), n)) <= 1
    for x in rng.normal(scale=1e3, size=500):
        b = lib.bound(float(x))
        assert abs(x) <= b <= abs(x) * 1.00001 + 0.01
