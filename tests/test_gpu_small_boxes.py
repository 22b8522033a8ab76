"""FP32 real pass of the molecule layout in boxes that need several images per
molecule pair, against the brute-force oracle: a search range beyond the box
width (125 images), several images along one axis only, molecules of one atom
up to 32, few molecules (several warps each) and many (one warp each); and a
cell grid whose half stencil is beyond the tiled kernels' table."""
import numpy as np
import pytest

from helpers import TRICLINIC, compare

pytestmark = pytest.mark.gpu

OPT = dict(binstep=0.02, nbins=300, n_random_samples=3, seed=74)


def whole_molecules(rng, H, n, apm, reach):
    """Molecules whose atoms lie within `reach` of their first one."""
    d = rng.normal(size=(n, apm, 3))
    d *= reach * rng.random((n, apm, 1)) / np.linalg.norm(d, axis=2, keepdims=True)
    d[:, 0] = 0.0
    return (rng.random((n, 1, 3)) @ H.T + d).reshape(1, -1, 3)


@pytest.mark.parametrize("aps,apv", [(12, 12), (32, 1), (5, 31), (1, 14)])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_range_beyond_the_box(cm, orc, gpu_ready, aps, apv, precision):
    """Atoms farther than half the box from the reference atom (the last one):
    the random insertion makes a molecule whole around that atom."""
    rng = np.random.default_rng(64)
    H = np.diag([12.0, 12.4, 11.8])
    self_mode = aps == apv
    ms, mv = (14, 14) if self_mode else (6, 20)
    xs = whole_molecules(rng, H, ms, aps, 5.5)
    xv = None if self_mode else whole_molecules(rng, H, mv, apv, 5.5)
    got, ref, st = compare(cm, orc, ms=ms, aps=aps, mv=mv, apv=apv, xs=xs, xv=xv, cells=H[None], self_mode=self_mode,
                           precision=precision, regime="pairs", backend="brute", groups="custom", irefatom=apv, cutoff=5.6,
                           dbulk=4.5, usecutoff=True, **OPT)
    assert ref["md"].sum() > 0 and ref["md_random"].sum() > 0


@pytest.mark.parametrize("apm,ms,mv", [(3, 40, 300), (14, 3, 100), (1, 1500, 1500)])
@pytest.mark.parametrize("narrow", [(0,), (1, 2)])
def test_several_images_along_some_axes(cm, orc, gpu_ready, apm, ms, mv, narrow):
    rng = np.random.default_rng(65)
    H = np.diag([14.0 if k in narrow else 48.0 + k for k in range(3)])
    self_mode = ms == mv
    xs = np.repeat(whole_molecules(rng, H, ms, apm, 1.5), 2, axis=0) + rng.normal(scale=0.1, size=(2, ms * apm, 3))
    xv = None if self_mode else np.repeat(whole_molecules(rng, H, mv, 3, 1.5), 2, axis=0)
    got, ref, st = compare(cm, orc, ms=ms, aps=apm, mv=mv, apv=apm if self_mode else 3, xs=xs, xv=xv,
                           cells=np.repeat(H[None], 2, axis=0), self_mode=self_mode, precision="fp32", regime="pairs",
                           backend="brute", irefatom=1, cutoff=6.0, dbulk=6.0, usecutoff=False, **OPT)
    assert ref["md"].sum() > 0


@pytest.mark.parametrize("apm", [3, 14])
@pytest.mark.parametrize("H", [np.diag([40.0, 41.0, 39.0]), TRICLINIC * 1.7], ids=["ortho", "triclinic"])
def test_half_stencil_beyond_the_tables(cm, orc, gpu_ready, apm, H):
    rng = np.random.default_rng(66)
    n = 900 // apm
    xs = whole_molecules(rng, H, n, apm, 2.0)
    got, ref, st = compare(cm, orc, ms=n, aps=apm, mv=n, apv=apm, xs=xs, xv=None, cells=H[None], self_mode=True,
                           precision="fp32", regime="pairs", backend="brute", cell_scale_pct=30, irefatom=2, cutoff=6.0,
                           dbulk=6.0, usecutoff=False, **OPT)
    assert ref["md"].sum() > 0
