"""The FP32 real pass of the molecule layout at the sizes where its kernels
change: molecules of 1-5 atoms (a lane per molecule pair), 6 and more (a lane
per solvent atom, solute atoms in pairs: odd and even), up to 32; home cells
and staged tables beyond one pass of the tiled kernels; frames whose stencil
the tiled kernels do not take; and cross systems with the same sizes."""
import numpy as np
import pytest

from helpers import TRICLINIC, compare, make_system

pytestmark = pytest.mark.gpu

BOX = np.diag([26.0, 27.0, 25.0])
OPT = dict(cutoff=4.0, binstep=0.02, nbins=200, n_random_samples=4, seed=71)


@pytest.mark.parametrize("apm", [1, 2, 3, 4, 5, 6, 7, 14, 31, 32])
@pytest.mark.parametrize("real_pass", ["auto", "warp"])
def test_self(cm, orc, gpu_ready, apm, real_pass):
    rng = np.random.default_rng(41)
    n = 1200 // apm + 30
    xs, xv, cells = make_system(rng, BOX, n, apm, n, apm, 3, True, spread=0.5)
    got, ref, st = compare(cm, orc, ms=n, aps=apm, mv=n, apv=apm, xs=xs, xv=xv, cells=cells, self_mode=True,
                           precision="fp32", regime="pairs", irefatom=apm, dbulk=3.0, usecutoff=True,
                           engine_kw=dict(real_pass=real_pass), **OPT)
    assert ref["md"].sum() > 0 and ref["md_random"].sum() > 0


@pytest.mark.parametrize("aps,apv", [(1, 3), (3, 1), (5, 14), (14, 5), (13, 31), (32, 2)])
def test_cross(cm, orc, gpu_ready, aps, apv):
    rng = np.random.default_rng(42)
    ms, mv = 40, 900 // apv + 10
    xs, xv, cells = make_system(rng, TRICLINIC, ms, aps, mv, apv, 3, False, spread=0.6)
    got, ref, st = compare(cm, orc, ms=ms, aps=aps, mv=mv, apv=apv, xs=xs, xv=xv, cells=cells, self_mode=False,
                           precision="fp32", regime="pairs", groups="custom", irefatom=1, dbulk=4.0, usecutoff=False, **OPT)
    assert ref["md"].sum() > 0


@pytest.mark.parametrize("apm", [1, 3, 7])
def test_crowded_cells(cm, orc, gpu_ready, apm):
    """A cluster: a home cell of more molecules than one pass takes (256 in the
    kernel of small molecules) and more staged ones (1,536 and 1,024)."""
    rng = np.random.default_rng(43)
    n = 2300
    centre = np.concatenate([rng.normal(scale=1.3, size=(1900, 3)) + 12.0, rng.random((400, 3)) * 25.0])
    mols = centre[:, None, :] + rng.normal(scale=0.4, size=(n, apm, 3))
    xs = np.stack([mols.reshape(-1, 3) + rng.normal(scale=0.1, size=(n * apm, 3)) for _ in range(2)])
    cells = np.repeat(BOX[None], 2, axis=0)
    got, ref, st = compare(cm, orc, ms=n, aps=apm, mv=n, apv=apm, xs=xs, xv=None, cells=cells, self_mode=True,
                           precision="fp32", regime="pairs", irefatom=1, dbulk=4.0, usecutoff=False, **OPT)
    assert ref["md"].sum() > 0


@pytest.mark.parametrize("apm", [1, 3, 14, 32])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_random_insertion_and_prep(cm, orc, gpu_ready, apm, dtype):
    """Many random samples on fine bins (slots inside the FP32 placement's band
    decided apart), molecules split over the periodic boundary, coordinates far
    outside the cell, and one molecule that the integer positions leave to the
    FP64 chain (beyond 2^22 A)."""
    rng = np.random.default_rng(44)
    n = 500 // apm + 8
    xs, _, cells = make_system(rng, TRICLINIC, n, apm, n, apm, 2, True, spread=0.5)
    H = TRICLINIC
    shift = rng.integers(-3, 4, size=(n, 3)) @ H.T
    xs = xs + np.repeat(shift, apm, axis=0)[None]
    frac = xs @ np.linalg.inv(H).T
    split = np.arange(n * apm) % (2 * apm) < apm
    xs[:, split] = ((frac - np.floor(frac)) @ H.T)[:, split]
    if dtype == np.float64:
        xs[1, -apm:] += 2.0**19 * H[:, 0]
    got, ref, st = compare(cm, orc, ms=n, aps=apm, mv=n, apv=apm, xs=xs, xv=None, cells=cells, self_mode=True,
                           precision="fp32", regime="pairs", irefatom=1, cutoff=5.0, dbulk=5.0, usecutoff=False, binstep=0.01,
                           nbins=500, n_random_samples=40, seed=72, dtype=dtype)
    assert ref["md_random"].sum() > 0 and st["guard_reevaluations"] > 0
