"""Candidate lists from the widest stencils the build takes (343 cells of
0.4 of the default edge): the cells that hold atoms and reach the home cell's
bound are moved to the front, 32 at a time, out of nearly full and nearly
empty stencils."""
import numpy as np
import pytest

from helpers import ORTHO, TRICLINIC, compare
from test_gpu_agrid import chain_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,spread", [(40, None), (900, None), (900, 7.0)])
@pytest.mark.parametrize("H", [ORTHO, TRICLINIC], ids=["ortho", "triclinic"])
@pytest.mark.parametrize("grid", [1, 2])
def test_wide_stencils_match_oracle(cm, orc, gpu_ready, n, spread, H, grid):
    rng = np.random.default_rng(71)
    xs, xv, cells = chain_system(rng, H, n=n, nframes=2, mv=200, apv=3, confined=spread)
    opt = dict(irefatom=2, cutoff=6.0, dbulk=6.0, usecutoff=False, n_random_samples=6, binstep=0.02, nbins=300, seed=92)
    got, ref, st = compare(cm, orc, ms=1, aps=n, mv=200, apv=3, xs=xs, xv=xv, cells=cells, self_mode=False, precision="fp32",
                           regime="atoms", cell_scale_pct=40, engine_kw=dict(atoms_grid=grid, atoms_grid_capacity=4000000), **opt)
    assert ref["md"].sum() > 0 and ref["md_random"].sum() > 0
