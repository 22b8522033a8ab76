"""Random-insertion slots in fine-cell order, a CTA per 8,192 fine cells of a
frame: exactly one CTA's cells, a few more, several CTAs, and frames of
different cell counts in one chunk."""
import numpy as np
import pytest

from helpers import compare
from test_gpu_agrid import chain_system

pytestmark = pytest.mark.gpu


# search cells of 3 A: 16 x 32 x 16 = 8,192, 16 x 32 x 17, 20^3 x 8 fine cells = 64,000
@pytest.mark.parametrize("cells,grid", [((16, 32, 16), 1), ((16, 32, 17), 1), ((20, 20, 20), 2)])
@pytest.mark.parametrize("vary", [False, True], ids=["equal", "varying"])
def test_pieces_of_the_fine_cells(cm, orc, gpu_ready, cells, grid, vary):
    rng = np.random.default_rng(72)
    H = np.diag([3.02 * n for n in cells])
    xs, xv, Hs = chain_system(rng, H, n=300, nframes=4, mv=700, apv=3, spread=0.4)
    if vary:
        Hs = np.stack([H * s for s in (1.0, 0.7, 1.3, 1.0)])
    opt = dict(irefatom=1, cutoff=3.0, dbulk=3.0, usecutoff=False, n_random_samples=12, binstep=0.02, nbins=150, seed=96)
    got, ref, st = compare(cm, orc, ms=1, aps=300, mv=700, apv=3, xs=xs, xv=xv, cells=Hs, self_mode=False, precision="fp32",
                           regime="atoms", engine_kw=dict(atoms_grid=grid), **opt)
    assert ref["md_random"].sum() > 0
