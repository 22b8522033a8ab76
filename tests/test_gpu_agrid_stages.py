"""Candidate lists of a solute whose atoms fill several stages of the build
(2,560 atoms): 2,500 atoms fit one, 2,700 and 5,200 take two and three.  The
cells around the cluster have no atoms of their own, so all of it is staged."""
import numpy as np
import pytest

from helpers import ORTHO, TRICLINIC, compare
from test_gpu_agrid import chain_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2500, 2700, 5200])
@pytest.mark.parametrize("H", [ORTHO, TRICLINIC], ids=["ortho", "triclinic"])
def test_stages_match_oracle(cm, orc, gpu_ready, n, H):
    rng = np.random.default_rng(51)
    xs, xv, cells = chain_system(rng, H, n=n, nframes=1, mv=130, apv=3, confined=1.5)
    opt = dict(irefatom=1, cutoff=6.0, dbulk=4.5, usecutoff=True, n_random_samples=4, binstep=0.01, nbins=600, seed=98)
    got, ref, st = compare(cm, orc, ms=1, aps=n, mv=130, apv=3, xs=xs, xv=xv, cells=cells, self_mode=False,
                           precision="fp32", regime="atoms", groups="custom",
                           engine_kw=dict(atoms_grid=1, atoms_grid_capacity=2000000), **opt)
    assert ref["md"].sum() > 0 and ref["md_random"].sum() > 0
