"""Random-insertion pieces of many samples of few solvent molecules: a piece
is one launch, and its grid holds at most 65,535 samples along an axis."""
import numpy as np
import pytest

from helpers import KEYS, ORTHO, compare
from test_gpu_agrid import chain_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mv,samples", [(20, 65535), (20, 65536), (8, 66000)])
def test_many_samples_of_few_molecules(cm, orc, gpu_ready, mv, samples):
    rng = np.random.default_rng(61)
    xs, xv, cells = chain_system(rng, ORTHO, n=40, nframes=1, mv=mv, apv=2)
    opt = dict(irefatom=1, cutoff=4.0, dbulk=4.0, usecutoff=False, n_random_samples=samples, binstep=0.05, nbins=80, seed=99)
    counts = []
    for precision, grid in (("fp32", 0), ("fp32", -1), ("fp64", -1)):
        got, ref, st = compare(cm, orc, ms=1, aps=40, mv=mv, apv=2, xs=xs, xv=xv, cells=cells, self_mode=False,
                               precision=precision, regime="atoms", engine_kw=dict(atoms_grid=grid), **opt)
        counts.append(got)
    assert ref["md_random"].sum() > 0
    assert all(np.array_equal(counts[0][k], c[k]) for c in counts[1:] for k in KEYS)


def test_samples_of_several_frames(cm, orc, gpu_ready):
    """2,048 samples in each of 33 frames: chunks of 32 frames are 65,536 samples."""
    rng = np.random.default_rng(62)
    xs, xv, cells = chain_system(rng, ORTHO, n=40, nframes=33, mv=8, apv=2)
    kw = dict(irefatom=1, cutoff=4.0, dbulk=4.0, usecutoff=False, n_random_samples=2048, binstep=0.05, nbins=80, seed=99)
    with cm.Engine(solute_nmols=1, solute_natomspermol=40, solvent_nmols=8, solvent_natomspermol=2, autocorrelation=False,
                   regime="atoms", **kw) as e:
        e.submit(xs, xv, cells)
        got = e.raw_counts()
    ref = orc.run(ms=1, aps=40, mv=8, apv=2, solute_xyz=xs, solvent_xyz=xv, cells=cells, frame_ids=list(range(1, 34)),
                  autocorrelation=False, backend="cells", **kw)
    assert ref["md_random"].sum() > 0
    assert all(np.array_equal(got[k], ref[k]) for k in KEYS)
