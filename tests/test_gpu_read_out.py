"""Read-outs larger than a pinned buffer (512 KB): counts of one weight class,
of two, and raw counts, against the oracle's half units.  The group blocks end
inside a buffer, and at 256 bins and 128 groups each is half of one."""
import numpy as np
import pytest

from helpers import KEYS, ORTHO, compare
from test_gpu_agrid import chain_system

pytestmark = pytest.mark.gpu

FIELDS = ("md_count", "md_count_random", "rdf_count", "rdf_count_random", "solute_group_count",
          "solute_group_count_random", "solvent_group_count", "solvent_group_count_random")


@pytest.mark.parametrize("n,nbins", [(128, 256), (200, 600), (257, 600)])
def test_read_out(cm, orc, gpu_ready, n, nbins):
    rng = np.random.default_rng(41)
    xs, xv, cells = chain_system(rng, ORTHO, n=n, nframes=2, mv=130, apv=3, spread=0.4)
    opt = dict(irefatom=1, cutoff=6.0, dbulk=6.0, usecutoff=False, n_random_samples=3, binstep=6.0 / nbins, nbins=nbins,
               seed=97)
    system = dict(ms=1, aps=n, mv=130, apv=3, self_mode=False, precision="fp32", regime="atoms")
    frame = []
    for f in range(2):
        got, ref, st = compare(cm, orc, xs=xs[f : f + 1], xv=xv[f : f + 1], cells=cells[f : f + 1], frame_ids=[f + 1],
                               **system, **opt)
        frame.append(ref)
    kw = dict(solute_nmols=1, solute_natomspermol=n, solvent_nmols=130, solvent_natomspermol=3, autocorrelation=False,
              regime="atoms", **opt)
    for w in ((0.75, 0.75), (0.5, 1.5)):
        with cm.Engine(**kw) as e:
            e.submit(xs, xv, cells, weights=w, frame_ids=[1, 2])
            c = e.counts()
        for key, field in zip(KEYS, FIELDS):
            a, b = (np.asarray(r[key], dtype=np.float64).reshape(c[field].shape) for r in frame)
            want = w[0] * ((a + b) / 2.0) if w[0] == w[1] else w[0] * (a / 2.0) + w[1] * (b / 2.0)
            assert np.array_equal(c[field], want), field
