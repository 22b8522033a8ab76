"""Random-insertion pieces of the candidate grid: the slots of a piece are
sorted by fine cell over the frames the piece touches, and the queries inside
the guard band are decided after it.  Pieces that end inside a frame, at a
frame's end and one sample after it, coordination-number runs (no pieces), and
a fused batch of systems with different numbers of pieces.
"""
import numpy as np
import pytest

from helpers import KEYS, ORTHO, TRICLINIC, compare
from test_gpu_agrid import chain_system

pytestmark = pytest.mark.gpu

# under a budget a piece is 58 samples for three-site molecules and 41 for one-site ones
BUDGET = 4 << 30


@pytest.mark.parametrize("apv,samples", [(3, 29), (3, 30), (3, 58), (3, 59), (1, 41), (1, 50)])
@pytest.mark.parametrize("H", [ORTHO, TRICLINIC], ids=["ortho", "triclinic"])
def test_pieces_match_oracle(cm, orc, gpu_ready, apv, samples, H):
    rng = np.random.default_rng(31)
    xs, xv, cells = chain_system(rng, H, n=200, nframes=3, mv=130, apv=apv, spread=0.4)
    opt = dict(irefatom=1, cutoff=6.0, dbulk=4.5, usecutoff=True, n_random_samples=samples, binstep=0.01, nbins=600,
               seed=95)
    got, ref, st = compare(cm, orc, ms=1, aps=200, mv=130, apv=apv, xs=xs, xv=xv, cells=cells, self_mode=False,
                           precision="fp32", regime="atoms", groups="custom",
                           engine_kw=dict(atoms_grid=3, hbm_budget_bytes=BUDGET), **opt)
    assert ref["md_random"].sum() > 0 and st["guard_reevaluations"] > 0


def test_coordination_number_has_no_pieces(cm, orc, gpu_ready):
    rng = np.random.default_rng(32)
    xs, xv, cells = chain_system(rng, TRICLINIC, n=200, nframes=3, mv=300)
    opt = dict(irefatom=1, cutoff=6.0, dbulk=6.0, usecutoff=False, n_random_samples=5, binstep=0.01, nbins=600, seed=95,
               coordination_number_only=True)
    got, ref, st = compare(cm, orc, ms=1, aps=200, mv=300, apv=3, xs=xs, xv=xv, cells=cells, self_mode=False,
                           precision="fp32", regime="atoms", engine_kw=dict(atoms_grid=3), **opt)
    assert ref["md"].sum() > 0 and st["guard_reevaluations"] > 0


def test_fused_batch_of_different_piece_counts(cm, gpu_ready):
    rng = np.random.default_rng(33)
    kw = dict(solute_nmols=1, solute_natomspermol=200, solvent_nmols=130, solvent_natomspermol=3, autocorrelation=False,
              irefatom=1, cutoff=6.0, binstep=0.02, dbulk=6.0, usecutoff=False, nbins=300, n_random_samples=40, seed=96,
              regime="atoms", atoms_grid=3)
    items = [chain_system(rng, ORTHO, n=200, nframes=4, mv=130) for _ in range(3)]
    budgets = (0, BUDGET, 0)
    alone = []
    for (xs, xv, cells), b in zip(items, budgets):
        with cm.Engine(hbm_budget_bytes=b, **kw) as e:
            e.submit(xs, xv, cells)
            alone.append(e.raw_counts())
    engines = [cm.Engine(hbm_budget_bytes=b, **kw) for b in budgets]
    with cm.Batch(engines) as batch:
        batch.submit(items)
        assert batch.graph_stats()["fused_rounds"] == 1
    for e, ref in zip(engines, alone):
        got = e.raw_counts()
        for k in KEYS:
            assert np.array_equal(got[k], ref[k]), k
        assert got["md_random"].sum() > 0
        e.close()


@pytest.mark.parametrize("apv,mv,aps", [(4, 120, 200), (5, 120, 200), (14, 60, 300), (32, 20, 150)])
def test_default_grid_of_larger_solvent_molecules(cm, orc, gpu_ready, apv, mv, aps):
    """Four lanes a query from five sites on (one below), by the default rule,
    against the oracle and with far fewer atom pairs than the walk."""
    rng = np.random.default_rng(34)
    H = np.diag([40.0, 38.0, 42.0])
    xs, xv, cells = chain_system(rng, H, n=aps, nframes=3, mv=mv, apv=apv, spread=1.2)
    opt = dict(irefatom=2, cutoff=6.0, dbulk=6.0, usecutoff=False, n_random_samples=20, binstep=0.01, nbins=600, seed=97)
    evals = {}
    for grid in (0, -1):
        got, ref, st = compare(cm, orc, ms=1, aps=aps, mv=mv, apv=apv, xs=xs, xv=xv, cells=cells, self_mode=False,
                               precision="fp32", regime="atoms", engine_kw=dict(atoms_grid=grid), **opt)
        evals[grid] = st["atom_pairs_evaluated"]
    assert ref["md_random"].sum() > 0 and evals[0] < evals[-1]
