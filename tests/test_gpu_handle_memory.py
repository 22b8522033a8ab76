"""Device memory of a handle in the atom layout: the evaluation queue holds a
chunk's real-pass items or a piece's slots, whichever are more, and a piece's
placement buffers at most 2^24 sites (20 bytes each)."""
import numpy as np
import pytest

from helpers import KEYS, ORTHO
from test_gpu_agrid import chain_system

pytestmark = pytest.mark.gpu


def run(cm, *, n, mv, apv, budget=0, frames=2, spread=0.9, **kw):
    rng = np.random.default_rng(81)
    xs, xv, cells = chain_system(rng, ORTHO, n=n, nframes=2, mv=mv, apv=apv, spread=spread)
    opt = dict(irefatom=1, cutoff=5.0, dbulk=5.0, usecutoff=False, binstep=0.05, nbins=100, seed=93)
    opt.update(kw)
    with cm.Engine(solute_nmols=1, solute_natomspermol=n, solvent_nmols=mv, solvent_natomspermol=apv, autocorrelation=False,
                   regime="atoms", max_frames_per_batch=frames, hbm_budget_bytes=budget, **opt) as e:
        e.submit(xs, xv, cells)
        return e.raw_counts(), e.device_bytes()


def test_small_system_takes_a_small_queue(cm, gpu_ready):
    got, used = run(cm, n=200, mv=181, apv=14, n_random_samples=10, atoms_grid=-1)
    # 2 frames x 10 samples x 181 slots: 58 KB of queue, 1 MB of placement buffers
    assert got["md_random"].sum() > 0 and used < (16 << 20)


def test_large_molecules_bound_the_piece(cm, gpu_ready):
    """2,000 samples of 20 2,000-site molecules (80 M sites): pieces of 419."""
    kw = dict(n=30, mv=20, apv=2000, n_random_samples=1000, spread=2.0)
    got, used = run(cm, **kw)
    assert used < (400 << 20)
    # a budget's pieces are 32 samples' worth of FP64 slots
    ref, _ = run(cm, budget=8 << 30, **kw)
    assert got["md_random"].sum() > 0
    assert all(np.array_equal(got[k], ref[k]) for k in KEYS)


@pytest.mark.parametrize("budget_mb", [520, 640, 800, 1100, 1500])
def test_budget_without_room_for_the_grids_cells(cm, gpu_ready, budget_mb):
    """A sparse box of 125,000 search cells: the grid's lists fit a quarter of
    the budget and its cells (1.5 GB) do not fit the rest, from the first frame
    on or with the second one; the stencil walk takes over."""
    rng = np.random.default_rng(82)
    xs, xv, _ = chain_system(rng, np.diag([400.0, 400.0, 400.0]), n=400, nframes=2, mv=300, apv=14)
    kw = dict(solute_nmols=1, solute_natomspermol=400, solvent_nmols=300, solvent_natomspermol=14, autocorrelation=False,
              irefatom=1, cutoff=8.0, dbulk=8.0, usecutoff=False, binstep=0.05, nbins=160, seed=94, n_random_samples=10,
              regime="atoms")
    for edges in ((400.0, 400.0), (100.0, 400.0)):
        cells = np.stack([np.diag([e] * 3) for e in edges])
        got = []
        for budget, grid in ((budget_mb << 20, 0), (0, -1)):
            with cm.Engine(hbm_budget_bytes=budget, atoms_grid=grid, **kw) as e:
                for f in range(2):
                    e.submit(xs[f : f + 1], xv[f : f + 1], cells[f : f + 1], frame_ids=[f + 1])
                got.append(e.raw_counts())
                assert budget == 0 or e.device_bytes() <= budget
        assert got[0]["md_random"].sum() > 0
        assert all(np.array_equal(got[0][k], got[1][k]) for k in KEYS)


def test_pairs_budget_holds_both_random_queues(cm, gpu_ready):
    """100 molecules, 1,000 samples a frame: the queue of a chunk's slots is
    25.6 MB, and the list of its slots inside the band as much again; a budget
    that held the first still does."""
    rng = np.random.default_rng(83)
    H = np.diag([30.0] * 3)
    xs = (rng.random((100, 1, 3)) @ H.T + rng.normal(scale=0.8, size=(100, 3, 3))).reshape(1, -1, 3)
    kw = dict(solute_nmols=100, solute_natomspermol=3, solvent_nmols=100, solvent_natomspermol=3, autocorrelation=True, irefatom=1,
              cutoff=8.0, dbulk=8.0, usecutoff=False, binstep=0.05, nbins=160, seed=3, n_random_samples=1000, regime="pairs")
    got = []
    for budget in (61 << 20, 0):
        with cm.Engine(hbm_budget_bytes=budget, **kw) as e:
            e.submit(np.repeat(xs, 2, 0), None, np.repeat(H[None], 2, 0))
            got.append(e.raw_counts())
    assert got[0]["md_random"].sum() > 0 and all(np.array_equal(got[0][k], got[1][k]) for k in KEYS)
