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
