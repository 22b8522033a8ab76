"""Fused batches of systems with different chains: the candidate grid with one
lane a query and with four, the stencil walk, several solute molecules, self
systems, coordination numbers (no random insertion), and different numbers of
random-insertion pieces.  Each system's counts are its own engine's."""
import numpy as np
import pytest

from helpers import KEYS, ORTHO, make_system
from test_gpu_agrid import chain_system

pytestmark = pytest.mark.gpu

OPT = dict(irefatom=1, cutoff=6.0, binstep=0.05, dbulk=6.0, usecutoff=False, nbins=120, seed=98, regime="atoms",
           max_frames_per_batch=2)
SYSTEMS = {
    "grid": dict(n=150, mv=60, apv=3, samples=8),
    "grid4": dict(n=150, mv=40, apv=7, samples=8),
    "walk": dict(n=150, mv=60, apv=3, samples=8, atoms_grid=-1),
    "pieces": dict(n=150, mv=130, apv=3, samples=70, hbm_budget_bytes=4 << 30),
    "solutes": dict(ms=3, n=20, mv=60, apv=3, samples=8),
    "self": dict(ms=30, n=5, mv=30, apv=5, samples=5, autocorrelation=True),
    "coordination": dict(n=150, mv=60, apv=3, samples=8, coordination_number_only=True),
}


def build(cm, name, rng):
    s = dict(SYSTEMS[name])
    ms, n, mv, apv, samples = s.pop("ms", 1), s.pop("n"), s.pop("mv"), s.pop("apv"), s.pop("samples")
    self_mode = s.pop("autocorrelation", False)
    if ms == 1:
        xs, xv, cells = chain_system(rng, ORTHO, n=n, nframes=5, mv=mv, apv=apv, spread=0.4)
    else:
        xs, xv, cells = make_system(rng, ORTHO, ms, n, mv, apv, 5, self_mode, spread=0.7)
    kw = dict(solute_nmols=ms, solute_natomspermol=n, solvent_nmols=mv, solvent_natomspermol=apv, autocorrelation=self_mode,
              n_random_samples=samples, **OPT, **s)
    return kw, (xs, xv, cells)


@pytest.mark.parametrize("names", [("grid", "walk"), ("walk", "grid4", "solutes"), ("coordination", "grid", "pieces"),
                                   ("pieces", "self", "walk", "grid4", "coordination", "solutes", "grid")],
                         ids=lambda n: "+".join(n))
def test_mixed_chains(cm, gpu_ready, names):
    rng = np.random.default_rng(67)
    systems = [build(cm, name, rng) for name in names]
    want = []
    for kw, (xs, xv, cells) in systems:
        with cm.Engine(**kw) as e:
            e.submit(xs, xv, cells)
            want.append(e.raw_counts())
    engines = [cm.Engine(**kw) for kw, _ in systems]
    with cm.Batch(engines) as b:
        b.submit([frames for _, frames in systems])
        st = b.graph_stats()
    assert st["fused_rounds"] == 3 and st["fused_systems"] == len(names)
    for e, ref, name in zip(engines, want, names):
        got = e.raw_counts()
        e.close()
        assert ref["md"].sum() > 0
        for k in KEYS:
            assert np.array_equal(got[k], ref[k]), (name, k)


@pytest.mark.parametrize("edge", [47.0, 95.0])
def test_zero_ranges_of_many_pieces(cm, gpu_ready, edge):
    """Boxes of 343 and 3,375 search cells (8 fine cells each, two frames): slot
    counts of 22 KB, less than one zero-fill range, and of 216 KB, four, the
    last one partial, beside another system's and over three rounds."""
    rng = np.random.default_rng(68)
    H = np.diag([edge] * 3)
    kw = dict(solute_nmols=1, solute_natomspermol=120, solvent_nmols=400, solvent_natomspermol=3, autocorrelation=False,
              n_random_samples=6, **OPT)
    frames = [chain_system(rng, H, n=120, nframes=2, mv=400, apv=3), chain_system(rng, ORTHO, n=120, nframes=2, mv=400, apv=3)]
    engines = [cm.Engine(**kw) for _ in frames]
    with cm.Batch(engines) as b:
        for _ in range(3):
            b.submit(frames)
        assert b.graph_stats()["fused_rounds"] == 3
    for e, (xs, xv, cells) in zip(engines, frames):
        with cm.Engine(**kw) as alone:
            for _ in range(3):
                alone.submit(xs, xv, cells)
            want = alone.raw_counts()
        got = e.raw_counts()
        e.close()
        assert want["md_random"].sum() > 0
        assert all(np.array_equal(got[k], want[k]) for k in KEYS)
