"""The tiled real pass in a box whose search cells are far wider than the
search range (at most 1,023 cells an axis: here up to 3,900 A against 8 A): its
squared-distance form |w|^2 / 2 - w q loses the difference of two positions
in such a cell to rounding, so those frames take the per-molecule kernel."""
import numpy as np
import pytest

from helpers import compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("apm", [1, 3, 7])
@pytest.mark.parametrize("edge", [30000.0, 4000000.0])
def test_wide_cells(cm, orc, gpu_ready, apm, edge):
    rng = np.random.default_rng(63)
    H = np.diag([edge, 60.0, 62.0])
    n = 600
    # clusters with neighbours at every distance up to the cutoff, far from their cell's origin
    centre = np.array([0.37, 0.5, 0.5]) @ H + rng.random((n, 3)) * np.array([14.0, 50.0, 50.0])
    centre[300:] += np.array([edge * 0.2513, 0.0, 0.0])
    xs = (centre[:, None, :] + rng.normal(scale=0.4, size=(n, apm, 3))).reshape(1, -1, 3)
    got, ref, st = compare(cm, orc, ms=n, aps=apm, mv=n, apv=apm, xs=xs, xv=None, cells=H[None], self_mode=True,
                           precision="fp32", regime="pairs", irefatom=1, cutoff=6.0, dbulk=6.0, usecutoff=False,
                           binstep=0.02, nbins=300, n_random_samples=2, seed=73)
    assert ref["md"].sum() > 0
