"""Frames of an ArrayTrajectory: callers own what frame_arrays returns, and
the driver's read-only access sees the same frames without a copy."""
import numpy as np
import pytest


def trajectory(cm, cls=None):
    rng = np.random.default_rng(3)
    sel = cm.AtomSelection.from_indices(list(range(1, 7)), natomspermol=3)
    other = cm.AtomSelection.from_indices(list(range(7, 13)), natomspermol=3)
    return (cls or cm.ArrayTrajectory)(sel, other, solute_frames=rng.random((5, 6, 3)), solvent_frames=rng.random((5, 6, 3)),
                                       cells=np.repeat(np.eye(3)[None] * 9.0, 5, 0))


@pytest.mark.parametrize("idx", [[0], [1, 2, 3], [0, 2, 4], [3, 2], [2, 2], [-2, -1], [4], []])
def test_frame_arrays_are_copies(cm, idx):
    t = trajectory(cm)
    stored = [a.copy() for a in (t._xs, t._xv, t._cells)]
    views = [np.array(a) for a in t._frames_to_submit(idx)]
    got = t.frame_arrays(idx)
    for a, v, s in zip(got, views, stored):
        assert np.array_equal(a, s[np.asarray(idx, dtype=np.int64)]) and np.array_equal(a, v)
        a += 1.0
    assert all(np.array_equal(a, s) for a, s in zip((t._xs, t._xv, t._cells), stored))


def test_consecutive_frames_are_submitted_without_a_copy(cm):
    t = trajectory(cm)
    assert all(np.shares_memory(a, b) for a, b in zip(t._frames_to_submit([1, 2, 3]), (t._xs, t._xv, t._cells)))


def test_an_override_is_what_the_driver_reads(cm):
    class Shifted(cm.ArrayTrajectory):
        def frame_arrays(self, idx):
            xs, xv, cells = super().frame_arrays(idx)
            return xs + 1.0, xv, cells

    t = trajectory(cm, Shifted)
    assert np.array_equal(t._frames_to_submit([1, 2])[0], t._xs[1:3] + 1.0)
