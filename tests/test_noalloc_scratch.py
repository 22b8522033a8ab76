"""Scratch of the allocation-free entry point: only what the chosen search
reads.  Systems beyond the limit report what they would need before any CUDA
call; the needs are sums of 256-byte aligned pieces."""
import ctypes as C

import numpy as np
import pytest

from test_zz_no_alloc import OPT, counts_len, desc_of


def needed(cm, *, ms, aps, mv, apv, self_mode, precision, coordination):
    N = cm._native
    lib = N.load()
    d = desc_of(N, ms=ms, aps=aps, mv=mv, apv=apv, self_mode=self_mode, precision=precision)
    if coordination:
        d.mode = N.CM_MODE_COORDINATION_NUMBER
    fr = N.cm_frames()
    fr.nframes, fr.coord_type, fr.memory = 1, N.CM_COORD_F32, N.CM_MEM_DEVICE
    fr.solute_xyz = fr.solvent_xyz = C.c_void_p(16)  # never dereferenced: the size check comes first
    cell, ids = np.eye(3).reshape(9) * 300.0, np.array([1], dtype=np.int64)
    fr.cells, fr.frame_ids = N.as_ptr(cell, C.c_double), N.as_ptr(ids, C.c_int64)
    n = counts_len(aps=aps, apv=apv, self_mode=self_mode)
    buf = np.zeros(n, dtype=np.int64)
    assert lib.cm_frame_counts_noalloc(C.byref(d), C.byref(fr), N.as_ptr(buf, C.c_int64), n, None) == N.CM_EINVAL
    msg = lib.cm_last_error(None).decode()
    assert "bytes of scratch" in msg
    return int(msg.split("needs ")[1].split()[0])


@pytest.mark.parametrize("ms,aps,mv,apv,self_mode", [(200000, 14, 200000, 14, True), (500000, 1, 500000, 1, True),
                                                     (20000, 3, 600000, 3, False)])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("coordination", [False, True])
def test_scratch(cm, ms, aps, mv, apv, self_mode, precision, coordination):
    sides = [(ms, aps)] if self_mode else [(ms, aps), (mv, apv)]
    atoms, mols = sum(n * k for n, k in sides), sum(n for n, _ in sides)
    # positions in the search's type, the molecules' cells and order
    need = atoms * 16 + mols * 20 + mv * 20
    if precision == "fp64":
        need += (atoms + mols) * 32
    else:
        need += 64 * (1 << 17)  # the guard and edge queues
    if not coordination:
        distinct = min(ms, OPT["n_random_samples"])
        # bulk flags and lists, the random queue, the sampled molecules
        need += 5 * distinct * mv + 8 * max(mv, min(OPT["n_random_samples"] * mv, 1 << 18)) + 4 * ms
    got = needed(cm, ms=ms, aps=aps, mv=mv, apv=apv, self_mode=self_mode, precision=precision, coordination=coordination)
    assert need <= got <= need + (1 << 18)
