"""Workspace of the digit products' Taylor series (csrc/k_ozgemm.cu), as the host sizes it; no device.

``n_chunks`` chunks share one workspace, sized for the first; the last is smaller where they do not divide the
walkers.  So a chunk of fewer walkers may never need more: the layout that a launch makes in the workspace depends
on its own walkers alone.
"""
import ctypes

import pytest


def _need(lib, n, o, W, n_chunks=1):
    from ad_afqmc_prototype_gb300 import _lib
    return int(lib.afq_apply_trotter_workspace(ctypes.byref(_lib.afq_dims(W, n, o, 40, 1, 0)), n_chunks))


@pytest.mark.parametrize("n,o,top", [(200, 30, 1300), (400, 50, 520), (120, 20, 3400), (100, 20, 4400), (65, 32, 5000)])
def test_fewer_walkers_never_need_more(engine_lib, n, o, top):
    last = 0
    for W in range(1, top):
        need = _need(engine_lib, n, o, W)
        assert need >= last, (W, need, last)
        last = need


@pytest.mark.parametrize("n,o,W,n_chunks", [(200, 30, 1843, 2), (400, 50, 479, 2), (100, 20, 6585, 2), (120, 20, 4993, 2),
                                            (200, 30, 2764, 3)])
def test_the_last_chunk_fits_the_first_s_workspace(engine_lib, n, o, W, n_chunks):
    first = -(-W // n_chunks)
    last = W - (n_chunks - 1) * first
    assert 0 < last < first
    assert _need(engine_lib, n, o, last) <= _need(engine_lib, n, o, W, n_chunks)
