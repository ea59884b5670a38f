"""Binary64 QR (csrc/k_walker.cu) over the column counts its warps split differently, against the oracle.

1e-12: the Householder forms agree to about cond(W) n eps; the walkers' condition is below 30 here.
"""
import ctypes

import numpy as np
import pytest
import torch

from ad_afqmc_prototype_gb300 import _lib, engine
from oracle import afqmc_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,o", [(1, 1), (3, 2), (31, 3), (32, 8), (33, 9), (50, 10), (65, 17), (64, 25), (90, 33),
                                 (130, 34), (64, 64), (200, 30), (512, 30)])
def test_qr_matches_oracle(n, o):
    rng = np.random.default_rng(n * 100 + o)
    w = rng.normal(size=(4, n, o)) + 1j * rng.normal(size=(4, n, o)) + 3 * np.sqrt(n) * np.eye(n, o)
    q, det = engine.orthogonalize(torch.as_tensor(w, device="cuda"))
    wq, wdet = O.orthogonalize(w)
    assert np.abs(q.cpu().numpy() - wq).max() < 1e-12
    det2 = (det * det).cpu().numpy()
    assert np.abs(det2 - wdet).max() < 1e-12 * np.abs(wdet).max()


def _householder(w):
    d = engine.make_dims(w.shape[0], w.shape[1], w.shape[2], 1, True)
    q, det = torch.empty_like(w), torch.empty(w.shape[0], dtype=torch.complex128, device="cuda")
    _lib.call("afq_orthogonalize", ctypes.byref(d), engine.ptr(w), engine.ptr(q), engine.ptr(det), engine.stream_ptr())
    return q, det


# digit products from 17 columns and n o^2 = 13000 on: edges of the 128 x 64 tiles, of a row's 32 k and of the elimination
@pytest.mark.parametrize("n,o", [(45, 17), (24, 24), (33, 32), (64, 33), (129, 18), (64, 64), (257, 25), (512, 17)])
@pytest.mark.parametrize("in_place", [False, True])
def test_digit_qr_and_its_householder_walkers(n, o, in_place):
    """Walkers near orthogonal by digits against the oracle; the others (a small column, nearly and exactly dependent
    columns, a zero column, nan, inf) give the Householder kernel's bits."""
    rng = np.random.default_rng(n * 100 + o)
    w = rng.normal(size=(9, n, o)) + 1j * rng.normal(size=(9, n, o)) + 3 * np.sqrt(n) * np.eye(n, o)
    w[1, :, 3] *= 1e-3
    w[2, :, o - 1] = w[2, :, 0] + 1e-4 * w[2, :, o - 1]
    w[4, :, 5] = w[4, :, 2]
    w[5, :, 7] = 0.0
    w[6, n - 1, 0] = np.nan
    w[7, 2, 1] = np.inf
    dev = torch.as_tensor(w, device="cuda")
    hq, hdet = _householder(dev)
    q, det = engine.orthogonalize(dev, out=dev if in_place else None)
    other = [1, 2, 4, 5, 6, 7]
    assert torch.equal(torch.view_as_real(q[other]).view(torch.int64), torch.view_as_real(hq[other]).view(torch.int64))
    assert torch.equal(torch.view_as_real(det[other]).view(torch.int64), torch.view_as_real(hdet[other]).view(torch.int64))
    good = [0, 3, 8]
    wq, wdet = O.orthogonalize(w[good])
    assert np.abs(q[good].cpu().numpy() - wq).max() < 1e-12
    assert np.abs((det[good] ** 2).cpu().numpy() - wdet).max() < 1e-12 * np.abs(wdet).max()
    assert not torch.equal(q[good], hq[good])
