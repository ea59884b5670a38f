"""Binary64 QR (csrc/k_walker.cu) over the column counts its warps split differently, against the oracle.

1e-12: the Householder forms agree to about cond(W) n eps; the walkers' condition is below 30 here.
"""
import numpy as np
import pytest
import torch

from ad_afqmc_prototype_gb300 import engine
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
