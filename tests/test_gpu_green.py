"""Overlap and Green's function kernels (csrc/k_green.cu) at the edges of their element counts, against the oracle.

Tolerance: numpy's own LU and solve carry about o eps cond(m); with walkers near the trial cond(m) < 10, so
1e-12 is fifty times that at o = 64 (overlaps are squares: twice).
"""
import numpy as np
import pytest
import torch

from ad_afqmc_prototype_gb300 import engine
from oracle import afqmc_oracle as O

pytestmark = pytest.mark.gpu


def _walkers(n, o, W, real, seed=0):
    rng = np.random.default_rng(seed)
    c = rng.normal(size=(n, o)) + (0 if real else 1j * rng.normal(size=(n, o)))
    c = np.linalg.qr(c)[0].astype(complex)
    w = c + 0.3 / np.sqrt(n) * (rng.normal(size=(W, n, o)) + 1j * rng.normal(size=(W, n, o)))
    return c, w


@pytest.mark.parametrize("real", [True, False])
@pytest.mark.parametrize("n,o", [(1, 1), (5, 2), (13, 11), (12, 12), (33, 16), (40, 17), (31, 22), (64, 23), (65, 32),
                                 (70, 33), (90, 41), (70, 51), (64, 64), (130, 40)])
def test_overlap_and_green_match_oracle(n, o, real):
    c, w = _walkers(n, o, 5, real)
    cd, wd = torch.as_tensor(c, device="cuda"), torch.as_tensor(w, device="cuda")
    ov, want = engine.overlap(wd, cd, real).cpu().numpy(), O.overlap_r(w, c)
    assert np.abs(ov - want).max() < 1e-12 * np.abs(want).max()
    g, ov2 = engine.half_green(wd, cd, real, with_overlap=True)
    wg = O.half_green(w, c)
    assert np.abs(g.cpu().numpy() - wg).max() < 1e-12 * np.abs(wg).max()
    np.testing.assert_array_equal(ov2.cpu().numpy(), ov)  # the same pivots with and without the inverse


@pytest.mark.parametrize("n,o", [(60, 20), (61, 23), (129, 33), (150, 64)])
def test_digit_green_matches_oracle(n, o):
    """Sizes from which m and G_half go by digits (n o^2 >= 24000), through the force bias' Green's function."""
    c, w = _walkers(n, o, 9, True)
    cd, wd = torch.as_tensor(c, device="cuda"), torch.as_tensor(w, device="cuda")
    # with L~_g picking single entries of G_half, fb = 2 G_half there
    rng = np.random.default_rng(1)
    pick = [(int(a), int(i)) for a, i in zip(rng.integers(0, o, 40), rng.integers(0, n, 40))]
    rot = np.zeros((40, o, n))
    for g, (a, i) in enumerate(pick):
        rot[g, a, i] = 0.5
    fb = engine.force_bias(wd, cd, torch.as_tensor(rot, device="cuda"), True).cpu().numpy()
    wg = O.half_green(w, c)
    want = np.stack([wg[:, a, i] for a, i in pick], 1)
    assert np.abs(fb - want).max() < 1e-12 * np.abs(wg).max()


def test_singular_and_permuted_overlap():
    """A zero column makes the overlap exactly 0; permuted unit columns give the permutation's sign squared."""
    n, o = 9, 5
    c = np.eye(n, o).astype(complex)
    w = np.stack([c, c[:, [1, 0, 3, 4, 2]], c[:, [4, 3, 2, 1, 0]], c])
    w[3, :, 2] = 0.0
    ov = engine.overlap(torch.as_tensor(w, device="cuda"), torch.as_tensor(c, device="cuda"), True).cpu().numpy()
    np.testing.assert_array_equal(ov, [1.0, 1.0, 1.0, 0.0])
    pair = torch.as_tensor(np.stack([w, np.broadcast_to(c, w.shape)]), device="cuda")
    det = engine.overlap_u(pair, torch.as_tensor(c, device="cuda"), True).cpu().numpy()
    np.testing.assert_array_equal(det, [1.0, -1.0, 1.0, 0.0])
