"""Longest sums of the digit products (csrc/k_ozgemm.cu): their 64-bit integer sums hold fewer than 2^16 of the largest
products of one sign; longer sums go on the binary64 pipe.

Reference: the exact product of the constant operands.  Tolerance: the bound of a binary64 chain of K equal terms,
K 1.1e-16 (1.5e-11 at 131072).
"""
import numpy as np
import pytest
import torch

from ad_afqmc_prototype_gb300 import engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("G", [65535, 65536, 131072])
def test_near_constant_vectors_of_one_sign(G):
    n, o, W = 4, 2, 9
    a, b, dt = 0.999 * 2.0**-20, 0.999, 0.005
    dev = lambda x, t=torch.float64: torch.as_tensor(x, dtype=t, device="cuda")  # noqa: E731
    rng = np.random.default_rng(0)
    w = rng.normal(size=(W, n, o)) + 1j * rng.normal(size=(W, n, o))
    out = engine.apply_trotter(dev(w, torch.complex128), dev(np.full((W, G), b + 0j), torch.complex128),
                               dev(np.full((G, n, n), a)), dev(np.eye(n)), np.sqrt(dt), 6)
    V = np.full((n, n), G * (a * b))
    t = want = w
    for k in range(1, 7):
        t = (1j * np.sqrt(dt) / k) * (V @ t)
        want = want + t
    got = out.cpu().numpy()
    assert np.linalg.norm(got - want) / np.linalg.norm(want) < 1.1e-16 * G
