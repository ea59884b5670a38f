"""The digit products (csrc/k_ozgemm.cu) past the scratch that one piece of their operands may take: calls that go in
several pieces of walkers or rows, and the walkers of ``n_chunks`` calls, which share a workspace.

References: the NumPy oracle on walkers at the pieces' edges.  Tolerance as in tests/test_gpu_ozgemm.py: 1e-13, ten times
what the oracle's own binary64 sums carry.
"""
import numpy as np
import pytest
import torch

from ad_afqmc_prototype_gb300 import engine
from oracle import afqmc_oracle as O

pytestmark = pytest.mark.gpu

RTOL = 1e-13


def _sym(b):
    return 0.5 * (b + np.swapaxes(b, -1, -2))


def _problem(n, o, G, W, seed=0, columns=None):
    """Hamiltonian, trial, walkers and fields; the walkers' columns may be others than the trial's."""
    rng = np.random.default_rng(seed)
    c = columns or o
    h1 = np.diag(np.linspace(-2.0, 0.5, n)) + 0.05 * _sym(rng.normal(size=(n, n)))
    chol = _sym(rng.normal(size=(G, n, n))) * (3.6 / n) * np.exp(-4.0 * np.arange(G) / G)[:, None, None]
    mo = np.ascontiguousarray(np.linalg.eigh(h1)[1])
    gen = torch.Generator("cuda").manual_seed(seed)
    rn = lambda *s: torch.randn(s, generator=gen, device="cuda", dtype=torch.float64)  # noqa: E731
    s = 0.2 / np.sqrt(n)
    w = torch.complex(torch.as_tensor(mo[:, :c], device="cuda") + s * rn(W, n, c), s * rn(W, n, c))
    xs = torch.complex(rn(W, G), 0.2 * rn(W, G))
    return h1, chol, np.ascontiguousarray(mo[:, :o]), w, xs


def _dev(x, dtype=torch.float64):
    return torch.as_tensor(x, dtype=dtype, device="cuda")


def _np(t, at):
    return t[at].cpu().numpy()


def _rel(got, want):
    return np.linalg.norm(got - want) / np.linalg.norm(want)


def _pctx(h1, chol, mo):
    return O.build_prop_ctx(0.0, h1, chol, O.get_rdm1(mo.astype(complex)), 0.005)


# 567 walkers of 200 x 30 a piece, 157 of 400 x 50: the first chunk is two pieces and the last is one
@pytest.mark.parametrize("n,o,W,n_chunks,edges", [(200, 30, 1135, 2, (0, 283, 284, 567, 568, 1134)),
                                                  (200, 30, 1843, 2, (0, 460, 461, 921, 922, 1842)),
                                                  (400, 50, 315, 2, (0, 78, 79, 157, 158, 314))])
def test_uneven_chunks_of_walkers(n, o, W, n_chunks, edges):
    G = 24
    h1, chol, mo, w, xs = _problem(n, o, G, W)
    pctx = _pctx(h1, chol, mo)
    out = engine.apply_trotter(w, xs, _dev(chol), _dev(pctx.exp_h1_half), pctx.sqrt_dt, 6, n_chunks=n_chunks)
    at = list(edges)
    assert _rel(_np(out, at), O.apply_trotter_r(_np(w, at), _np(xs, at), pctx, chol.reshape(G, -1), 6)) < RTOL
