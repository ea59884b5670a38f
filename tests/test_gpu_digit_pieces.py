"""The digit products (csrc/k_ozgemm.cu) past the 1 GiB that one piece of their operands may take: the walkers, vectors or
rows of a later piece, uneven last pieces, and what shares a workspace with them.

References: the NumPy oracle on the pieces' edges.  Tolerance 1e-13 as in tests/test_gpu_ozgemm.py (ten times the oracle's
own sums), 1e-12 for the QR (condition below 30), 1e-7 in norm for dE/dh1 as in tests/test_gpu_grad.py.
"""
import numpy as np
import pytest
import torch

from ad_afqmc_prototype_gb300 import engine
from oracle import afqmc_oracle as O
from tests.test_gpu_digit_chunks import _dev, _np, _pctx, _problem, _rel
from tests.test_gpu_grad import _case, _grad

pytestmark = pytest.mark.gpu

RTOL = 1e-13


def test_green_of_several_pieces(cuda):
    """2370 walkers of 200 x 30 a piece."""
    n, o, W = 200, 30, 2501
    _, _, mo, w, _ = _problem(n, o, 2, W)
    g, ov = engine.half_green(w, _dev(mo, torch.complex128), True, with_overlap=True)
    at = [0, 1249, 1250, 1251, 2499, 2500]
    assert _rel(_np(g, at), O.half_green(_np(w, at), mo)) < 10 * RTOL  # the solves' condition, below 10
    assert _rel(_np(ov, at), O.overlap_r(_np(w, at), mo)) < 10 * RTOL


def test_energy_of_several_pieces(cuda):
    """74 walkers of 30 columns and 1000 vectors a piece."""
    n, o, G, W = 64, 30, 1000, 151
    h1, chol, mo, w, _ = _problem(n, o, G, W)
    ctx = O.build_meas_ctx(h1, chol, mo.astype(complex))
    e = engine.energy(w, 0.0, _dev(mo, torch.complex128), _dev(ctx.rot_h1, torch.complex128),
                      _dev(np.ascontiguousarray(ctx.rot_chol.real)), True)
    at = [0, 50, 51, 101, 102, 150]
    assert _rel(_np(e, at), O.energy_r(_np(w, at), 0.0, ctx, mo)) < 10 * RTOL


def test_qr_of_several_pieces_with_householder_walkers(cuda):
    """1864 walkers of 200 x 30 a piece; dependent columns in either."""
    n, o, W = 200, 30, 2001
    gen = torch.Generator("cuda").manual_seed(5)
    rn = lambda *s: torch.randn(s, generator=gen, device="cuda", dtype=torch.float64)  # noqa: E731
    w = torch.complex(rn(W, n, o), rn(W, n, o)) + 3 * np.sqrt(n) * torch.eye(n, o, device="cuda", dtype=torch.float64)
    bad = [3, 1000, 1001, 1999]
    w[bad, :, 7] = w[bad, :, 2] + 1e-4 * w[bad, :, 7]
    q, det = engine.orthogonalize(w)
    at = [0, 999, 1002, 2000]
    wq, wdet = O.orthogonalize(_np(w, at))
    assert np.abs(_np(q, at) - wq).max() < 1e-12
    assert np.abs(_np(det, at) ** 2 - wdet).max() < 1e-12 * np.abs(wdet).max()
    alone, dalone = engine.orthogonalize(w[bad].contiguous())
    assert torch.equal(q[bad], alone) and torch.equal(det[bad], dalone)


@pytest.mark.parametrize("sym", [True, False])
def test_vbuild_of_several_pieces_of_rows(cuda, sym):
    """38016 of 40000 rows of 2000 vectors a piece (symmetric: all 20800 blocks' rows in the first)."""
    n, o, G, W = 200, 3, 2000, 9
    h1, chol, mo, w, xs = _problem(n, o, G, W)
    if not sym:
        chol[3, 0, 1] *= 1.5
        chol[7, n - 1, n - 2] *= 1.5
    pctx = O.PropCtx(dt=0.005, sqrt_dt=np.sqrt(0.005), exp_h1_half=np.eye(n) + 0.01 * h1, mf_shifts=None, h0_prop=0.0)
    out = engine.apply_trotter(w, xs, _dev(chol), _dev(pctx.exp_h1_half), pctx.sqrt_dt, 6)
    want = O.apply_trotter_r(w.cpu().numpy(), xs.cpu().numpy(), pctx, chol.reshape(G, -1), 6)
    assert _rel(out.cpu().numpy(), want) < RTOL


def test_force_bias_of_several_pieces_of_walkers(cuda):
    """31488 walkers of 1200 entries a piece."""
    n, o, G, W = 60, 20, 9, 33001
    h1, chol, mo, w, _ = _problem(n, o, G, W)
    ctx = O.build_meas_ctx(h1, chol, mo.astype(complex))
    fb = engine.force_bias(w, _dev(mo, torch.complex128), _dev(np.ascontiguousarray(ctx.rot_chol.real)), True)
    at = [0, 31487, 31488, 31489, W - 1]
    assert _rel(_np(fb, at), O.force_bias_r(_np(w, at), ctx, mo)) < 10 * RTOL


@pytest.mark.parametrize("n_chunks", [1, 2])
def test_two_spins_past_one_piece(cuda, n_chunks):
    """Both spins of 409 walkers of 200 x 30 fit a piece; with more, each spin goes by itself."""
    n, o, G, W = 200, 30, 24, 451 if n_chunks == 1 else 901
    h1, chol, mo, w, xs = _problem(n, o, G, W)
    pctx = _pctx(h1, chol, mo)
    both = torch.stack([w, 1j * w.flip(0)]).contiguous()
    out = engine.apply_trotter_u(both, xs, _dev(chol), _dev(pctx.exp_h1_half), pctx.sqrt_dt, 6, n_chunks=n_chunks)
    at = [0, 225, 226, 450, W - 1]
    for p in range(2):
        want = O.apply_trotter_r(_np(both[p], at), _np(xs, at), pctx, chol.reshape(G, -1), 6)
        assert _rel(_np(out[p], at), want) < RTOL


# V-bar: 89 walkers of 66 x 33 and 60 terms a piece; Taylor tape and reverse: 580 of 200 x 4
@pytest.mark.parametrize("n,o,W,terms", [(66, 33, 101, 60), (200, 4, 601, 6)])
def test_gradient_of_several_pieces(cuda, n, o, W, terms):
    from oracle import adjoint_oracle as A
    G, seed = 6, 9
    c = _case(n, o, G, W, steps=1, qr_every=0)
    c["params"] = c["params"]._replace(n_exp_terms=terms) if hasattr(c["params"], "_replace") else \
        __import__("dataclasses").replace(c["params"], n_exp_terms=terms)
    g, e, _, _ = _grad(c, 1, seed, 1)
    H, st0 = c["H"], c["st0"]
    ost = O.State(walkers=torch.as_tensor(st0.walkers).cpu().numpy(), weights=st0.weights.cpu().numpy(),
                  overlaps=st0.overlaps.cpu().numpy(), pop_control_ene_shift=float(st0.pop_control_ene_shift),
                  e_estimate=float(st0.e_estimate))
    fields = [np.stack([engine.fill_normal((W, G), seed, 0).cpu().numpy()])]
    zetas = [float(engine.fill_uniform((1,), seed, 1).cpu()[0])]
    prob = O.make_problem(H["h0"], H["h1"], H["chol"], H["mo_coeff"], 0.01)
    op = O.Params(dt=0.01, n_prop_steps=1, n_exp_terms=terms)
    es, ws, tapes = A.run_forward(prob, op, ost, fields, zetas)
    np.testing.assert_allclose(e.cpu().numpy(), es, rtol=1e-10, atol=0)
    h1bar, _ = A.run_backward(prob, op, tapes, *A.mixed_energy_bar(es, ws), W)
    assert np.linalg.norm(g.cpu().numpy() - h1bar) <= 1e-7 * np.linalg.norm(h1bar)
