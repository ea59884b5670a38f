"""Operands of a wide range in the binary64 form's digit products (csrc/oz_digits.cuh, oz_lost).

A row's digits hold it to 2^-55 of its largest entry.  Where large entries of one operand meet only small ones of the
other, or a sum cancels, that is not enough for the result, and the product goes on the binary64 pipe.

References: the NumPy oracle in binary64.  Tolerance 1e-12: its chains of at most 2000 products carry 2000 1.1e-16 =
2.2e-13, the factorisations of the graded overlap matrices (condition below 1e3) as much.  By digits alone the cases
here are off by 1e-9 and more (2^-56 times the 10^8 and more by which the scales' product passes the results).
"""
import numpy as np
import pytest
import torch

from ad_afqmc_prototype_gb300 import engine
from oracle import afqmc_oracle as O
from tests.test_gpu_grad import _case, _grad

pytestmark = pytest.mark.gpu

RTOL = 1e-12


def _dev(x, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(x), dtype=dtype, device="cuda")


def _cdev(x):
    return _dev(x, torch.complex128)


def _rel(got, want):
    return np.linalg.norm(got.cpu().numpy() - want) / np.linalg.norm(want)


def _crandn(rng, *s):
    return rng.normal(size=s) + 1j * rng.normal(size=s)


def _prop(E, G):
    return O.PropCtx(dt=0.005, sqrt_dt=np.sqrt(0.005), exp_h1_half=E, mf_shifts=np.zeros(G), h0_prop=0.0)


def _graded(n, o, G, W, decades, seed=0):
    """Trial on the first orbitals, walkers whose rows grow by `decades` and vectors that shrink as much."""
    rng = np.random.default_rng(seed)
    s = 10.0 ** (decades * np.arange(n) / n)
    mo = np.eye(n)[:, :o]
    w = (mo + 0.3 * _crandn(rng, W, n, o)) * s[:, None]
    h1, chol = rng.normal(size=(n, n)), rng.normal(size=(G, n, n)) / s
    return mo, w, h1, chol


@pytest.mark.parametrize("n,o,G,W", [(40, 3, 60, 20), (60, 7, 500, 150), (48, 7, 900, 3)])
def test_force_bias_and_energy_of_graded_rows(n, o, G, W):
    mo, w, h1, chol = _graded(n, o, G, W, 12)
    ctx = O.build_meas_ctx(h1, chol, mo.astype(complex))
    rot = _dev(ctx.rot_chol.real)
    assert _rel(engine.force_bias(_cdev(w), _cdev(mo), rot, True), O.force_bias_r(w, ctx, mo)) < RTOL
    en = engine.energy(_cdev(w), 0.0, _cdev(mo), _cdev(ctx.rot_h1), rot, True)
    assert _rel(en, O.energy_r(w, 0.0, ctx, mo)) < RTOL


def test_only_the_walkers_concerned(cuda):
    """Graded walkers among others, past one tile of 64."""
    n, o, G, W = 40, 3, 80, 150
    mo, w, h1, chol = _graded(n, o, G, W, 12)
    plain = np.random.default_rng(1).normal(size=(W, n, o)) * 10.0 ** (-12 * np.arange(n) / n)[:, None] + mo
    w[::7] = plain[::7]
    ctx = O.build_meas_ctx(h1, chol, mo.astype(complex))
    got = engine.force_bias(_cdev(w), _cdev(mo), _dev(ctx.rot_chol.real), True).cpu().numpy()
    want = O.force_bias_r(w, ctx, mo)
    assert np.max(np.linalg.norm(got - want, axis=1) / np.linalg.norm(want, axis=1)) < RTOL


@pytest.mark.parametrize("n,o", [(60, 20), (130, 17)])
def test_green_of_graded_columns(n, o):
    """The trial's rows shrink as the walkers' grow."""
    rng = np.random.default_rng(2)
    s = 10.0 ** (10 * np.arange(n) / n)
    mo = rng.normal(size=(n, o)) / s[:, None]
    w = (rng.normal(size=(n, o)) + 0.3 * _crandn(rng, 5, n, o)) * s[:, None]
    g = engine.half_green(_cdev(w), _cdev(mo), True)
    ov = engine.overlap(_cdev(w), _cdev(mo), True)
    # m of random rows: condition below 1e3
    assert _rel(g, O.half_green(w, mo)) < RTOL and _rel(ov, O.overlap_r(w, mo)) < 10 * RTOL


@pytest.mark.parametrize("n,o,W", [(60, 20, 5), (130, 17, 70)])
def test_force_bias_from_a_graded_green(n, o, W):
    """The same, where m and G_half are products by digits (n o^2 from 24000 on); every third walker is of one size."""
    rng = np.random.default_rng(6)
    s = 10.0 ** (10 * np.arange(n) / n)
    mo = rng.normal(size=(n, o)) / s[:, None]
    w = (rng.normal(size=(n, o)) + 0.3 * _crandn(rng, W, n, o)) * s[:, None]
    w[::3] /= s[:, None]
    rot = rng.normal(size=(40, o, n)) / s
    got = engine.force_bias(_cdev(w), _cdev(mo), _dev(rot), True).cpu().numpy()
    ctx = O.MeasCtx(rot_h1=None, rot_chol=rot, rot_chol_flat=rot.reshape(40, -1))
    want = O.force_bias_r(w, ctx, mo)
    # conditions of m: below 3e3 in the graded walkers, 1e6 in those of one size (the trial's first rows are all they
    # meet); 30 roundings each
    each = np.linalg.norm(got - want, axis=1) / np.linalg.norm(want, axis=1)
    graded = np.arange(W) % 3 != 0
    assert each[graded].max() < 1e-11 and each[~graded].max() < 3e-9


@pytest.mark.parametrize("n,o,G,W,sym", [(40, 7, 200, 9, False), (40, 7, 900, 9, False), (120, 8, 40, 70, True),
                                         (36, 5, 64, 700, True)])
def test_vectors_and_fields_graded_in_opposite_directions(n, o, G, W, sym):
    rng = np.random.default_rng(3)
    s = 10.0 ** (12 * np.arange(G) / G)
    chol = rng.normal(size=(G, n, n)) / np.sqrt(n)
    if sym:
        chol = 0.5 * (chol + np.swapaxes(chol, 1, 2))
    chol /= s[:, None, None]
    xs = _crandn(rng, W, G) * s / np.sqrt(G)
    w = _crandn(rng, W, n, o)
    E = np.eye(n) + 0.01 * rng.normal(size=(n, n))
    pctx = _prop(E, G)
    got = engine.apply_trotter(_cdev(w), _cdev(xs), _dev(chol), _dev(E), pctx.sqrt_dt, 6)
    assert _rel(got, O.apply_trotter_r(w, xs, pctx, chol.reshape(G, -1), 6)) < RTOL


def _small_e(n, o, G, W, grade, seed=4):
    """E_half far below the identity, or a similarity transform of a plain problem by D: V's entries over 2 `grade` decades."""
    rng = np.random.default_rng(seed)
    chol = rng.normal(size=(G, n, n)) / np.sqrt(n * G)
    d = 10.0 ** (grade * np.arange(n) / n)
    E = np.eye(n) + 0.01 * rng.normal(size=(n, n))
    if grade:
        chol, E = d[:, None] * chol / d, d[:, None] * E / d
    else:
        E = 1e-9 * E
    return chol, E, d, rng


@pytest.mark.parametrize("grade", [0, 9])
@pytest.mark.parametrize("n,o,W", [(7, 2, 300), (30, 7, 11), (61, 18, 200), (80, 9, 6), (130, 7, 3)])
def test_taylor_series_that_the_digits_cannot_hold(n, o, W, grade):
    G = 12
    chol, E, d, rng = _small_e(n, o, G, W, grade)
    xs = _crandn(rng, W, G)
    w = _crandn(rng, 2, W, n, o) * (d[:, None] if grade else 1.0)
    pctx = _prop(E, G)
    row = 1.0 / d[:, None] if grade else np.ones((n, 1))  # rows of one size again
    want = [row * O.apply_trotter_r(x, xs, pctx, chol.reshape(G, -1), 6) for x in w]
    got = engine.apply_trotter(_cdev(w[0]), _cdev(xs), _dev(chol), _dev(E), pctx.sqrt_dt, 6)
    assert _rel(torch.as_tensor(row, device="cuda") * got, want[0]) < RTOL
    both = engine.apply_trotter_u(_cdev(w), _cdev(xs), _dev(chol), _dev(E), pctx.sqrt_dt, 6)
    for p in range(2):
        assert _rel(torch.as_tensor(row, device="cuda") * both[p], want[p]) < RTOL


@pytest.mark.parametrize("where", ["walker", "vectors"])
def test_infinities_as_in_a_binary64_sum(where):
    """One infinite entry: its products are infinities, not nan, and the other walkers or vectors keep their values."""
    n, o, G, W = 40, 3, 60, 20
    mo, w, h1, chol = _graded(n, o, G, W, 0)
    ctx = O.build_meas_ctx(h1, chol, mo.astype(complex))
    rot = ctx.rot_chol.real.copy()
    if where == "vectors":
        rot[7, 1, 30] = np.inf
        got = engine.force_bias(_cdev(w), _cdev(mo), _dev(rot), True).cpu().numpy()
        g = O.half_green(w, mo)[:, 1, 30]
        np.testing.assert_array_equal(got[:, 7].real, np.inf * np.sign(g.real))
        np.testing.assert_array_equal(got[:, 7].imag, np.inf * np.sign(g.imag))
        keep = np.arange(G) != 7
        want = O.force_bias_r(w, ctx, mo)[:, keep]
        assert np.linalg.norm(got[:, keep] - want) < RTOL * np.linalg.norm(want)
    else:
        w[3, 2, 1] = np.nan
        got = engine.force_bias(_cdev(w), _cdev(mo), _dev(rot), True).cpu().numpy()
        keep = np.arange(W) != 3
        want = O.force_bias_r(w[keep], ctx, mo)
        assert np.isnan(got[3]).all() and np.linalg.norm(got[keep] - want) < RTOL * np.linalg.norm(want)


@pytest.mark.parametrize("n,o", [(30, 3), (66, 4)])
def test_gradient_with_a_small_e_half(cuda, n, o):
    """h1 raised by a constant: E_half shrinks to 1e-3 of the identity, the weights stay as they are."""
    from ad_afqmc_prototype_gb300.ham.chol import ham_chol
    from ad_afqmc_prototype_gb300.prop.afqmc import init_prop_state
    from oracle import adjoint_oracle as A
    G, W, B, S, seed = 20, 4, 2, 2, 9
    c = _case(n, o, G, W, steps=S, qr_every=0)
    H = dict(c["H"])
    H["h1"] = np.asarray(H["h1"]) + 1380.0 * np.eye(n)  # exp(-0.005 1380) = 1e-3
    c["ham"] = ham_chol(h0=H["h0"], h1=H["h1"], chol=H["chol"])
    st0 = init_prop_state(sys=c["sys"], n_walkers=W, seed=11, ham_data=c["ham"], trial_ops_=c["t_ops"],
                          trial_data=c["trial"], meas_ops=c["m_ops"])
    c["st0"] = st0
    g, e, w, _ = _grad(c, B, seed, S)
    ost = O.State(walkers=torch.as_tensor(st0.walkers).cpu().numpy(), weights=st0.weights.cpu().numpy(),
                  overlaps=st0.overlaps.cpu().numpy(), pop_control_ene_shift=float(st0.pop_control_ene_shift),
                  e_estimate=float(st0.e_estimate))
    fields, zetas = [], []
    for b in range(B):
        cb = b * (S + 1)
        fields.append(np.stack([engine.fill_normal((W, G), seed, cb + s).cpu().numpy() for s in range(S)]))
        zetas.append(float(engine.fill_uniform((1,), seed, cb + S).cpu()[0]))
    prob = O.make_problem(H["h0"], H["h1"], H["chol"], H["mo_coeff"], 0.01)
    es, ws, tapes = A.run_forward(prob, O.Params(dt=0.01, n_prop_steps=S), ost, fields, zetas)
    np.testing.assert_allclose(e.cpu().numpy(), es, rtol=1e-10, atol=0)
    np.testing.assert_allclose(w.cpu().numpy(), ws, rtol=1e-8, atol=0)  # exponents of 1e2: 1e-16 1e4 in the energies
    assert np.all(ws > 0)
    eb, wb = A.mixed_energy_bar(es, ws)
    h1bar, _ = A.run_backward(prob, O.Params(dt=0.01, n_prop_steps=S), tapes, eb, wb, W)
    assert np.linalg.norm(g.cpu().numpy() - h1bar) <= 1e-7 * np.linalg.norm(h1bar)
