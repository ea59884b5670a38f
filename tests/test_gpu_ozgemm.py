"""Digit products of the binary64 form (csrc/k_ozgemm.cu) at the edges of their tiles, against the NumPy oracle.

Sizes: orbitals around the 32 from which the Taylor series goes by digits and around the 128-row tile, columns
around the 64-wide tile (2 nocc, 2 W), K around the 16-, 32-, 256- and 512-wide steps and drains, K splits.
Tolerance: the oracle's own binary64 sums of K products carry about sqrt(K) 1.1e-16 of the result (7e-15 at
the longest, K = 4225); 1e-13 allows it ten times that.
"""
import numpy as np
import pytest
import torch

from ad_afqmc_prototype_gb300 import engine
from ad_afqmc_prototype_gb300.core.system import system
from ad_afqmc_prototype_gb300.ham.chol import ham_chol
from ad_afqmc_prototype_gb300.meas.rhf import make_rhf_meas_ops
from ad_afqmc_prototype_gb300.prop.afqmc import afqmc_step, init_prop_state
from ad_afqmc_prototype_gb300.prop.blocks import afqmc_block
from ad_afqmc_prototype_gb300.prop.chol_afqmc_ops import make_chol_afqmc_ops
from ad_afqmc_prototype_gb300.prop.types import afqmc_params
from ad_afqmc_prototype_gb300.trial.rhf import get_rdm1, make_rhf_trial_ops, rhf_trial
from oracle import afqmc_oracle as O

pytestmark = pytest.mark.gpu

RTOL = 1e-13
SIZES = [(33, 7, 31, 5), (34, 8, 32, 33), (45, 9, 257, 31), (64, 8, 256, 32), (65, 65 - 1, 40, 2), (127, 7, 33, 3),
         (128, 32, 48, 2), (129, 33, 49, 2), (65, 33, 513, 65), (200, 16, 16, 4), (130, 7, 1025, 2)]


def _problem(n, o, G, W, seed=0):
    rng = np.random.default_rng(seed)
    h1 = np.diag(np.linspace(-2.0, 0.5, n)) + 0.05 * O_sym(rng.normal(size=(n, n)))
    chol = O_sym(rng.normal(size=(G, n, n))) * (3.6 / n) * np.exp(-4.0 * np.arange(G) / G)[:, None, None]
    mo = np.ascontiguousarray(np.linalg.eigh(h1)[1][:, :o])
    w = mo + 0.2 / np.sqrt(n) * (rng.normal(size=(W, n, o)) + 1j * rng.normal(size=(W, n, o)))
    xs = rng.normal(size=(W, G)) + 0.2j * rng.normal(size=(W, G))
    return h1, chol, mo, w, xs


def O_sym(b):
    return 0.5 * (b + np.swapaxes(b, -1, -2))


def _rel(got, want):
    return np.linalg.norm(got.cpu().numpy() - want) / np.linalg.norm(want)


def _dev(x, dtype=torch.float64):
    return torch.as_tensor(x, dtype=dtype, device="cuda")


@pytest.mark.parametrize("n,o,G,W", SIZES)
def test_digit_products_match_oracle(n, o, G, W):
    h1, chol, mo, w, xs = _problem(n, o, G, W)
    ctx = O.build_meas_ctx(h1, chol, mo.astype(complex))
    pctx = O.build_prop_ctx(0.0, h1, chol, O.get_rdm1(mo.astype(complex)), 0.005)
    cm, wd = _dev(mo, torch.complex128), _dev(w, torch.complex128)
    rot = _dev(np.ascontiguousarray(ctx.rot_chol.real))
    fb = engine.force_bias(wd, cm, rot, True)
    assert _rel(fb, O.force_bias_r(w, ctx, mo.astype(complex))) < RTOL
    out = engine.apply_trotter(wd, _dev(xs, torch.complex128), _dev(chol), _dev(pctx.exp_h1_half), pctx.sqrt_dt, 6)
    assert _rel(out, O.apply_trotter_r(w, xs, pctx, chol.reshape(G, -1), 6)) < RTOL
    e = engine.energy(wd, 0.0, cm, _dev(ctx.rot_h1, torch.complex128), rot, True)
    assert _rel(e, O.energy_r(w, 0.0, ctx, mo.astype(complex))) < RTOL


@pytest.mark.parametrize("n,o,W", [(1, 1, 300), (7, 7, 257), (8, 1, 3), (9, 4, 2), (16, 16, 3), (17, 5, 2), (31, 9, 2),
                                   (32, 32, 2), (33, 12, 2), (48, 20, 2), (49, 10, 153), (64, 10, 2), (63, 23, 2)])
@pytest.mark.parametrize("n_terms", [1, 6])
def test_small_taylor_matches_oracle(n, o, W, n_terms):
    """One kernel a walker (csrc/k_trotter_oz.cu): row tiles of 16, column tiles of 8, K steps of 16, its limits."""
    G = 20
    h1, chol, mo, w, xs = _problem(n, o, G, W)
    pctx = O.build_prop_ctx(0.0, h1, chol, O.get_rdm1(mo.astype(complex)), 0.005)
    out = engine.apply_trotter(_dev(w, torch.complex128), _dev(xs, torch.complex128), _dev(chol),
                               _dev(pctx.exp_h1_half), pctx.sqrt_dt, n_terms)
    assert _rel(out, O.apply_trotter_r(w, xs, pctx, chol.reshape(G, -1), n_terms)) < RTOL


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_digit_products_keep_nonfinite_rows_apart(bad):
    n, o, G, W = 45, 9, 100, 6
    h1, chol, mo, w, xs = _problem(n, o, G, W)
    pctx = O.build_prop_ctx(0.0, h1, chol, O.get_rdm1(mo.astype(complex)), 0.005)
    want = O.apply_trotter_r(w, xs, pctx, chol.reshape(G, -1), 6)
    xs[2, 17] = bad
    out = engine.apply_trotter(_dev(w, torch.complex128), _dev(xs, torch.complex128), _dev(chol),
                               _dev(pctx.exp_h1_half), pctx.sqrt_dt, 6).cpu()
    assert not torch.isfinite(torch.view_as_real(out[2])).any()
    keep = [i for i in range(W) if i != 2]
    assert _rel(out[keep], want[keep]) < RTOL


@pytest.mark.parametrize("n,o,W", [(33, 5, 3), (61, 9, 17), (64, 17, 4), (130, 33, 2)])
def test_blocks_sharing_a_v_match_single_ones(n, o, W):
    """Two spins (or halves) taken as one tile's columns give each column what it gets alone (either route's)."""
    G = 40
    h1, chol, mo, w, xs = _problem(n, o, G, 2 * W)
    pctx = O.build_prop_ctx(0.0, h1, chol, O.get_rdm1(mo.astype(complex)), 0.005)
    x, L, e = _dev(xs[:W], torch.complex128), _dev(chol), _dev(pctx.exp_h1_half)
    pair = _dev(w, torch.complex128).reshape(2, W, n, o)
    both = engine.apply_trotter_u(pair, x, L, e, pctx.sqrt_dt, 6)
    for spin in range(2):
        one = engine.apply_trotter(pair[spin].contiguous(), x, L, e, pctx.sqrt_dt, 6)
        assert _rel(both[spin], one.cpu().numpy()) < RTOL
    if o % 2 == 0 or o > 32:
        return
    c = o - 1  # a generalized walker's halves are n x 2 nocc
    halves = pair[:, :, :, :c].permute(1, 0, 2, 3).contiguous()
    g = engine.apply_trotter_g(halves.reshape(W, 2 * n, c), x, L, e, pctx.sqrt_dt, 6).reshape(W, 2, n, c)
    for p in range(2):
        one = engine.apply_trotter(halves[:, p].contiguous(), x, L, e, pctx.sqrt_dt, 6)
        assert _rel(g[:, p], one.cpu().numpy()) < RTOL


# more than a wave of 128 x 64 tiles, n^2 well above its 8 x 8 blocks I <= J: the rule of the half V-build
@pytest.mark.parametrize("n,o,W", [(29, 4, 705), (40, 9, 400), (65, 10, 161), (130, 7, 33), (200, 16, 20)])
def test_symmetric_vectors_halve_the_v_build(n, o, W):
    """Symmetric vectors' V from half its rows is the whole V's, bit for bit: a further vector that is not symmetric,
    with fields of zero, takes the whole product and adds zeros."""
    G = 40
    h1, chol, mo, w, xs = _problem(n, o, G, W)
    pctx = O.build_prop_ctx(0.0, h1, chol, O.get_rdm1(mo.astype(complex)), 0.005)
    odd = np.concatenate([chol, 0.01 * chol[:1]])
    odd[G, n - 1, 0] *= 1.5
    wd, e = _dev(w, torch.complex128), _dev(pctx.exp_h1_half)
    half = engine.apply_trotter(wd, _dev(xs, torch.complex128), _dev(chol), e, pctx.sqrt_dt, 6)
    x0 = np.concatenate([xs, np.zeros((W, 1))], axis=1)
    whole = engine.apply_trotter(wd, _dev(x0, torch.complex128), _dev(odd), e, pctx.sqrt_dt, 6)
    assert torch.equal(half, whole)
    few = slice(0, W, max(1, W // 8))
    assert _rel(half[few], O.apply_trotter_r(w[few], xs[few], pctx, chol.reshape(G, -1), 6)) < RTOL
    odd[G, n - 1, 0] *= 100.0
    x0[:, G] = xs[:, 0]
    got = engine.apply_trotter(wd, _dev(x0, torch.complex128), _dev(odd), e, pctx.sqrt_dt, 6)
    assert _rel(got[few], O.apply_trotter_r(w[few], x0[few], pctx, odd.reshape(G + 1, -1), 6)) < RTOL


def _run_objects(h1, chol, mo, w, **params):
    n, o = mo.shape
    sys_ = system(norb=n, nelec=(o, o), walker_kind="restricted")
    ham, trial, params = ham_chol(h0=0.0, h1=_dev(h1), chol=_dev(chol)), rhf_trial(_dev(mo)), afqmc_params(**params)
    m_ops, p_ops = make_rhf_meas_ops(sys_), make_chol_afqmc_ops(ham, "restricted")
    kw = dict(params=params, ham_data=ham, trial_data=trial, meas_ops=m_ops, prop_ops=p_ops,
              prop_ctx=p_ops.build_prop_ctx(get_rdm1(trial), params.dt), meas_ctx=m_ops.build_meas_ctx(ham, trial))
    st = init_prop_state(sys=sys_, n_walkers=params.n_walkers, seed=1, ham_data=ham, trial_ops_=make_rhf_trial_ops(sys_),
                         trial_data=trial, meas_ops=m_ops, initial_walkers=_dev(w, torch.complex128))
    return st, kw, sys_


@pytest.mark.parametrize("symmetric", [True, False])
def test_kept_vector_digits_match_the_step_s(symmetric):
    """A block cuts the vectors once, in either order of rows: its weights are those of single steps."""
    n, o, G, W, steps = 65, 10, 40, 161, 2
    h1, chol, mo, w, xs = _problem(n, o, G, W)
    if not symmetric:
        chol[G // 2, 3, 50] *= 1.5
    st, kw, sys_ = _run_objects(h1, chol, mo, mo + 0.05 * (w - mo), n_walkers=W, n_prop_steps=steps, qr_every=0,
                                precision="fp64")
    fields = torch.randn((steps, W, G), generator=torch.Generator("cuda").manual_seed(3), device="cuda",
                         dtype=torch.float64)
    _, obs = afqmc_block(st, sys=sys_, fields=fields, zeta=0.5, **kw)
    for i in range(steps):
        st = afqmc_step(st, fields=fields[i], **kw)
    # phases and magnitudes of overlaps through two steps of ~40 products each: 1e-13 a walker, ten times that
    assert abs(float(obs.scalars["weight"]) / float(st.weights.sum()) - 1.0) < 1e-12


@pytest.mark.parametrize("precision,n,o,G,W", [
    ("mixed", 36, 5, 40, 70), ("mixed", 40, 7, 33, 3), ("mixed", 132, 9, 40, 65), ("mixed_fast", 132, 9, 40, 7), ("mixed_fast", 160, 12, 40, 70),
    ("mixed_fast", 200, 30, 50, 129), ("mixed_fast", 264, 8, 40, 33)])
def test_mixed_symmetric_vectors_halve_the_v_build(precision, n, o, G, W):
    """One zero of a vector with a minus sign makes it unsymmetric in bits and changes no value: a step through the
    whole V-build gives the bits of one through half of it."""
    h1, chol, mo, w, _ = _problem(n, o, G, W)
    chol[0, n - 1, 2] = chol[0, 2, n - 1] = 0.0
    out = []
    for sign in (1.0, -1.0):
        chol[0, n - 1, 2] = sign * 0.0
        st, kw, _ = _run_objects(h1, chol, mo, mo + 0.05 * (w - mo), n_walkers=W, precision=precision)
        fields = torch.randn((W, G), generator=torch.Generator("cuda").manual_seed(3), device="cuda", dtype=torch.float64)
        out.append(afqmc_step(st, fields=fields, **kw))
    assert torch.equal(out[0].walkers, out[1].walkers)
    assert torch.equal(out[0].weights, out[1].weights)
    assert bool(torch.isfinite(out[0].weights).all())
