"""Small binary64 products (csrc/k_gemm.cu, k_zgemm_small) through the force bias and the propagation's V-build, against
the oracle, at the edges of their 8-, 16- and 32-row and 16-column tiles and of the 32 k staged at a time.

1e-13: sums of at most 300 products in another order carry about 20 x 1.1e-16 of the result; fifty times that.
"""
import numpy as np
import pytest
import torch

from ad_afqmc_prototype_gb300 import engine
from oracle import afqmc_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,o,G,W", [(1, 1, 1, 1), (4, 2, 16, 8), (5, 2, 17, 9), (8, 4, 32, 31), (8, 4, 33, 32), (9, 3, 64, 33),
                                     (12, 6, 48, 256), (11, 3, 31, 700), (16, 2, 65, 100), (17, 17, 15, 40), (6, 1, 300, 7)])
def test_small_products_match_oracle(n, o, G, W):
    rng = np.random.default_rng(n + o + G)
    chol = rng.normal(size=(G, n, n)) / n
    chol = 0.5 * (chol + chol.transpose(0, 2, 1))
    h1 = np.diag(np.linspace(-2.0, 0.5, n))
    mo = np.ascontiguousarray(np.linalg.qr(rng.normal(size=(n, n)))[0][:, :o])
    w = mo + 0.1 * (rng.normal(size=(W, n, o)) + 1j * rng.normal(size=(W, n, o))) / np.sqrt(n)
    xs = rng.normal(size=(W, G)) + 0.2j * rng.normal(size=(W, G))
    ctx = O.build_meas_ctx(h1, chol, mo.astype(complex))
    pctx = O.build_prop_ctx(0.0, h1, chol, O.get_rdm1(mo.astype(complex)), 0.005)
    dev = lambda x, t=torch.float64: torch.as_tensor(x, dtype=t, device="cuda")  # noqa: E731
    wd = dev(w, torch.complex128)
    fb = engine.force_bias(wd, dev(mo, torch.complex128), dev(np.ascontiguousarray(ctx.rot_chol.real)), True)
    want = O.force_bias_r(w, ctx, mo.astype(complex))
    assert np.linalg.norm(fb.cpu().numpy() - want) < 1e-13 * np.linalg.norm(want)
    out = engine.apply_trotter(wd, dev(xs, torch.complex128), dev(chol), dev(pctx.exp_h1_half), pctx.sqrt_dt, 6)
    want = O.apply_trotter_r(w, xs, pctx, chol.reshape(G, -1), 6)
    assert np.linalg.norm(out.cpu().numpy() - want) < 1e-13 * np.linalg.norm(want)
