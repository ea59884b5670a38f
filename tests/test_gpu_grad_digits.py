"""The differentiated step's Taylor series and its reverse by digits (launch_taylor_tape_oz, launch_taylor_adj_oz in
csrc/k_ozgemm.cu), for walkers past the one-kernel form's 64 orbitals or its shared memory, against the oracle's adjoint.

Sizes: one orbital past the small kernel's, a ragged row tile past 128, columns past one 64-wide tile.  The bound, 1e-7 of
the gradient, is the one that the small sizes are held to (tests/test_gpu_grad.py): the oracle's own finite-difference pin.
"""
import numpy as np
import pytest

from .test_gpu_grad import _case, _grad

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,o,G,W", [(65, 5, 20, 6), (130, 3, 12, 3), (66, 33, 10, 2), (50, 40, 12, 2)])
def test_digit_taylor_adjoint_matches_oracle(cuda, n, o, G, W):
    import torch

    from ad_afqmc_prototype_gb300 import engine
    from oracle import adjoint_oracle as A
    from oracle import afqmc_oracle as O
    B, S, seed = 2, 3, 9
    c = _case(n, o, G, W, steps=S, qr_every=2)
    g, e, w, _ = _grad(c, B, seed, S)
    H, st0 = c["H"], c["st0"]
    ost = O.State(walkers=torch.as_tensor(st0.walkers).cpu().numpy(), weights=st0.weights.cpu().numpy(),
                  overlaps=st0.overlaps.cpu().numpy(), pop_control_ene_shift=float(st0.pop_control_ene_shift),
                  e_estimate=float(st0.e_estimate))
    fields, zetas = [], []
    for b in range(B):
        cb = b * (S + 1)
        fields.append(np.stack([engine.fill_normal((W, G), seed, cb + s).cpu().numpy() for s in range(S)]))
        zetas.append(float(engine.fill_uniform((1,), seed, cb + S).cpu()[0]))
    op = O.Params(dt=0.01, n_prop_steps=S, qr_every=2)
    prob = O.make_problem(H["h0"], H["h1"], H["chol"], H["mo_coeff"], 0.01)
    es, ws, tapes = A.run_forward(prob, op, ost, fields, zetas)
    np.testing.assert_allclose(e.cpu().numpy(), es, rtol=1e-10, atol=0)
    np.testing.assert_allclose(w.cpu().numpy(), ws, rtol=1e-10, atol=0)
    eb, wb = A.mixed_energy_bar(es, ws)
    h1bar, _ = A.run_backward(prob, op, tapes, eb, wb, W)
    assert np.linalg.norm(g.cpu().numpy() - h1bar) <= 1e-7 * np.linalg.norm(h1bar)
