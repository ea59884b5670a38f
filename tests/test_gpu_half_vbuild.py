"""The mixed forms' V-build on both sides of the line where half of it is taken: more than a wave of 128 x 256 tiles, sums
of 1024 and longer.

Reference: one step's first walkers among many and among few take different V-builds of the same sums.  The operands are
bf16 splits of 2^-24 (mixed) and 2^-17 (mixed_fast) and the sums fp32, so the walkers agree within 1e-6 and 1e-5.
"""
import numpy as np
import pytest
import torch

from tests.test_gpu_ozgemm import O_sym

pytestmark = pytest.mark.gpu


# 44 orbitals: eight tiles a row of 128; 64: sixteen; 60 orbitals are no multiple of 8 (no tensor-core Taylor series)
@pytest.mark.parametrize("precision,n,o,G,few,many", [("mixed", 44, 7, 171, 64, 1400), ("mixed", 64, 8, 176, 300, 700),
                                                      ("mixed", 40, 7, 160, 8, 1500), ("mixed_fast", 60, 9, 343, 64, 1300),
                                                      ("mixed", 160, 8, 171, 8, 200)])
def test_few_and_many_walkers_agree(cuda, precision, n, o, G, few, many):
    from ad_afqmc_prototype_gb300.core.system import system
    from ad_afqmc_prototype_gb300.ham.chol import ham_chol
    from ad_afqmc_prototype_gb300.meas.rhf import make_rhf_meas_ops
    from ad_afqmc_prototype_gb300.prop.afqmc import afqmc_step, init_prop_state
    from ad_afqmc_prototype_gb300.prop.chol_afqmc_ops import make_chol_afqmc_ops
    from ad_afqmc_prototype_gb300.prop.types import afqmc_params
    from ad_afqmc_prototype_gb300.trial.rhf import get_rdm1, make_rhf_trial_ops, rhf_trial
    rng = np.random.default_rng(7)
    h1 = np.diag(np.linspace(-2.0, 0.5, n)) + 0.05 * O_sym(rng.normal(size=(n, n)))
    chol = O_sym(rng.normal(size=(G, n, n))) * (3.6 / n) * np.exp(-4.0 * np.arange(G) / G)[:, None, None]
    mo = np.ascontiguousarray(np.linalg.eigh(h1)[1][:, :o])
    w = mo + 0.2 / np.sqrt(n) * (rng.normal(size=(many, n, o)) + 1j * rng.normal(size=(many, n, o)))
    fields = torch.as_tensor(rng.normal(size=(many, G)), device="cuda")
    sys_ = system(norb=n, nelec=(o, o), walker_kind="restricted")
    ham, trial = ham_chol(h0=0.0, h1=h1, chol=chol), rhf_trial(mo)
    t_ops, m_ops = make_rhf_trial_ops(sys_), make_rhf_meas_ops(sys_)
    p_ops = make_chol_afqmc_ops(ham, "restricted")
    meas_ctx, got = m_ops.build_meas_ctx(ham, trial), []
    for W in (many, few, many):  # the operand laid out for the most serves all
        params = afqmc_params(n_walkers=W, precision=precision, dt=0.005)
        st = init_prop_state(sys=sys_, n_walkers=W, seed=3, ham_data=ham, trial_ops_=t_ops, trial_data=trial,
                             meas_ops=m_ops, initial_walkers=torch.as_tensor(w[:W], device="cuda"),
                             initial_e_estimate=0.0)
        new = afqmc_step(st, params=params, ham_data=ham, trial_data=trial, meas_ops=m_ops, prop_ops=p_ops,
                         prop_ctx=p_ops.build_prop_ctx(get_rdm1(trial), params.dt), meas_ctx=meas_ctx,
                         fields=fields[:W])
        got.append(torch.as_tensor(new.walkers)[:few].clone())
    tol = 1e-6 if precision == "mixed" else 1e-5
    assert torch.linalg.norm(got[0] - got[1]) / torch.linalg.norm(got[0]) < tol
    assert torch.equal(got[0], got[2])
