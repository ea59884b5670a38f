"""The driver's look at the workspace's status word: an expired wait, written there by the host as a kernel would, ends the
run with an error; marks that are no error stay for their reader."""
import pytest
import torch

from tests.test_gpu_driver import _objects

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [True, False])
def test_expired_wait_ends_the_run(cuda, graph):
    from ad_afqmc_prototype_gb300 import _lib, engine
    from ad_afqmc_prototype_gb300.driver import make_run_blocks
    from ad_afqmc_prototype_gb300.prop.afqmc import init_prop_state
    from ad_afqmc_prototype_gb300.prop.blocks import afqmc_block
    from ad_afqmc_prototype_gb300.prop.chol_afqmc_ops import make_chol_afqmc_ops
    sys_, ham, trial, t_ops, m_ops, params = _objects(32)
    p_ops = make_chol_afqmc_ops(ham, "restricted")
    kw = dict(sys=sys_, params=params, ham_data=ham, trial_data=trial, meas_ops=m_ops, prop_ops=p_ops,
              prop_ctx=p_ops.build_prop_ctx(t_ops.get_rdm1(trial), params.dt),
              meas_ctx=m_ops.build_meas_ctx(ham, trial))
    st = init_prop_state(sys=sys_, n_walkers=32, seed=params.seed, ham_data=ham, trial_ops_=t_ops, trial_data=trial,
                         meas_ops=m_ops)
    run = make_run_blocks(lambda s: afqmc_block(s, **kw), kw if graph else None)
    _, want, _ = run(st, n_blocks=2)
    engine.workspace_counters()
    word = engine._arena.buf[torch.cuda.current_device()][:4].view(torch.int32)
    word.fill_(_lib.AFQ_STATUS_WAIT_EXPIRED)
    with pytest.raises(_lib.EngineError):
        run(st, n_blocks=2)
    _, again, _ = run(st, n_blocks=2)  # the word has been cleared
    assert torch.equal(again, want)
    word.fill_(_lib.AFQ_STATUS_NONFINITE)
    run(st, n_blocks=2)
    assert engine.workspace_counters()[0] == _lib.AFQ_STATUS_NONFINITE
