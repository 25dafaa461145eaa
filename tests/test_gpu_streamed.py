"""The streamed solver kernel against the FP64 restatement of the reference's solver
where its weights do not fit in shared memory (very wide and very tall costs), where
they just do, and with partial float4 chunks and row blocks of one row."""
import numpy as np
import pytest

from parity import assert_parity
from test_gpu_persistent import CFG, _problem, _reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('I,J', [(40, 30001), (30001, 44), (613, 9001), (2049, 3003)])
def test_weights_in_and_out_of_shared_memory(I, J):
    from wot_gb300 import ot
    C, G = _problem(I, J, I)
    cfg = dict(CFG, max_iter=60)
    got, _ = ot.compute_transport_matrix(solver=ot.optimal_transport_duality_gap, C=C, G=G, **cfg)
    assert_parity(got, _reference(C, G, cfg), what=(I, J))


@pytest.mark.parametrize('I,J', [(5003, 6001), (131, 200003)])
def test_costs_past_l2_against_the_on_the_fly_form(I, J):
    """Costs of more than 100 MB are loaded another way, lines asked for ahead: with
    the weights in shared memory, and with more than fit there."""
    from wot_gb300.ot import device as D
    rng = np.random.default_rng(J)
    x, y = rng.normal(size=(I, 12)).astype(np.float32), rng.normal(size=(J, 12)).astype(np.float32)
    cost, g = D.default_cost(x, y), rng.lognormal(0, 0.3, I)
    T = {form: D.solve(cost, g, dict(CFG, max_iter=45), 0, form=form).tmap.cpu().numpy()
         for form in ('materialized', 'onthefly')}
    assert_parity(T['onthefly'], T['materialized'], marginals=False, what=(I, J))
