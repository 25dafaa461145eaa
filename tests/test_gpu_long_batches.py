"""Batches (the iterations between two duality-gap checks) longer than a launch of the
persistent solvers, and longer than their barriers can count: the map after max_iter
iterations in one batch is that of batches of five whose checks never hold, for each
solver, with and without absorptions."""
import pytest

from parity import assert_parity
from test_gpu_onthefly_persistent import _points
from test_gpu_persistent import CFG

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('form,I,J,n', [
    ('materialized', 90, 121, 4321),       # resident: launches of 2000 iterations
    ('materialized', 1203, 4907, 1501),    # streamed: launches of some 880
    ('materialized', 40000, 3, 38001),     # streamed: 2^24 arrivals are some 36800 iterations
    ('onthefly', 300, 411, 2503),
    ('onthefly', 1601, 1501, 28001),       # on the fly, all CTAs: 2^24 arrivals are some 27600
])
@pytest.mark.parametrize('tau', [10000, 5])
def test_one_batch(form, I, J, n, tau):
    from wot_gb300.ot import device as D
    x, y, g = _points(I, J, 8, I + J)
    cost = D.default_cost(x, y)
    cfg = dict(CFG, tau=tau, max_iter=n)
    one = D.solve(cost, g, dict(cfg, batch_size=10 ** 6), 0, form=form)
    many = D.solve(cost, g, dict(cfg, batch_size=5, tolerance=-1.0), 0, form=form)
    assert one.stats['iterations'] == many.stats['iterations'] == n
    assert one.stats['hit_max_iter'] and many.stats['hit_max_iter']
    assert_parity(one.tmap.cpu().numpy(), many.tmap.cpu().numpy(), marginals=False, what=(form, I, J, tau))
