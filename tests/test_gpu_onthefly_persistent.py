"""The persistent on-the-fly kernel against the materialised form of the same
problem, at the sizes where its partition can go wrong: fewer tiles than virtual
CTAs, one row tile shared by many CTAs and its transpose, several row tiles per
CTA, tile remainders of one point, both operand widths (up to 30 and up to 62
dimensions), absorptions, and more iterations than one launch runs."""
import numpy as np
import pytest

from parity import assert_parity

pytestmark = pytest.mark.gpu

CFG = dict(growth_iters=1, epsilon=0.05, lambda1=1, lambda2=50, epsilon0=1, tau=10000, scaling_iter=3000,
           inner_iter_max=50, tolerance=1e-8, max_iter=1e7, batch_size=5, extra_iter=1000)


def _points(I, J, d, seed):
    rng = np.random.default_rng(seed)
    k = rng.normal(size=(4, d)) * 2
    x = (rng.normal(size=(I, d)) + k[rng.integers(0, 4, I)]).astype(np.float32)
    y = (rng.normal(size=(J, d)) + k[rng.integers(0, 4, J)] + 0.2).astype(np.float32)
    return x, y, rng.lognormal(0, 0.3, I)


def _compare(I, J, d, cfg, solver):
    from wot_gb300.ot import device as D
    x, y, g = _points(I, J, d, I + J + d)
    cost = D.default_cost(x, y)
    T = {form: D.solve(cost, g, cfg, solver, form=form).tmap.cpu().numpy() for form in ('onthefly', 'materialized')}
    # the two forms may stop a batch apart, so marginals are not compared here
    assert_parity(T['onthefly'], T['materialized'], marginals=False, what=(I, J, d, solver))


@pytest.mark.parametrize('I,J,d', [(2, 3, 2), (128, 128, 30), (257, 129, 31), (60, 12001, 30), (12001, 60, 30),
                                   (2561, 2177, 30), (3001, 4097, 62)])
def test_sizes(I, J, d):
    _compare(I, J, d, CFG, 0)


@pytest.mark.parametrize('over,solver', [(dict(tau=5), 0), (dict(batch_size=1, max_iter=23), 0),
                                         (dict(tau=5, scaling_iter=2100, extra_iter=3, inner_iter_max=7), 1)])
@pytest.mark.parametrize('I,J,d', [(300, 411, 30), (1500, 1100, 50)])
def test_options(I, J, d, over, solver):
    _compare(I, J, d, dict(CFG, **over), solver)
