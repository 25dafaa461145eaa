"""The batch's loop kernel (and, past its limits, the launches) against the
single-problem driver on the same device cost, at the sizes where its partition and
its groups can go wrong: one row per tile and fewer than a round, several rounds,
more columns than fit in shared memory at once, one entry, an entry alone after a
full group, more entries than a group, batches that end apart, absorptions, an
iteration limit, and more items of a pair than a tile picks from (the launches)."""
import numpy as np
import pytest

from parity import coupling_err

pytestmark = pytest.mark.gpu

SAME_DEVICE_TOL = 1e-5
DEFAULTS = dict(growth_iters=1, epsilon=0.05, lambda1=1, lambda2=50, epsilon0=1, tau=10000, scaling_iter=3000,
                inner_iter_max=50, tolerance=1e-8, max_iter=1e7, batch_size=5, extra_iter=1000)


def _pair(I, J, seed, d=8):
    from wot_gb300 import synthetic
    from wot_gb300.ot import batch as Bt, device as D
    x = synthetic.gaussian_mixture_points(I, d=d, seed=seed)
    y = synthetic.gaussian_mixture_points(J, d=d, seed=seed + 100)
    return Bt.prepare_pair(D.default_cost(x, y), np.random.default_rng(seed).lognormal(0, 0.3, I))


def _compare(pairs, items):
    from wot_gb300.ot import batch as Bt, device as D
    for (p, cfg), m in zip(items, Bt.solve_batched(pairs, items)):
        one = D.solve(pairs[p].cost, pairs[p].G, cfg, 0, form='materialized')
        err = coupling_err(m.dense().cpu().numpy(), one.tmap.cpu().numpy())
        assert err <= SAME_DEVICE_TOL, (pairs[p].cost.I, pairs[p].cost.J, cfg, err)


@pytest.mark.parametrize('I,J', [(1, 5), (7, 3), (129, 4001), (6500, 70), (1023, 1029)])
def test_sizes(I, J):
    _compare([_pair(I, J, I)], [(0, dict(DEFAULTS, epsilon=e)) for e in (0.05, 0.1)])


@pytest.mark.parametrize('n', [1, 8, 9, 17, 33])
def test_entries(n):
    _compare([_pair(150, 211, n)], [(0, dict(DEFAULTS, epsilon=0.05 + 0.01 * k)) for k in range(n)])


@pytest.mark.parametrize('over', [dict(tau=5), dict(batch_size=1), dict(batch_size=3, max_iter=41),
                                  dict(growth_iters=2, batch_size=7), dict(tau=3, lambda1=0.1)])
def test_options_on_pairs(over):
    pairs = [_pair(90, 60, 1), _pair(400, 700, 2), _pair(33, 501, 3)]
    _compare(pairs, [(k % 3, dict(DEFAULTS, epsilon=(0.05, 0.08)[k % 2], **over)) for k in range(7)])
