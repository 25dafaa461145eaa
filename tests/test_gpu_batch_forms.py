"""Which form a batch runs in: the loop kernel (one record of the replay profile for 60
iterations), or the launches (a record per 8 iterations) where the loop's tiles would come
out uneven or half full, one item streams a cost past L2, or a pair has very many items.
Against the single-problem driver either way."""
import pytest

from parity import coupling_err
from test_gpu_batch_loop import DEFAULTS, SAME_DEVICE_TOL, _pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('I,J,pairs,n,loop', [
    (300, 400, 4, 5, True), (1560, 1570, 4, 5, True), (350, 300, 30, 2, True), (700, 800, 1, 32, True),
    (5200, 5300, 1, 1, False),      # one item, cost past L2
    (5200, 5300, 1, 2, True),
    (500, 510, 77, 2, False),       # 75 pairs in two tiles, two in one
    (3300, 3310, 1, 25, False),     # 25 items, 2.7e8 exponentials
    (7001, 7003, 1, 5, False),      # 46 rows a tile
])
def test_forms(I, J, pairs, n, loop):
    from wot_gb300 import _native as N
    from wot_gb300.ot import batch as Bt, device as D
    ps = [_pair(I, J, k) for k in range(pairs)]
    items = [(p, dict(DEFAULTS, epsilon=0.05 + 0.01 * k, max_iter=60)) for p in range(pairs) for k in range(n)]
    maps = Bt.solve_batched(ps, items)
    records = N.load().wotg_batch_replay_profile(None, None, 0)
    assert records == 1 if loop else records >= 7
    for k in {0, len(items) // 2, len(items) - 1}:
        p, cfg = items[k]
        one = D.solve(ps[p].cost, ps[p].G, cfg, 0, form='materialized')
        err = coupling_err(maps[k].dense().cpu().numpy(), one.tmap.cpu().numpy())
        assert err <= SAME_DEVICE_TOL, (I, J, pairs, n, k, err)
