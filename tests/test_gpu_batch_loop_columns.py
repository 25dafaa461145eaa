"""The batch's loop kernel where the weights of all columns do not fit in shared memory
at once (some 52000 of them, over the entries of a group): groups that take their
columns in steps, in one round of rows and in several, and a single entry that reads its
weights from global memory. Against the single-problem driver on the same device cost."""
import pytest

from parity import coupling_err
from test_gpu_batch_loop import DEFAULTS, SAME_DEVICE_TOL, _pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('I,J,n', [(37, 27003, 2), (7003, 41, 8), (9001, 11003, 6), (33, 53001, 1), (53001, 5, 1),
                                   (19, 53001, 9)])
def test_columns_in_steps(I, J, n):
    from wot_gb300 import _native as N
    from wot_gb300.ot import batch as Bt, device as D
    pair = _pair(I, J, I)
    items = [(0, dict(DEFAULTS, epsilon=0.05 + 0.01 * k, max_iter=60)) for k in range(n)]
    maps = Bt.solve_batched([pair], items)
    assert N.load().wotg_batch_replay_profile(None, None, 0) == 1   # one launch of the loop, not replays of 8
    for k in {0, n // 2, n - 1}:
        one = D.solve(pair.cost, pair.G, items[k][1], 0, form='materialized')
        err = coupling_err(maps[k].dense().cpu().numpy(), one.tmap.cpu().numpy())
        assert err <= SAME_DEVICE_TOL, (I, J, n, k, err)
