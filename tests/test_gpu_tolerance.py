"""A tolerance that no gap exceeds: the final stage runs no iteration, as in the
reference's `while duality_gap > tolerance`, and the map is the final epsilon's kernel
at the potentials of the stage before."""
import math

import numpy as np
import pytest

from parity import assert_parity
from test_gpu_onthefly_persistent import _points
from test_gpu_persistent import CFG

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('form,I,J', [('materialized', 90, 121), ('materialized', 1203, 4907), ('onthefly', 300, 411)])
def test_no_final_iteration(form, I, J):
    import torch
    from oracle import torch_ot
    from wot_gb300.ot import device as D
    x, y, g = _points(I, J, 8, I + J)
    cost = D.default_cost(x, y)
    cfg = dict(CFG, tolerance=math.inf, batch_size=50)
    stats = {}
    C = cost.C[:, :J].double() * cost.scale
    ref = torch_ot.optimal_transport_duality_gap(C, torch.as_tensor(g, device='cuda'), stats=stats, **cfg).cpu().numpy()
    got = D.solve(cost, g, cfg, 0, form=form)
    T = got.tmap.cpu().numpy()
    # each of the five stages before may end a batch of five apart (its test is 1e-6 on
    # scalings), which the map's bounds cover; a batch of the final stage is 50
    assert abs(got.stats['iterations'] - stats['iterations']) <= 25
    assert_parity(T, ref, marginals=False, what=(form, I, J))
    assert got.stats['gap'] == math.inf
    np.testing.assert_allclose(got.row_sums.cpu().numpy(), T.sum(1), rtol=1e-5)
