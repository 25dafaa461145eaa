"""wotg_apply_points gives the same bits on every run: its population weights share
the column tiles' ring in shared memory, whose places are refilled while sums run."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('I,J,d,k', [(3001, 20003, 50, 8), (20003, 3001, 30, 8), (5000, 9000, 3, 3), (129, 60001, 62, 9)])
def test_repeats(I, J, d, k):
    import torch
    from wot_gb300.ot import device as D
    rng = np.random.default_rng(I)
    x, y = rng.normal(size=(I, d)).astype(np.float32), rng.normal(size=(J, d)).astype(np.float32)
    w, P = rng.normal(size=J), (rng.random((k, J)) < 0.05).astype(np.float64)
    first = D.apply_points(x, y, w, np.zeros(I), P, 0.5)
    for _ in range(8):
        assert torch.equal(D.apply_points(x, y, w, np.zeros(I), P, 0.5), first)
