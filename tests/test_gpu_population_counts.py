"""wotg_apply_points has kernels for up to four and up to eight populations: each
population's sums are the same, bit for bit, whichever of them takes it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('I,J,d', [(1, 1, 2), (129, 257, 30), (700, 900, 31), (5003, 6007, 62)])
@pytest.mark.parametrize('k', [1, 3, 4, 5, 9, 12, 13])
def test_counts(I, J, d, k):
    import torch
    from wot_gb300.ot import device as D
    rng = np.random.default_rng(I + k)
    x, y = rng.normal(size=(I, d)).astype(np.float32), rng.normal(size=(J, d)).astype(np.float32)
    w, b, P = rng.normal(size=J), rng.normal(size=I), rng.random((k, J))
    got = D.apply_points(x, y, w, b, P, 0.3)
    # the kernel of eight, with other populations beside each group of eight
    fill = rng.random((8, J))
    for k0 in range(0, k, 8):
        n = min(8, k - k0)
        ref = D.apply_points(x, y, w, b, np.concatenate([P[k0:k0 + n], fill[n:]]), 0.3)
        assert torch.equal(got[k0:k0 + n], ref[:n]), (I, J, d, k, k0)
