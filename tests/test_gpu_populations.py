"""wotg_apply_coupling_f64 with every number of populations (each its own kernel) and
more than one pass holds, on odd shapes, against NumPy FP64: an FP64 sum of n terms in
any order is within n 2^-52 of the sum of their magnitudes."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('k', list(range(1, 18)) + [33])
@pytest.mark.parametrize('I,J', [(1, 1), (37, 65), (300, 97), (65, 1031)])
def test_pull_and_push(I, J, k):
    import torch
    from wot_gb300 import _native as N
    rng = np.random.default_rng(I + J + k)
    X, pj, pi = rng.normal(size=(I, J)), rng.normal(size=(k, J)), rng.normal(size=(k, I))
    Xt = torch.as_tensor(X, device='cuda')
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    for p, transpose, ref, mags, n in ((pj, 1, pj @ X.T, np.abs(pj) @ np.abs(X).T, J),
                                       (pi, 0, pi @ X, np.abs(pi) @ np.abs(X), I)):
        pt = torch.as_tensor(p, device='cuda')
        out = torch.empty(ref.shape, dtype=torch.float64, device='cuda')
        assert N.load().wotg_apply_coupling_f64(Xt.data_ptr(), I, J, pt.data_ptr(), k, transpose, 0, out.data_ptr(),
                                                st) == 0
        assert np.all(np.abs(out.cpu().numpy() - ref) <= (n + 4) * 2.0 ** -52 * mags)
