"""wotg_gemm_f64 with the product written over its left operand (up to 64 columns, a
row tile is read before it is written), and over a right operand of one row tile. Bound:
an FP64 sum of n terms in any order is within n 2^-52 of the sum of their magnitudes."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('M,r', [(1, 1), (64, 64), (257, 40), (4500, 33), (40000, 64)])
def test_over_the_left_operand(M, r):
    import torch
    from wot_gb300 import _native as N
    rng = np.random.default_rng(M + r)
    A, B = rng.normal(size=(M, r)), rng.normal(size=(r, r))
    At, Bt = torch.as_tensor(A, device='cuda'), torch.as_tensor(B, device='cuda')
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert N.load().wotg_gemm_f64(At.data_ptr(), r, Bt.data_ptr(), r, None, At.data_ptr(), r, M, r, r, st) == 0
    assert np.all(np.abs(At.cpu().numpy() - A @ B) <= (r + 4) * 2.0 ** -52 * (np.abs(A) @ np.abs(B)))


@pytest.mark.parametrize('r', [1, 40, 64])
def test_over_the_right_operand(r):
    import torch
    from wot_gb300 import _native as N
    rng = np.random.default_rng(r)
    A, B = rng.normal(size=(r, r)), rng.normal(size=(r, r))
    At, Bt = torch.as_tensor(A, device='cuda'), torch.as_tensor(B, device='cuda')
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert N.load().wotg_gemm_f64(At.data_ptr(), r, Bt.data_ptr(), r, None, Bt.data_ptr(), r, r, r, r, st) == 0
    assert np.all(np.abs(Bt.cpu().numpy() - A @ B) <= (r + 4) * 2.0 ** -52 * (np.abs(A) @ np.abs(B)))
