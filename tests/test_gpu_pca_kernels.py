"""The FP64 kernels of the PCA against NumPy at the widths and lengths where their
partitions change: one column, 32 and 64 columns, one row block and several, rows
short and long enough for a CTA each, narrow products up to their limit and past it.
Bounds: an FP64 sum of n terms in any order is within n 2^-52 of the sum of their
magnitudes."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _stream():
    import torch
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def _near(got, ref, mags, terms):
    assert np.all(np.abs(got - ref) <= (terms + 4) * 2.0 ** -52 * mags)


@pytest.mark.parametrize('r', [1, 31, 32, 33, 40, 64])
@pytest.mark.parametrize('n', [1, 31, 257, 4500])
def test_gram_vecmat_narrow_gemm(n, r):
    import torch
    from wot_gb300 import _native as N
    from wot_gb300.ot import util
    rng = np.random.default_rng(n + r)
    A, w, B = rng.normal(size=(n, r)), rng.normal(size=n), rng.normal(size=(r, r))
    At, wt, Bt = (torch.as_tensor(v, device='cuda') for v in (A, w, B))
    lib = N.load()
    G = torch.empty((r, r), dtype=torch.float64, device='cuda')
    ws = torch.empty(lib.wotg_gram_workspace_bytes(n, r), dtype=torch.uint8, device='cuda')
    assert lib.wotg_gram_f64(At.data_ptr(), n, r, G.data_ptr(), ws.data_ptr(), ws.numel(), _stream()) == 0
    _near(G.cpu().numpy(), A.T @ A, np.abs(A).T @ np.abs(A), n)
    assert torch.equal(G, G.T)
    _near(util.vec_mat(wt, At).cpu().numpy(), w @ A, np.abs(w) @ np.abs(A), n)
    _near(util.mat_mul(At, Bt).cpu().numpy(), A @ B, np.abs(A) @ np.abs(B), r)


@pytest.mark.parametrize('M,K,Nc', [(1, 1, 1), (130, 64, 64), (65, 65, 64), (65, 64, 65), (7, 3, 61)])
def test_gemm_on_both_sides_of_narrow(M, K, Nc):
    import torch
    from wot_gb300.ot import util
    rng = np.random.default_rng(M + K + Nc)
    A, B = rng.normal(size=(M, K)), rng.normal(size=(K, Nc))
    got = util.mat_mul(torch.as_tensor(A, device='cuda'), torch.as_tensor(B, device='cuda')).cpu().numpy()
    _near(got, A @ B, np.abs(A) @ np.abs(B), K)


@pytest.mark.parametrize('n,p,density', [(5, 700, 0.9), (300, 90, 0.3), (1, 33, 1.0)])
@pytest.mark.parametrize('r', [1, 33, 40])
def test_spmm(n, p, density, r):
    import torch
    from wot_gb300 import _native as N
    rng = np.random.default_rng(n + p)
    X = rng.normal(size=(n, p)) * (rng.random((n, p)) < density)
    counts = np.concatenate([[0], np.cumsum((X != 0).sum(1))])
    Q, a, b, c = rng.normal(size=(p, r)), rng.normal(size=r), rng.normal(size=r), rng.normal(size=n)
    rows, cols = np.nonzero(X)
    t = [torch.as_tensor(v, device='cuda') for v in
         (counts.astype(np.int64), cols.astype(np.int32), X[rows, cols], Q, a, c, b)]
    Y = torch.empty((n, r), dtype=torch.float64, device='cuda')
    assert N.load().wotg_spmm_centred(t[0].data_ptr(), t[1].data_ptr(), t[2].data_ptr(), n, t[3].data_ptr(), r,
                                      t[4].data_ptr(), t[5].data_ptr(), t[6].data_ptr(), Y.data_ptr(), _stream()) == 0
    ref = X @ Q - a[None, :] - np.outer(c, b)
    _near(Y.cpu().numpy(), ref, np.abs(X) @ np.abs(Q) + np.abs(a)[None, :] + np.abs(np.outer(c, b)), p)
