"""The persistent solver kernels on a materialised cost against the FP64
restatement of the reference's solver, at the sizes where their partitions can
go wrong: one row block or column per CTA and fewer, float4 tails, CTAs with two
row blocks, merges of more than 64 and 128 row blocks, costs just too large for
shared memory (the streamed kernel), absorptions, weights and offsets beyond
+-1024 (the FP64 branches), and more iterations than one launch runs."""
import numpy as np
import pytest

from parity import COUPLING_TOL, ELEMENT_TOL, assert_parity, errors

pytestmark = pytest.mark.gpu

CFG = dict(growth_iters=1, epsilon=0.05, lambda1=1, lambda2=50, epsilon0=1, tau=10000, scaling_iter=3000,
           inner_iter_max=50, tolerance=1e-8, max_iter=1e7, batch_size=5, extra_iter=1000)


def _problem(I, J, seed):
    rng = np.random.default_rng(seed)
    x = rng.normal(size=(I, 4)) + rng.integers(0, 3, size=(I, 1))
    y = rng.normal(size=(J, 4)) + rng.integers(0, 3, size=(J, 1)) + 0.2
    C = ((x * x).sum(1)[:, None] + (y * y).sum(1)[None, :] - 2 * x @ y.T).clip(0)
    return C / np.median(C), rng.lognormal(0, 0.3, I)


def _reference(C, G, cfg):
    import torch
    from oracle import torch_ot
    T = torch_ot.optimal_transport_duality_gap(torch.as_tensor(C, device='cuda'), torch.as_tensor(G, device='cuda'),
                                               **cfg)
    return T.cpu().numpy()


@pytest.mark.parametrize('I,J', [(2, 3), (5, 130), (130, 5), (13, 33), (161, 1027), (1100, 517), (1601, 50),
                                 (2500, 700), (1200, 5001)])
def test_sizes(I, J):
    from wot_gb300 import ot
    C, G = _problem(I, J, I + J)
    got, _ = ot.compute_transport_matrix(solver=ot.optimal_transport_duality_gap, C=C, G=G, **CFG)
    assert_parity(got, _reference(C, G, CFG), what=(I, J))


@pytest.mark.parametrize('over', [dict(tau=5), dict(epsilon=0.01, lambda1=10), dict(batch_size=1, max_iter=23),
                                  dict(lambda1=0.1, epsilon=0.1, epsilon0=3)])
@pytest.mark.parametrize('shape', [(230, 311), (1203, 4907)])
def test_options(shape, over):
    from wot_gb300 import ot
    cfg = dict(CFG, **over)
    C, G = _problem(*shape, seed=7)
    got, _ = ot.compute_transport_matrix(solver=ot.optimal_transport_duality_gap, C=C, G=G, **cfg)
    assert_parity(got, _reference(C, G, cfg), what=(shape, over))


@pytest.mark.parametrize('shape', [(90, 121), (1203, 4907)])
def test_far_weights(shape):
    """Exponents of several thousand (a small epsilon): the FP32 storage of C puts
    about max(C) / eps 2^-24 on an entry, and the potentials carry as much again."""
    from wot_gb300 import ot
    cfg = dict(CFG, epsilon=0.002, max_iter=1200)
    C, G = _problem(*shape, seed=3)
    assert C.max() / 0.002 * 1.45 > 2048
    got, _ = ot.compute_transport_matrix(solver=ot.optimal_transport_duality_gap, C=C, G=G, **cfg)
    e = errors(got, _reference(C, G, cfg))
    tol = 2 * C.max() / 0.002 * 2.0 ** -24
    assert e['coupling_max_rel_err'] <= max(COUPLING_TOL, tol), e
    assert e['element_max_rel_err'] <= max(ELEMENT_TOL, tol), e
