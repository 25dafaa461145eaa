"""The streamed solver where a CTA merges its rows in more than one round of 512 (more
than 77824 rows), and where most CTAs own rows and no column while single rows call for
an absorption (a flag of the barrier that such CTAs reach first): against the FP64
restatement of the reference's solver, absorptions counted."""
import pytest

from parity import assert_parity
from test_gpu_persistent import CFG, _problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('I,J', [(80003, 9), (30001, 44), (20001, 595)])
@pytest.mark.parametrize('tau', [10000, 5, 1.5])
def test_rows_and_absorptions(I, J, tau):
    import torch
    from oracle import torch_ot
    from wot_gb300.ot import device as D
    C, G = _problem(I, J, I)
    cfg = dict(CFG, tau=tau, max_iter=60)
    stats = {}
    ref = torch_ot.optimal_transport_duality_gap(torch.as_tensor(C, device='cuda'), torch.as_tensor(G, device='cuda'),
                                                 stats=stats, **cfg).cpu().numpy()
    got = D.solve(D.cost_from_dense(C), G, cfg, 0)
    assert got.stats['iterations'] == stats['iterations'] and got.stats['absorptions'] == stats['absorptions']
    assert_parity(got.tmap.cpu().numpy(), ref, what=(I, J, tau))
