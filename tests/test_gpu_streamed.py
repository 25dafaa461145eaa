"""The streamed solver kernel against the FP64 restatement of the reference's solver
where its weights do not fit in shared memory (very wide and very tall costs), where
they just do, and with partial float4 chunks and row blocks of one row."""
import numpy as np
import pytest

from parity import assert_parity
from test_gpu_persistent import CFG, _problem, _reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('I,J', [(40, 30001), (30001, 44), (613, 9001), (2049, 3003)])
def test_weights_in_and_out_of_shared_memory(I, J):
    from wot_gb300 import ot
    C, G = _problem(I, J, I)
    cfg = dict(CFG, max_iter=60)
    got, _ = ot.compute_transport_matrix(solver=ot.optimal_transport_duality_gap, C=C, G=G, **cfg)
    assert_parity(got, _reference(C, G, cfg), what=(I, J))
