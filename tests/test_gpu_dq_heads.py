"""dQ of padded head counts, whose rows lie sixteen to a lane quarter: queries split over a cluster, alone on an SM, and two CTAs per SM."""
import pytest
import torch

from test_operator_b200.inputs import Workload, make_sequence
from tests.metrics import assert_backward_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h_q", [8, 16, 24, 40, 48, 56, 64])
@pytest.mark.parametrize("s_q,topk", [(2, 1000), (30, 513), (60, 64), (120, 300)])
def test_heads(h_q, s_q, topk):
    from oracle.sparse_mla_ref import sparse_mla_bwd_ref
    from test_operator_b200 import op
    s = make_sequence(Workload("heads", 1, s_q, 1200, h_q, topk, "uniform", invalid_frac=0.1), device="cuda:0", seed=h_q + s_q)
    args = [s[k] for k in ("q", "kv", "dO", "lse", "O", "indices")]
    args[5][-1] = -1
    dq, dkv = op.mla_bwd(*args, q_start_index_s=None, check_device_status=True)
    assert_backward_close(dq, dkv, *sparse_mla_bwd_ref(*args, q_start_index_s=None))
    assert bool((dq[-1] == 0).all())
