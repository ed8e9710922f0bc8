"""dKV ranges of 128-key tiles: queries with an odd number of them, few queries over many clusters, empty queries between, range borders
inside queries."""
import pytest
import torch

from test_operator_b200.inputs import Workload, make_sequence
from tests.metrics import assert_backward_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h_q", [64, 128])
@pytest.mark.parametrize("s_q,topk", [(1, 129), (1, 2000), (3, 1000), (74, 256), (75, 257), (200, 640)])
@pytest.mark.parametrize("used", ["all", "mixed"])
def test_ranges(h_q, s_q, topk, used):
    from oracle.sparse_mla_ref import sparse_mla_bwd_ref
    from test_operator_b200 import op
    s = make_sequence(Workload("ranges", 1, s_q, 2500, h_q, topk, "uniform", invalid_frac=0.0), device="cuda:0", seed=s_q + topk)
    args = [s[k] for k in ("q", "kv", "dO", "lse", "O", "indices")]
    if used == "mixed":             # 0, 1, 128, 129, 256, 257 slots in use in turn
        for i, n in enumerate((0, 1, 128, 129, 256, 257)):
            args[5][i::6, n:] = -1
    dq, dkv = op.mla_bwd(*args, q_start_index_s=None, check_device_status=True)
    assert_backward_close(dq, dkv, *sparse_mla_bwd_ref(*args, q_start_index_s=None))
