"""The dQ kernel around the sizes where it changes between one CTA per SM with many stages and two with few (148 SMs on a B200,
three CTAs a query): 49 queries against 50, one work tile against two, and fewer key tiles than stages; against the oracle."""
import pytest
import torch

from oracle.sparse_mla_ref import sparse_mla_bwd_ref
from test_operator_b200.inputs import Workload, make_sequence
from tests.metrics import assert_backward_close

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("h_q", [64, 128])
@pytest.mark.parametrize("s_q,topk", [(49, 256), (49, 257), (50, 257), (49, 700), (30, 330)])
def test_dq_around_the_change(s_q, topk, h_q):
    from test_operator_b200 import op
    s = make_sequence(Workload("stages", 1, s_q, 2 * topk, h_q, topk, "uniform", invalid_frac=0.1), device=DEV, seed=23)
    for r in range(s_q):                     # all slots, a ragged front part, one slot, none
        s["indices"][r, [topk, (r * 37) % topk, 1, 0][r % 4]:] = -1
    args = [s[k] for k in ("q", "kv", "dO", "lse", "O", "indices")]
    ref = sparse_mla_bwd_ref(*args, q_start_index_s=None, chunk_s=16)
    runs = [op.mla_bwd(*args, q_start_index_s=None, check_device_status=True) for _ in range(2)]
    assert_backward_close(*runs[0], *ref)
    assert torch.equal(runs[0][0].view(torch.int16), runs[1][0].view(torch.int16))
