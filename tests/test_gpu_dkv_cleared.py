"""dKV is cleared inside the kernel that computes S and dS, every block its share: rows that no slot names come back as +0 whatever
the buffer held, for shares of a few bytes and of many copies, for several queries per cluster, clusters without a tile and calls
without a valid slot; with several passes it is cleared once."""
import pytest
import torch

from oracle.sparse_mla_ref import sparse_mla_bwd_ref
from test_operator_b200.inputs import Workload, make_sequence
from tests.metrics import assert_backward_close

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("s_q,s_kv,h_q,topk,empty", [
    (3, 5, 16, 4, False),              # 80 pieces of 16 bytes a block
    (90, 997, 128, 520, False),        # three tiles a query, queries cut over clusters
    (400, 30001, 64, 100, False),      # five queries a cluster, 467 KB a block
    (2, 50000, 128, 300, False),       # more blocks than the tiles need
    (100, 3001, 64, 300, True),        # no valid slot at all
])
def test_unnamed_rows_are_zero(s_q, s_kv, h_q, topk, empty):
    from test_operator_b200 import op
    s = make_sequence(Workload("cleared", 1, s_q, s_kv, h_q, topk, "uniform", invalid_frac=0.1), device=DEV, seed=29)
    idx = s["indices"]
    if empty:
        idx.fill_(-1)
    args = [s[k] for k in ("q", "kv", "dO", "lse", "O")] + [idx]
    dkv = torch.full((s_kv, 576), float("nan"), device=DEV)
    dq, out = op.mla_bwd(*args, q_start_index_s=None, out_dkv=dkv, check_device_status=True)
    named = torch.zeros(s_kv, dtype=torch.bool, device=DEV)
    named[idx[(idx >= 0) & (idx < s_kv)].long()] = True
    assert torch.all(out.view(torch.int32)[~named] == 0)
    if empty:
        assert torch.all(dq == 0)
        return
    ref = sparse_mla_bwd_ref(*args, q_start_index_s=None, chunk_s=16)
    assert_backward_close(dq, out, *ref)
    # two or more passes over the queries
    per_pass = 4 * 256 * ((topk + 255) // 256) * (64 if h_q <= 64 else 128)
    dkv.fill_(float("nan"))
    dq2, out2 = op.mla_bwd(*args, q_start_index_s=None, out_dkv=dkv, workspace_budget=per_pass * max(1, s_q // 2) + (s_q * (h_q + 1) * 4 + 2048))
    assert_backward_close(dq2, out2, *ref)
