"""The forward's second contraction goes over groups of 64 keys up to a query's last slot in use: at the edges of the groups, with
queries of different lengths next to one another in a cluster, and with values beyond that slot that must take no part."""
import pytest
import torch

from oracle.sparse_mla_ref import cosine, sparse_mla_fwd_ref
from test_operator_b200.inputs import LOG2E, Workload, make_sequence

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("h_q", [64, 128])
@pytest.mark.parametrize("topk", [64, 300, 512])
def test_last_slot_at_the_edges_of_the_groups(h_q, topk):
    from test_operator_b200 import op
    s_q, s_kv = 300, 2048                      # several queries a cluster
    s = make_sequence(Workload("groups", 1, s_q, s_kv, h_q, topk, "uniform", invalid_frac=0.1), device=DEV, seed=31, with_forward=False)
    q, kv, idx = s["q"], s["kv"], s["indices"]
    kv[-1] = float("nan")                      # named by slots that the causal rule masks
    start = s_kv - 400
    idx[idx > start] = 0
    last = [n for n in (1, 63, 64, 65, 128, 129, 192, 193, 256, 257, 320, 321, 449, 512) if n <= topk]
    for r in range(s_q):
        idx[r, last[r % len(last)] - 1] = r    # the last slot in use is a valid one
        idx[r, last[r % len(last)]:] = -1 if r % 2 else s_kv - 1
    o_ref, lse_ref = sparse_mla_fwd_ref(q, torch.nan_to_num(kv), idx, q_start_index_s=start)
    o, lse = op.mla_fwd(q, kv, idx, q_start_index_s=start, check_device_status=True)
    assert (lse - lse_ref * LOG2E).abs().max().item() <= 2e-4
    assert (o.float() - o_ref.float()).abs().max().item() <= 2 ** -6 * o_ref.float().abs().max().item()
    assert cosine(o.float().cpu(), o_ref.float().cpu()) > 0.9999
