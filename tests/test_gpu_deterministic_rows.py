"""Reproducible dKV where the segment sum's blocks have no row, one row or many, in one pass and in several of equal size."""
import pytest
import torch

from test_operator_b200.inputs import Workload, make_sequence

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("s_kv", [1, 9, 2368, 2369, 7000])
@pytest.mark.parametrize("s_q,per_pass", [(1, 1), (80, 80), (81, 40), (83, 21)])
def test_rows_and_passes(s_kv, s_q, per_pass):
    from test_operator_b200 import op
    topk = min(300, s_kv)
    s = make_sequence(Workload("rows", 1, s_q, s_kv, 64, topk, "uniform", invalid_frac=0.1), device="cuda:0", seed=s_kv + s_q)
    args = [s[k] for k in ("q", "kv", "dO", "lse", "O", "indices")]
    want = op.mla_bwd(*args, q_start_index_s=None)
    topk_pad = (topk + 255) // 256 * 256
    runs = [op.mla_bwd(*args, q_start_index_s=None, deterministic=True, staging_budget=per_pass * topk_pad * 2304, check_device_status=True)
            for _ in range(3)]
    for dq, dkv in runs:
        assert torch.equal(dq.view(torch.int16), want[0].view(torch.int16))
        assert torch.equal(dkv, runs[0][1])
        assert (dkv - want[1]).abs().max().item() <= 1e-5 * max(want[1].abs().max().item(), 1e-30)
