"""Calls with at most one tile of 256 slots per cluster: work ranges from the shape alone, no look at the indices first.  Around
the size where that form ends (74 clusters on a B200), with queries and whole tiles that have no valid slot, against the oracle."""
import pytest
import torch

from oracle.sparse_mla_ref import cosine, sparse_mla_bwd_ref, sparse_mla_fwd_ref
from test_operator_b200.inputs import LOG2E, Workload, make_sequence
from tests.metrics import assert_backward_close

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

# (s_q, topk): one tile of one query; 74 and 75 tiles of one; 37 and 38 queries of two; eight tiles a query; one query of 74 and 75
SIZES = [(1, 1), (1, 256), (74, 200), (75, 200), (37, 300), (38, 300), (9, 2048), (10, 2048), (1, 74 * 256), (1, 74 * 256 + 1)]


def _inputs(s_q, topk, h_q, holes):
    s_kv = 40000 if topk == 3 else max(2 * topk, 64)       # (a large dKV to clear beside a single tile)
    s = make_sequence(Workload("every_slot", 1, s_q, s_kv, h_q, topk, "uniform", invalid_frac=0.0), device=DEV, seed=17)
    idx = s["indices"]
    if holes:
        for r in range(s_q):        # nothing at all / nothing in front of slot 256 / nothing behind it / as it is
            idx[r, [0, 0, 256, topk][r % 4]:[topk, 256, topk, topk][r % 4]] = -1 if r % 2 else s_kv
    return s, idx, s_kv


@pytest.mark.parametrize("holes", [False, True], ids=["full", "holes"])
@pytest.mark.parametrize("h_q", [16, 128])
@pytest.mark.parametrize("s_q,topk", SIZES)
def test_forward(s_q, topk, h_q, holes):
    from test_operator_b200 import op
    s, idx, s_kv = _inputs(s_q, topk, h_q, holes)
    o_ref, lse_ref = sparse_mla_fwd_ref(s["q"], s["kv"], idx, q_start_index_s=None)
    o, lse = op.mla_fwd(s["q"], s["kv"], idx, q_start_index_s=None, check_device_status=True)
    empty = ((idx < 0) | (idx >= s_kv)).all(dim=1)
    assert torch.all(o[empty] == 0) and torch.equal(torch.isposinf(lse), empty[:, None].expand_as(lse))
    if empty.all():
        return
    fin = ~empty
    # as for the other forward tests: o passes through bf16 twice, lse is fp32
    assert (lse[fin] - lse_ref[fin] * LOG2E).abs().max().item() <= 2e-4
    assert (o.float() - o_ref.float()).abs().max().item() <= 2 ** -6 * o_ref.float().abs().max().item()
    assert cosine(o.float().cpu(), o_ref.float().cpu()) > 0.9999


def test_forward_logits_of_minus_infinity():
    """A query whose valid slots all have logits of -inf is not one without a valid slot: o NaN, lse -inf, as in plain torch."""
    from test_operator_b200 import op
    s, idx, _ = _inputs(4, 600, 16, False)
    q, kv = s["q"].clone(), s["kv"].clone()
    q[..., 0] = 1.0
    kv[:, 0] = float("-inf")
    idx[1] = -1
    o, lse = op.mla_fwd(q, kv, idx, q_start_index_s=None, check_device_status=True)
    assert torch.all(torch.isneginf(lse[[0, 2, 3]])) and torch.all(torch.isnan(o[[0, 2, 3], :, 0].float()))
    assert torch.all(torch.isposinf(lse[1])) and torch.all(o[1] == 0)


@pytest.mark.parametrize("holes", [False, True], ids=["full", "holes"])
@pytest.mark.parametrize("h_q", [16, 128])
# (not one slot a query: its softmax is constant, dP - Delta is 0 up to the rounding of two sums, and so is all of dQ)
@pytest.mark.parametrize("s_q,topk", [(1, 3)] + SIZES[1:])
def test_backward(s_q, topk, h_q, holes):
    from test_operator_b200 import op
    s, idx, s_kv = _inputs(s_q, topk, h_q, holes)
    args = (s["q"], s["kv"], s["dO"], s["lse"], s["O"], idx)
    ref = sparse_mla_bwd_ref(*args, q_start_index_s=None, chunk_s=16)
    dkv_dirty = torch.full((s_kv, 576), 7.0, device=DEV)          # cleared beside the kernel that computes S and dS
    for out_dkv in (None, dkv_dirty):
        dq, dkv = op.mla_bwd(*args, q_start_index_s=None, check_device_status=True, out_dkv=out_dkv)
        assert_backward_close(dq, dkv, *ref)
    dkv2 = torch.ones_like(dkv)
    op.mla_bwd(*args, q_start_index_s=None, out_dkv=dkv2, accumulate=True)
    # added to ones: rounded to 2^-24 of the sum's size at every addition
    assert (dkv2 - 1 - dkv).abs().max().item() <= (dkv.abs().max().item() + 1) * 2.0 ** -24 * (s_q + 2) * 2
    unused = torch.ones(s_kv, dtype=torch.bool, device=DEV)
    unused[idx[(idx >= 0) & (idx < s_kv)].long()] = False
    assert torch.all(dkv[unused] == 0) and torch.all(dq[((idx < 0) | (idx >= s_kv)).all(dim=1)] == 0)
