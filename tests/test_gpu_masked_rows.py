"""Slots that take no part - behind the query's own position, or behind its number of slots in use - may name kv rows that hold NaN or
infinities (rows of a cache that nobody has written): o, lse, dQ and dKV are those of the same call with ordinary rows in their place,
bit for bit where nothing is added up in a varying order.  Masked slots in front of the last valid one, tiles behind it, and queries
without a valid slot; on both sides of the size where the work ranges come from the shape alone (74 clusters on a B200)."""
import pytest
import torch

from oracle.sparse_mla_ref import cosine, sparse_mla_bwd_ref, sparse_mla_fwd_ref
from test_operator_b200.inputs import LOG2E
from tests.metrics import assert_backward_close

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
S_KV, POS, HIDDEN = 1200, 600, 1000          # rows from HIDDEN on lie behind every query's position


def _inputs(s_q, topk, h_q, why):
    g = torch.Generator(device=DEV).manual_seed(41)
    new = lambda *shape: torch.randn(*shape, generator=g, device=DEV).bfloat16()          # noqa: E731
    q, kv, dO = new(s_q, h_q, 576), new(S_KV, 576), new(s_q, h_q, 512)
    idx = torch.randint(0, POS, (s_q, topk), generator=g, device=DEV, dtype=torch.int32)
    hidden = torch.randint(HIDDEN, S_KV, (s_q, topk), generator=g, device=DEV, dtype=torch.int32)
    slots = torch.arange(topk, device=DEV)
    lengths = torch.tensor([(topk, 70, 1, 0)[r % 4] for r in range(s_q)], device=DEV)
    if why == "causal":      # every third slot hidden, all behind slot 70, all behind the first, all
        masked = (slots % 3 == 1) & (lengths[:, None] == topk) | (slots >= lengths[:, None])
        meta = None
    else:                    # by the number of slots in use: the others are in range and in front of the position
        masked = slots >= lengths[:, None]
        meta = torch.tensor([[0, S_KV, S_KV, int(n)] for n in lengths], dtype=torch.int32, device=DEV)
    return q, kv, dO, torch.where(masked, hidden, idx).contiguous(), masked, meta


@pytest.mark.parametrize("why", ["causal", "slots_in_use"])
@pytest.mark.parametrize("value", [float("nan"), float("inf")], ids=["nan", "inf"])
@pytest.mark.parametrize("s_q,topk,h_q", [(8, 600, 16), (9, 2048, 128), (40, 200, 64), (10, 2048, 128), (80, 300, 16), (300, 300, 128)])
def test_hidden_rows_take_no_part(s_q, topk, h_q, value, why):
    from test_operator_b200 import op
    q, kv, dO, idx, masked, meta = _inputs(s_q, topk, h_q, why)
    kw = {"q_start_index_s": POS, "query_meta": meta, "check_device_status": True}
    shown = idx.masked_fill(masked, -1)
    o_ref, lse_ref = sparse_mla_fwd_ref(q, kv, shown)
    o, lse = op.mla_fwd(q, kv, idx, **kw)
    some = torch.isfinite(lse_ref)
    assert (lse[some] - lse_ref[some] * LOG2E).abs().max().item() <= 2e-4           # (the other forward tests' tolerances)
    assert (o.float() - o_ref.float()).abs().max().item() <= 2 ** -6 * o_ref.float().abs().max().item()
    assert cosine(o.float().cpu(), o_ref.float().cpu()) > 0.9999
    dq, dkv = op.mla_bwd(q, kv, dO, lse, o, idx, **kw)
    ref = sparse_mla_bwd_ref(q, kv, dO, lse, o, shown, q_start_index_s=None)
    assert_backward_close(dq, dkv, *ref)

    kv_bad = kv.clone()
    kv_bad[HIDDEN:] = value
    o2, lse2 = op.mla_fwd(q, kv_bad, idx, **kw)
    assert torch.equal(o2, o) and torch.equal(lse2, lse)
    dq2, dkv2 = op.mla_bwd(q, kv_bad, dO, lse, o, idx, **kw)
    assert torch.equal(dq2, dq)
    assert_backward_close(dq2, dkv2, *ref)
    empty = masked.all(dim=1)
    assert torch.all(o2[empty] == 0) and torch.all(dq2[empty] == 0)
