"""The kernel that adds up a query's partial results passes over the parts without a valid slot: many parts of which a few count (in
front, in the middle, at the end, on both sides of the 32 that are looked at together), fewer than are in flight at once, none, and head
counts that fill no warp; against the oracle."""
import pytest
import torch

from oracle.sparse_mla_ref import cosine, sparse_mla_fwd_ref
from test_operator_b200.inputs import LOG2E

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("h_q", [8, 72, 128])
@pytest.mark.parametrize("s_q,topk,tiles", [
    (1, 18944, [0]), (1, 18944, [73]), (1, 18944, [3, 4, 35, 36, 40, 73]), (1, 18944, list(range(74))), (1, 18944, [1, 68]), (1, 18944, []),
    (1, 9217, list(range(37))), (1, 9217, [36]), (2, 9000, [5, 6, 7, 8, 9, 30]), (8, 2048, [7]), (9, 2048, [1, 2, 3, 4, 5]),
    (37, 512, [1]), (2, 30000, list(range(1, 118, 9))), (80, 1030, [4]),
])
def test_parts_that_count(s_q, topk, tiles, h_q):
    from test_operator_b200 import op
    g = torch.Generator(device=DEV).manual_seed(61)
    s_kv = 5000
    q = torch.randn(s_q, h_q, 576, generator=g, device=DEV).bfloat16()
    kv = torch.randn(s_kv, 576, generator=g, device=DEV).bfloat16()
    idx = torch.full((s_q, topk), -1, dtype=torch.int32, device=DEV)
    for t in tiles:
        part = idx[:, 256 * t:256 * t + 256]
        rows = torch.randint(0, s_kv, part.shape, generator=g, device=DEV, dtype=torch.int32)
        part.copy_(torch.where(torch.rand(part.shape, generator=g, device=DEV) < 0.3, -1, rows))
    if s_q > 2 and tiles:
        idx[1] = -1                                    # a query without a valid slot among them
    o_ref, lse_ref = sparse_mla_fwd_ref(q, kv, idx, chunk_s=1)
    o, lse = op.mla_fwd(q, kv, idx, q_start_index_s=None, check_device_status=True)
    empty = (idx < 0).all(dim=1)
    assert torch.all(o[empty] == 0) and torch.equal(torch.isposinf(lse), empty[:, None].expand_as(lse))
    if empty.all():
        return
    # as for the other forward tests: o passes through bf16 twice, lse is fp32
    assert (lse[~empty] - lse_ref[~empty] * LOG2E).abs().max().item() <= 2e-4
    assert (o.float() - o_ref.float()).abs().max().item() <= 2 ** -6 * o_ref.float().abs().max().item()
    assert cosine(o.float().cpu(), o_ref.float().cpu()) > 0.9999
