"""The one-pass forward kernel at the sizes where it can go wrong: a query over many clusters (partial results added up),
tiles of one to 256 keys, several queries per cluster, queries without a valid slot, logits that outgrow the softmax
reference from tile to tile.  Against the oracle (fp32 on the GPU)."""
import pytest
import torch

from oracle.sparse_mla_ref import cosine, sparse_mla_fwd_ref
from test_operator_b200.inputs import LOG2E, Workload, make_sequence

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

CASES = [
    # name, s_q, s_kv, h_q, topk, factor on q
    ("one_query_all_clusters", 1, 40000, 128, 20000, 1.0),
    ("one_query_64_heads", 1, 4096, 64, 2048, 1.0),
    ("one_key", 1, 64, 128, 1, 1.0),
    ("tile_plus_one", 3, 600, 128, 257, 1.0),
    ("tile_exact", 3, 600, 16, 256, 1.0),
    ("ragged_8_heads", 5, 900, 8, 777, 1.0),
    ("padded_heads", 7, 600, 72, 300, 1.0),
    ("ranges_inside_queries", 80, 1200, 128, 1000, 1.0),
    ("many_queries_per_cluster", 700, 700, 64, 300, 1.0),
    # scaled logits of standard deviation 20: the reference of the exponentials moves several times in a query
    ("growing_logits_128", 40, 3000, 128, 2048, 20.0),
    ("growing_logits_64", 90, 3000, 64, 1030, 20.0),
]


@pytest.mark.parametrize("case", CASES, ids=[c[0] for c in CASES])
def test_forward_ranges(case):
    from test_operator_b200 import op
    name, s_q, s_kv, h_q, topk, factor = case
    s = make_sequence(Workload(name, 1, s_q, s_kv, h_q, topk, "uniform", invalid_frac=0.1 if topk > 1 else 0.0), device=DEV,
                      seed=61, with_forward=False)
    q, kv, idx = s["q"], s["kv"], s["indices"]
    if factor != 1.0:
        q = (q.float() * factor).bfloat16()
        # the largest logits of the first heads last, so that every tile exceeds the ones before it
        p = torch.einsum("sd,std->st", q[:, 0].float(), kv[idx.clamp(0).long()].float())
        idx = idx.gather(1, p.argsort(dim=1)).contiguous()
    if s_q > 2:
        for r in range(s_q):
            idx[r, [topk, (r * 53) % (topk + 1), min(257, topk), 0][r % 4]:] = s_kv if r % 2 else -1
    o_ref, lse_ref = sparse_mla_fwd_ref(q, kv, idx, q_start_index_s=None)
    runs = [op.mla_fwd(q, kv, idx, q_start_index_s=None, check_device_status=True) for _ in range(3)]
    o, lse = runs[0]
    for o2, lse2 in runs[1:]:
        assert torch.equal(o.view(torch.int16), o2.view(torch.int16)) and torch.equal(lse.view(torch.int32), lse2.view(torch.int32))
    fin = torch.isfinite(lse_ref)
    assert torch.equal(torch.isposinf(lse), ~fin)
    # 2e-4 as elsewhere for logits of order one; an fp32 dot product of 576 terms may be off by 576 * 2^-24 of the sum of
    # its terms' sizes, which grows with the factor (|q| |k| of 0.8 each on average, scaled by 1/24 and log2 e)
    atol = 2e-4 + (576 * 2.0 ** -24 * 576 * 0.64 * factor / 24 * LOG2E if factor != 1.0 else 0.0)
    assert (lse[fin] - lse_ref[fin] * LOG2E).abs().max().item() <= atol
    assert (o.float() - o_ref.float()).abs().max().item() <= 2 ** -6 * o_ref.float().abs().max().item()
    assert cosine(o.float().cpu(), o_ref.float().cpu()) > 0.9999
    empty = ((idx < 0) | (idx >= s_kv)).all(dim=1)
    assert torch.all(o[empty] == 0)


def test_forward_with_a_workspace_too_small_to_spread_queries():
    """Without room for partial results one cluster takes every query whole; the results stay within the tolerances."""
    from test_operator_b200 import op
    s = make_sequence(Workload("small_ws", 1, 9, 700, 64, 600, "uniform", invalid_frac=0.1), device=DEV, seed=62, with_forward=False)
    args = (s["q"], s["kv"], s["indices"])
    o_ref, lse_ref = sparse_mla_fwd_ref(*args, q_start_index_s=None)
    o, lse = op.mla_fwd(*args, q_start_index_s=None, workspace_budget=4096, check_device_status=True)
    assert (lse - lse_ref * LOG2E).abs().max().item() <= 2e-4
    assert (o.float() - o_ref.float()).abs().max().item() <= 2 ** -6 * o_ref.float().abs().max().item()


@pytest.mark.parametrize("h_q", [64, 128])
def test_the_heaviest_slot_enters_unrounded(h_q):
    """All rows of V are equal, so o / V is the sum of the weights.  The heaviest slot of the first tile and a heavier one (by 2^1.2
    to 2^6.6) in the third enter as exactly 1 of their tile's maximum and are only scaled in fp32 afterwards; the other 698
    slots weigh 2^-30 each.  So the sum is 1 to a few 2^-24, far from half a bf16 step, and o must be V bit for bit."""
    from test_operator_b200 import op
    s_q, topk, s_kv = 90, 700, 1024
    g = torch.Generator(device=DEV).manual_seed(64)
    kv = torch.zeros(s_kv, 576, device=DEV)
    kv[:, :512] = torch.randn(512, generator=g, device=DEV)
    kv[:, 512] = -500.0                                                     # times log2 e / 24 in the exponent
    kv[:129, 512] = torch.arange(129, device=DEV).float()
    kv = kv.bfloat16()
    q = torch.zeros(s_q, h_q, 576, dtype=torch.bfloat16, device=DEV)
    q[:, :, 512] = 1.0
    idx = torch.arange(200, 200 + topk, device=DEV, dtype=torch.int32).repeat(s_q, 1)
    idx[:, 5] = 0
    idx[:, 600] = torch.arange(s_q, device=DEV, dtype=torch.int32) + 20
    o, _ = op.mla_fwd(q, kv, idx, q_start_index_s=None, check_device_status=True)
    assert torch.equal(o.view(torch.int16), kv[0, :512].expand_as(o).contiguous().view(torch.int16))
