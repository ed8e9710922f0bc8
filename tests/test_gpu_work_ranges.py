"""The persistent kernels' work ranges (256-key tiles of all queries cut into equal pieces, tiles behind a query's last valid
slot left out) and the dQ kernel's key split, at the sizes where they can go wrong, against the oracle at the parity
tolerances; the per-query table of packed sequences built on the GPU against the one built on the host."""
import pytest
import torch

from oracle.sparse_mla_ref import sparse_mla_bwd_ref
from test_operator_b200.inputs import Workload, make_sequence
from tests.metrics import assert_backward_close

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

CASES = [
    # name, s_q, s_kv, h_q, topk: one query over the whole chip (key split 8), splits of 4 and 2, the last size that is
    # split and the first that is not, a split with fewer key tiles than CTAs
    ("one_query", 1, 2304, 128, 2048),
    ("split_4", 12, 1200, 64, 1100),
    ("split_2", 7, 640, 128, 600),
    ("last_split", 24, 600, 16, 513),
    ("first_whole", 25, 600, 16, 513),
    # more queries than one round of the range search covers, several per cluster and clusters within a query
    ("search_rounds", 1100, 1024, 64, 300),
    ("few_per_cluster", 80, 1024, 128, 1000),
]


@pytest.mark.parametrize("case", CASES, ids=[c[0] for c in CASES])
def test_ranges_with_empty_and_short_queries(case):
    from test_operator_b200 import op
    name, s_q, s_kv, h_q, topk = case
    s = make_sequence(Workload(name, 1, s_q, s_kv, h_q, topk, "uniform", invalid_frac=0.1), device=DEV, seed=51)
    idx = s["indices"]
    # slots in use: everything, a ragged front part, one slot on a tile's edge, nothing - also at both ends and in a row
    for r in range(s_q):
        keep = [topk, (r * 37) % (topk + 1), min(257, topk), 0][r % 4] if s_q > 1 else topk
        idx[r, keep:] = s_kv if r % 2 else -1
    if s_q > 64:
        idx[:3] = -1
        idx[30:60] = s_kv
        idx[-3:] = -1
    args = [s[k] for k in ("q", "kv", "dO", "lse", "O", "indices")]
    ref = sparse_mla_bwd_ref(*args, q_start_index_s=None, chunk_s=16)
    dq, dkv = op.mla_bwd(*args, q_start_index_s=None, check_device_status=True)
    assert_backward_close(dq, dkv, *ref, name)
    empty = (idx < 0).logical_or(idx >= s_kv).all(dim=1)
    assert torch.all(dq[empty] == 0)


def test_early_tokens_of_a_long_causal_prefix():
    """Slots past a query's own position are out of range by the causal rule alone (the indices themselves are in range)."""
    from test_operator_b200 import op
    s = make_sequence(Workload("prefix", 1, 300, 700, 64, 520, "uniform"), device=DEV, seed=52)
    s["indices"] = s["indices"].sort(dim=1).values.contiguous()      # valid slots first
    args = [s[k] for k in ("q", "kv", "dO", "lse", "O", "indices")]
    ref = sparse_mla_bwd_ref(*args, q_start_index_s=0, chunk_s=16)
    dq, dkv = op.mla_bwd(*args, q_start_index_s=0, check_device_status=True)
    assert_backward_close(dq, dkv, *ref, "prefix")


@pytest.mark.parametrize("n_seq", [1, 128, 129, 300])      # one launch of the table kernel covers 128 sequences
def test_query_table_on_the_gpu_equals_the_host_one(n_seq):
    from test_operator_b200 import op
    g = torch.Generator().manual_seed(n_seq)
    lens = torch.randint(0, 9, (n_seq,), generator=g).tolist()
    lens[0] += 1
    kv_lens = torch.randint(1, 50, (n_seq,), generator=g).tolist()
    q0 = [sum(lens[:i]) for i in range(n_seq)]
    kv0 = [sum(kv_lens[:i]) for i in range(n_seq)]
    used = torch.randint(-3, 90, (sum(lens),), generator=g)
    for q_start, length in ((0, None), (17, used), (None, used)):
        want = op.query_meta_for(q0, lens, kv0, kv_lens, "cpu", q_start, 64, length)
        got = op.query_meta_for(q0, lens, kv0, kv_lens, DEV, q_start, 64, None if length is None else length.to(DEV))
        assert torch.equal(got.cpu(), want)


@pytest.mark.parametrize("q0,lens,kv0,kv_lens", [
    ([-100], [28], [0], [300]),                              # the shard of a sequence that begins 100 queries earlier
    ([5, 8], [3, 4], [0, 40], [40, 50]),                     # rows counted from elsewhere
    ([0, 3, 7], [3, 4], [0, 40, 90], [40, 50, 0]),           # offsets with the end behind them, as cu_seqlens are
    (torch.tensor([0, 3]), torch.tensor([3, 4]), torch.tensor([0, 40]), torch.tensor([40, 50])),
    ([0, 0], [0, 0], [0, 0], [1, 1]),
])
def test_query_table_of_other_forms_equals_the_host_one(q0, lens, kv0, kv_lens):
    from test_operator_b200 import op
    want = op.query_meta_for(q0, lens, kv0, kv_lens, "cpu", 7, 64)
    got = op.query_meta_for(q0, lens, kv0, kv_lens, DEV, 7, 64)
    assert got.is_cuda and torch.equal(got.cpu(), want)


def test_query_table_refuses_what_the_host_one_refuses():
    from test_operator_b200 import op
    for bad in (dict(kv_lens=[40]), dict(kv0=[0, 1 << 31]), dict(lens=[3, -4])):
        args = {**dict(q0=[0, 3], lens=[3, 4], kv0=[0, 40], kv_lens=[40, 50]), **bad}
        for device in ("cpu", DEV):
            with pytest.raises((RuntimeError, IndexError, ValueError)):
                op.query_meta_for(*args.values(), device, 0, 64)


# the last slot in use on, before and behind the edges of what is worked on as one: 32 keys (a drain warp's registers), 64 (a dQ
# tile), 128 (a dKV tile, one CTA's half of a work tile), 256 (a work tile)
EDGES = [1, 31, 32, 33, 63, 64, 65, 96, 97, 127, 128, 129, 160, 161, 255, 256, 257, 384, 385, 500]


@pytest.mark.parametrize("h_q", [16, 64, 128])
@pytest.mark.parametrize("deterministic", [False, True])
def test_last_slot_at_the_edges_of_the_key_groups(h_q, deterministic):
    """What lies behind a query's last slot is neither computed nor added: a call with every slot in use leaves the scratch full
    of other values first."""
    from test_operator_b200 import op
    s = make_sequence(Workload("edges", 1, 4 * len(EDGES), 900, h_q, 500, "uniform"), device=DEV, seed=53)
    full = [s[k] for k in ("q", "kv", "dO", "lse", "O", "indices")]
    op.mla_bwd(*full, q_start_index_s=None, deterministic=deterministic, check_device_status=True)
    s["indices"] = s["indices"].clone()
    for r in range(s["indices"].shape[0]):
        s["indices"][r, EDGES[r % len(EDGES)]:] = -1
    args = [s[k] for k in ("q", "kv", "dO", "lse", "O", "indices")]
    ref = sparse_mla_bwd_ref(*args, q_start_index_s=None, chunk_s=16)
    dq, dkv = op.mla_bwd(*args, q_start_index_s=None, deterministic=deterministic, check_device_status=True)
    assert_backward_close(dq, dkv, *ref, "edges")
