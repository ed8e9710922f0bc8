"""The index inverse without a sort, bit for bit against the oracle: groups of one and of several queries, queries shorter and longer than a
batch, the largest number of rows, and queries that name rows more than once."""
import numpy as np
import pytest
import torch

from oracle.index_inverse_ref import index_inverse_ref

pytestmark = pytest.mark.gpu

CASES = [
    # s_q, topk, s_kv, causal start
    (5, 2048, 8192, None),        # a query a group, one unfinished batch
    (148, 1500, 3001, 2000),      # as many groups as there may be
    (149, 1501, 3001, 2000),      # two queries a group, an odd top-k, the last group with one
    (1040, 1365, 5000, None),     # eight queries a group
    (450, 8192, 9000, None),      # queries of more than a batch
    (300, 8193, 9000, 8800),      # one slot more
    (700, 2047, 30000, None),
    (4096, 2048, 53243, None),    # the most rows
    (600, 1024, 7, None),         # every query names every row many times
]


def repeats(idx, g):
    few = g.random(idx.shape) < 0.02
    idx[few] = idx[:, ::-1][few]
    return idx


PATTERNS = {
    "distinct": lambda idx, s_kv, g: idx,
    "unused": lambda idx, s_kv, g: np.where(g.random(idx.shape) < 0.4, -1, idx),
    "few_repeats": lambda idx, s_kv, g: repeats(idx, g),
    "half_one_row": lambda idx, s_kv, g: np.where(np.arange(idx.shape[1]) * 2 < idx.shape[1], idx, s_kv // 3),
    "two_rows": lambda idx, s_kv, g: 0 * idx + np.where(np.arange(idx.shape[1]) % 2 == 0, s_kv // 2, s_kv - 1),
    "random": lambda idx, s_kv, g: g.integers(-1, s_kv + 1, size=idx.shape),
}


@pytest.mark.parametrize("s_q,topk,s_kv,q_start", CASES)
@pytest.mark.parametrize("pattern", PATTERNS)
def test_direct_form(s_q, topk, s_kv, q_start, pattern):
    from test_operator_b200 import op
    g = np.random.default_rng(s_q + topk)
    base = np.stack([g.permutation(max(s_kv, topk))[:topk] for _ in range(8)])[g.integers(0, 8, s_q)]
    idx = ((base + g.integers(0, s_kv, (s_q, 1))) % max(s_kv, topk)).astype(np.int64)
    idx = np.ascontiguousarray(PATTERNS[pattern](idx, s_kv, g).astype(np.int32))
    row_ptr, entries = op.index_inverse(torch.from_numpy(idx).cuda(), s_kv, q_start_index_s=q_start)
    ref_ptr, ref_entries = index_inverse_ref(idx, s_kv, q_start)
    assert np.array_equal(row_ptr.cpu().numpy(), ref_ptr)
    assert np.array_equal(entries.cpu().numpy(), ref_entries)


def test_a_workspace_for_the_sort_only_is_enough():
    """A caller's workspace that holds the sort but not the counters gets the sort."""
    from test_operator_b200 import op
    lib = op.load_library()
    s_q, topk, s_kv = 5, 2048, 20000
    idx = torch.randint(-1, s_kv, (s_q, topk), dtype=torch.int32, device="cuda")
    row_ptr = torch.empty(s_kv + 1, dtype=torch.int32, device="cuda")
    entries = torch.empty(s_q * topk, dtype=torch.int32, device="cuda")
    whole = lib.smla_index_inverse_workspace_size(s_q, topk, s_kv)
    counters = s_q * (s_kv + 4) * 4
    ws = torch.empty(whole, dtype=torch.uint8, device="cuda")
    for n_bytes in (whole, counters - 1024):
        entries.fill_(-7)
        rc = lib.smla_index_inverse(idx.data_ptr(), s_q, topk, s_kv, op.NO_CAUSAL,
                                    row_ptr.data_ptr(), entries.data_ptr(), ws.data_ptr(),
                                    n_bytes, torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        assert rc == 0
        ref_ptr, ref_entries = index_inverse_ref(idx.cpu().numpy(), s_kv, None)
        assert np.array_equal(row_ptr.cpu().numpy(), ref_ptr) and np.array_equal(entries.cpu().numpy(), ref_entries)


@pytest.mark.parametrize("at_in,at_out", [(0, 1), (1, 0), (2, 3), (3, 3)])
@pytest.mark.parametrize("topk", [1500, 1501])
def test_buffers_off_a_16_byte_boundary(at_in, at_out, topk):
    from test_operator_b200 import op
    lib = op.load_library()
    s_q, s_kv = 300, 4000
    flat = torch.randint(-1, s_kv, (s_q * topk + 8,), dtype=torch.int32, device="cuda")
    idx = flat[at_in:at_in + s_q * topk].view(s_q, topk)
    out = torch.full((s_q * topk + 8,), -7, dtype=torch.int32, device="cuda")
    row_ptr = torch.empty(s_kv + 1, dtype=torch.int32, device="cuda")
    ws = torch.empty(lib.smla_index_inverse_workspace_size(s_q, topk, s_kv), dtype=torch.uint8, device="cuda")
    assert lib.smla_index_inverse(idx.data_ptr(), s_q, topk, s_kv, op.NO_CAUSAL, row_ptr.data_ptr(), out.data_ptr() + 4 * at_out, ws.data_ptr(),
                                  ws.numel(), torch.cuda.current_stream().cuda_stream) == 0
    ref_ptr, ref_entries = index_inverse_ref(idx.cpu().numpy(), s_kv, None)
    got = out.cpu().numpy()
    assert np.array_equal(row_ptr.cpu().numpy(), ref_ptr) and np.array_equal(got[at_out:at_out + s_q * topk], ref_entries)
    assert (got[:at_out] == -7).all() and (got[at_out + s_q * topk:] == -7).all()
