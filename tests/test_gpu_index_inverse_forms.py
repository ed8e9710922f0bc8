"""Which form of the index inverse a call takes (the one without a sort makes three launches), each form bit for bit against the oracle at
the edges of its pieces, and the time where queries name a row more than once."""
import numpy as np
import pytest
import torch

from oracle.index_inverse_ref import index_inverse_ref

pytestmark = pytest.mark.gpu
DIRECT = 3                      # launches
ROUND14, ROUND16 = 296 * 7168, 296 * 8192


def _same_as_the_oracle(idx, s_kv, q_start=None):
    from test_operator_b200 import op
    row_ptr, entries = op.index_inverse(torch.from_numpy(idx).cuda(), s_kv, q_start_index_s=q_start)
    launches = op.last_launch_count()
    ref_ptr, ref_entries = index_inverse_ref(idx, s_kv, q_start)
    assert np.array_equal(row_ptr.cpu().numpy(), ref_ptr)
    assert np.array_equal(entries.cpu().numpy(), ref_entries)
    return launches


# a warp's piece is 320 slots, a batch sixteen of them: less than a piece, whole ones, one slot in the next piece, batch or round of turns
@pytest.mark.parametrize("slots", [57, 320, 321, 5119, 5120, 5121, 5440, 10241])
@pytest.mark.parametrize("rows", ["any", "one", "two", "same mark", "none", "rising"])
def test_pieces_and_turns(slots, rows):
    """`same mark`: rows that are different and share a mark (512 apart)."""
    s_q, s_kv = 148, 4000
    g = np.random.default_rng(slots)
    shape = (s_q, slots)
    idx = {"any": lambda: g.integers(-1, s_kv + 1, shape), "one": lambda: np.full(shape, 77), "two": lambda: g.choice([5, 3999], shape),
           "same mark": lambda: 3 + 512 * g.integers(0, 7, shape), "none": lambda: np.full(shape, -1),
           "rising": lambda: np.broadcast_to(np.arange(slots) % s_kv, shape)}[rows]()
    assert _same_as_the_oracle(np.ascontiguousarray(idx.astype(np.int32)), s_kv, 2000) == DIRECT


@pytest.mark.parametrize("s_q,topk", [(149, 320), (295, 163), (1481, 29), (10240, 2048), (9, 3000)])
def test_groups(s_q, topk):
    """The last group smaller, more queries a group, the most slots that are placed without a sort, few groups."""
    g = np.random.default_rng(s_q)
    assert _same_as_the_oracle(g.integers(-1, 6000, (s_q, topk)).astype(np.int32), 6000) == DIRECT


# (8192 slots: one block sorts them alone)
@pytest.mark.parametrize("s_kv", [255, 4096, 9000, 32768])
@pytest.mark.parametrize("slots", [8192, 20000, (1 << 20) - 1, 1 << 20, ROUND14, ROUND14 + 1, 297 * 7168 - 5, ROUND16 + 1, 2 * ROUND14 + 1])
def test_sort_of_few_long_queries(slots, s_kv):
    g = np.random.default_rng(slots + s_kv)
    for idx in (g.integers(-1, s_kv + 1, (1, slots)), g.choice([0, s_kv // 2, s_kv], (1, slots))):
        assert _same_as_the_oracle(idx.astype(np.int32), s_kv) != DIRECT


@pytest.mark.parametrize("s_q,topk,s_kv,q_start", [(1025, 1024, 60000, 30000), (3, 400000, 60000, 20000), (3, 300000, 255, 100), (300, 1024, 60000, 3),
                                                   (10241, 2048, 8192, None)])
def test_sort_of_other_shapes(s_q, topk, s_kv, q_start):
    """Causal bounds with several slots a query, in every size of block; more slots than are placed without a sort."""
    g = np.random.default_rng(s_q + topk)
    assert _same_as_the_oracle(g.integers(-1, s_kv + 1, (s_q, topk)).astype(np.int32), s_kv, q_start) != DIRECT


@pytest.mark.parametrize("s_kv", [8192, 32768])
def test_rows_named_again_do_not_slow_it_down(s_kv):
    """4096 x 2048 slots of distinct rows 67 and 76 us; of two rows 57 and 66 (466 and 475 where such slots were placed one after the other)."""
    from test_operator_b200 import op

    def best_us(idx):
        times = []
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            op.index_inverse(idx, s_kv)
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b) * 1e3)
        return min(times[1:])

    step = torch.arange(2048, device="cuda", dtype=torch.int32)
    first = torch.randint(0, s_kv, (4096, 1), dtype=torch.int32, device="cuda")
    distinct = (first + step * 1021) % s_kv
    limit = 2 * best_us(distinct)
    for idx in ((step % 2 * (s_kv // 2)).repeat(4096, 1), torch.full_like(distinct, 9), torch.randint(0, s_kv, (4096, 2048), dtype=torch.int32, device="cuda"),
                torch.randint(0, 64, (4096, 2048), dtype=torch.int32, device="cuda")):
        assert best_us(idx) < limit
