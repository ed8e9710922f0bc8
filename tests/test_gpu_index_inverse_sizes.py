"""The index inverse at the edges of its kernels' size ranges, bit for bit against the oracle: the one-block sort, four and
sixteen entries per thread, 16- and 32-bit keys, rows without slots over more than one block of the row_ptr kernel, all slots
on one row.  Which form a shape takes goes by a rule on its slots and rows: `tests/test_gpu_index_inverse_forms.py` checks that with each."""
import numpy as np
import pytest
import torch

from oracle.index_inverse_ref import index_inverse_ref

pytestmark = pytest.mark.gpu

CASES = [
    # s_q, topk, s_kv, causal start
    (1, 1, 1, None),
    (4, 2048, 65535, None),      # exactly one block, the largest 16-bit key
    (4, 2048, 65536, None),      # the same with 32-bit keys
    (8193, 1, 3000, None),       # one slot more: four entries per thread
    (5, 2048, 100000, None),     # long stretches of rows without a slot
    (512, 2047, 4096, 100),      # just below the large form
    (512, 2048, 4096, None),     # exactly the large form's smallest input
    (1025, 1024, 70000, None),   # three passes of the large form, ragged end
    (1200, 1000, 255, 0),        # one pass
]


@pytest.mark.parametrize("s_q,topk,s_kv,q_start", CASES)
@pytest.mark.parametrize("pattern", ["random", "one_row"])
def test_sizes(s_q, topk, s_kv, q_start, pattern):
    from test_operator_b200 import op
    g = np.random.default_rng(s_q + topk)
    idx = g.integers(-1, s_kv + 1, size=(s_q, topk)).astype(np.int32)
    if pattern == "one_row":
        idx[:, ::2] = s_kv // 2
        idx[:, 1::2] = s_kv // 3
    row_ptr, entries = op.index_inverse(torch.from_numpy(idx).cuda(), s_kv, q_start_index_s=q_start)
    ref_ptr, ref_entries = index_inverse_ref(idx, s_kv, q_start)
    assert np.array_equal(row_ptr.cpu().numpy(), ref_ptr)
    assert np.array_equal(entries.cpu().numpy(), ref_entries)


@pytest.mark.parametrize("s_kv", [65535, 65536, (1 << 20) - 1, 1 << 20, (1 << 20) + 5000])     # 64, 65, 1024, 1025, 1029 blocks of rows
@pytest.mark.parametrize("used", ["first_rows", "last_row", "two_far_rows", "none"])
def test_long_stretches_of_unused_rows(s_kv, used):
    from test_operator_b200 import op
    g = np.random.default_rng(s_kv)
    idx = {"first_rows": lambda n: g.integers(-1, 700, n), "last_row": lambda n: np.full(n, s_kv - 1),
           "two_far_rows": lambda n: np.where(g.integers(0, 2, n) == 0, 1023, s_kv * 2 // 3), "none": lambda n: np.full(n, -1)}[used]((9, 2000))
    idx = idx.astype(np.int32)
    row_ptr, entries = op.index_inverse(torch.from_numpy(idx).cuda(), s_kv)
    ref_ptr, ref_entries = index_inverse_ref(idx, s_kv, None)
    assert np.array_equal(row_ptr.cpu().numpy(), ref_ptr)
    assert np.array_equal(entries.cpu().numpy(), ref_entries)


def test_time_is_linear_in_the_rows():
    """Slots on the first rows of a long kv pool only: four times the rows take at most about four times as long (42 and 78 us), not
    sixteen times."""
    from test_operator_b200 import op
    idx = torch.randint(0, 1024, (16, 2048), dtype=torch.int32, device="cuda")

    def best_us(s_kv):
        times = []
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            op.index_inverse(idx, s_kv)
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b) * 1e3)
        return min(times[1:])

    assert best_us(1 << 22) < 8 * best_us(1 << 20)
