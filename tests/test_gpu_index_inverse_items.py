"""The index inverse where it changes between fourteen and sixteen entries a thread (one, two and three rounds of 296 blocks of 7168 or
8192 slots), full and ragged last blocks, 16- and 32-bit keys; bit for bit against the oracle."""
import numpy as np
import pytest
import torch

from oracle.index_inverse_ref import index_inverse_ref

pytestmark = pytest.mark.gpu
ROUND14, ROUND16 = 296 * 7168, 296 * 8192


@pytest.mark.parametrize("s_kv", [9000, 65535, 70001])
@pytest.mark.parametrize("slots", [8192, 8191, ROUND14 + 1, ROUND16, ROUND16 + 1, 2 * ROUND14, 2 * ROUND14 + 1, 2 * ROUND16, 2 * ROUND16 + 1])
def test_around_the_changes(slots, s_kv):
    from test_operator_b200 import op
    g = np.random.default_rng(slots + s_kv)
    idx = g.integers(-1, s_kv + 1, size=(slots, 1)).astype(np.int32)
    row_ptr, entries = op.index_inverse(torch.from_numpy(idx).cuda(), s_kv)
    ref_ptr, ref_entries = index_inverse_ref(idx, s_kv, None)
    assert np.array_equal(row_ptr.cpu().numpy(), ref_ptr)
    assert np.array_equal(entries.cpu().numpy(), ref_entries)
