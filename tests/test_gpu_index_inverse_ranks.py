"""The index inverse where its kernels change how they rank (the large form: up to 296 blocks of 7168 slots by shared-memory words,
above by ballots), with ragged last blocks, digits of seven and eight bits, 16- and 32-bit keys, and many equal keys in a step; bit
for bit against the oracle."""
import numpy as np
import pytest
import torch

from oracle.index_inverse_ref import index_inverse_ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("slots,s_kv", [(296 * 7168, 8192), (296 * 7168 + 1, 32768), (297 * 7168 - 5, 70000), (300 * 7168, 65535), (1 << 20, 65536)])
@pytest.mark.parametrize("spread", ["all_rows", "three_rows"])
def test_around_the_change(slots, s_kv, spread):
    from test_operator_b200 import op
    g = np.random.default_rng(slots + s_kv)
    rows = g.integers(-1, s_kv + 1, size=(slots, 1)) if spread == "all_rows" else g.choice([0, s_kv // 2, s_kv], size=(slots, 1))
    idx = rows.astype(np.int32)
    row_ptr, entries = op.index_inverse(torch.from_numpy(idx).cuda(), s_kv)
    ref_ptr, ref_entries = index_inverse_ref(idx, s_kv, None)
    assert np.array_equal(row_ptr.cpu().numpy(), ref_ptr)
    assert np.array_equal(entries.cpu().numpy(), ref_entries)
