"""What a workspace held before a call does not matter: not its scratch, and of its first 256 bytes only the error word does."""
import pytest
import torch

from oracle.sparse_mla_ref import sparse_mla_bwd_ref, sparse_mla_fwd_ref
from test_operator_b200.inputs import LOG2E, Workload, make_sequence
from tests.metrics import assert_backward_close

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
KEYS = ("q", "kv", "dO", "lse", "O", "indices")


@pytest.mark.parametrize("s_q,h_q", [(3, 16), (90, 128), (700, 64)])
@pytest.mark.parametrize("byte", [0, 1, 255])
def test_results_do_not_depend_on_what_the_workspace_held(s_q, h_q, byte):
    from test_operator_b200 import op
    s = make_sequence(Workload("garbage", 1, s_q, 900, h_q, 300, "uniform", invalid_frac=0.1), device=DEV, seed=71)
    args = [s[k] for k in KEYS]
    ws = op.workspace_for(s["q"], s["kv"], s["indices"])
    ws.buf.fill_(byte)
    dq, dkv = op.mla_bwd(*args, q_start_index_s=None, workspace=ws)
    assert_backward_close(dq, dkv, *sparse_mla_bwd_ref(*args, q_start_index_s=None, chunk_s=16))
    ws = op.Workspace(64 << 20, DEV)
    ws.buf.fill_(byte)
    o, lse = op.mla_fwd(s["q"], s["kv"], s["indices"], q_start_index_s=None, workspace=ws)
    o_ref, lse_ref = sparse_mla_fwd_ref(s["q"], s["kv"], s["indices"], q_start_index_s=None)
    assert (lse - lse_ref * LOG2E).abs().max().item() <= 2e-4
    assert (o.float() - o_ref.float()).abs().max().item() <= 2 ** -6 * o_ref.float().abs().max().item()
