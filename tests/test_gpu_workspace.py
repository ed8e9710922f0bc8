"""What a workspace held before a call does not matter: not its scratch, and of its first 256 bytes only the error word does."""
import ctypes

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


@pytest.mark.parametrize("s_q,h_q", [(1, 64), (3, 128)])
def test_the_forward_gets_from_the_size_it_asked_for_what_it_gets_from_more(s_q, h_q):
    """A query's tiles go to as many clusters with a workspace of exactly the size asked for as with a larger one: same bits."""
    from test_operator_b200 import op
    s = make_sequence(Workload("exact", 1, s_q, 900, h_q, 700, "uniform", invalid_frac=0.1), device=DEV, seed=73, with_forward=False)
    args = (s["q"], s["kv"], s["indices"])
    lib = op.load_library()
    p = op._FwdParams(0, 0, 0, 0, 0, s_q, 900, h_q, 700, 0.0, op.NO_CAUSAL, 1, None)
    need = lib.smla_fwd_workspace_size(ctypes.byref(p), 0)
    (o1, lse1), (o2, lse2) = (op.mla_fwd(*args, q_start_index_s=None, workspace=op.Workspace(n, DEV)) for n in (need, 2 * need))
    assert torch.equal(o1.view(torch.int16), o2.view(torch.int16)) and torch.equal(lse1, lse2)
