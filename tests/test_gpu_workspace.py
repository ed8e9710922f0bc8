"""What a workspace held before a call does not matter: not its scratch, and of its first 256 bytes only the error word does.
Tensors need no more than the alignment they are checked for."""
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


@pytest.mark.parametrize("s_q,h_q", [(3, 128), (200, 64)])
def test_tensors_at_the_smallest_alignment(s_q, h_q):
    """Every tensor of the C ABI 16 bytes (bf16) or 4 bytes (indices, lse) off a larger power of two."""
    from test_operator_b200 import op
    lib = op.load_library()
    s = make_sequence(Workload("align", 1, s_q, 900, h_q, 301, "uniform", invalid_frac=0.1), device=DEV, seed=72)

    def off(t, elements):
        room = torch.empty(t.numel() + 64, dtype=t.dtype, device=DEV)
        view = room[elements:elements + t.numel()].view(t.shape)
        assert view.data_ptr() % 512 == elements * t.element_size()
        return view.copy_(t)

    q, kv, dO, O, idx, lse = (off(s[k], n) for k, n in (("q", 8), ("kv", 8), ("dO", 8), ("O", 8), ("indices", 1), ("lse", 1)))
    stream = torch.cuda.current_stream().cuda_stream
    o_ref, lse_ref = op.mla_fwd(s["q"], s["kv"], s["indices"], q_start_index_s=None)
    o, lse_out = off(torch.zeros_like(o_ref), 8), off(torch.zeros_like(lse_ref), 1)
    ws = op.Workspace(64 << 20, DEV)
    p = op._FwdParams(q.data_ptr(), kv.data_ptr(), idx.data_ptr(), o.data_ptr(), lse_out.data_ptr(), s_q, 900, h_q, 301, 0.0, op.NO_CAUSAL, 1, None)
    assert lib.smla_fwd_run(ctypes.byref(p), ws.ptr, ws.nbytes, stream) == 0 and op.device_status(ws) == 0
    assert torch.equal(o.view(torch.int16), o_ref.view(torch.int16)) and torch.equal(lse_out, lse_ref)
    dq_ref, dkv_ref = op.mla_bwd(*[s[k] for k in KEYS], q_start_index_s=None)
    dq, dkv = off(torch.zeros_like(dq_ref), 8), off(torch.zeros_like(dkv_ref), 4)
    op.mla_bwd(q, kv, dO, lse, O, idx, q_start_index_s=None, out_dq=dq, out_dkv=dkv, check_device_status=True)
    assert torch.equal(dq.view(torch.int16), dq_ref.view(torch.int16))
    assert (dkv - dkv_ref).abs().max().item() <= 1e-5 * dkv_ref.abs().max().item()
