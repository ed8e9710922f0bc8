"""Backward calls that are given Delta: the same bits of dQ as with O, in small calls (ranges by the shape) and larger ones."""
import pytest
import torch

from oracle.sparse_mla_ref import sparse_mla_bwd_ref
from test_operator_b200.inputs import Workload, make_sequence
from tests.metrics import assert_backward_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("s_q,h_q,topk", [(3, 16, 100), (130, 64, 300), (700, 128, 130)])
def test_given_delta(s_q, h_q, topk):
    from test_operator_b200 import op
    s = make_sequence(Workload("given", 1, s_q, 900, h_q, topk, "uniform", invalid_frac=0.1), device="cuda:0", seed=s_q)
    s["indices"][s_q // 2] = -1
    args = [s[k] for k in ("q", "kv", "dO", "lse", "O", "indices")]
    delta = torch.empty(s_q, h_q, dtype=torch.float32)
    job = op._host().delta_start(s["O"].cpu(), s["dO"].cpu(), delta, 2)
    assert op._host().delta_wait(job, delta.numel(), True)
    want = op.mla_bwd(*args, q_start_index_s=None)
    oracle = sparse_mla_bwd_ref(*args, q_start_index_s=None)
    args[4] = torch.full_like(s["O"], float("nan"))          # not read
    got = op.mla_bwd(*args, q_start_index_s=None, delta=delta.cuda(), check_device_status=True)
    assert torch.equal(got[0].view(torch.int16), want[0].view(torch.int16))
    assert (got[1] - want[1]).abs().max().item() <= 1e-5 * want[1].abs().max().item()
    assert_backward_close(*got, *oracle)


def test_host_entry_without_threads_copies_o(monkeypatch):
    from test_operator_b200 import op
    s = make_sequence(Workload("host", 1, 130, 512, 64, 128, "uniform"), device="cpu", seed=3)
    args = [s[k].pin_memory() for k in ("q", "kv", "dO", "lse", "O", "indices")]
    given = []
    real = op.mla_bwd
    monkeypatch.setattr(op, "mla_bwd", lambda *a, **k: (given.append("delta" in k), real(*a, **k))[1])
    monkeypatch.setattr(op, "_HOST_DELTA_BYTES", 0)          # calls of this size copy O, whatever the threads
    monkeypatch.setattr(op, "_idle_cores", lambda: 64)
    results = []
    for threads in (1, 64):
        monkeypatch.setattr(torch, "get_num_threads", lambda: threads)
        results.append(op.mla_bwd_host(*args, device="cuda:0", q_start_index_s=None, n_chunks=4))
    assert given == [False] * 4 + [True] * 4
    assert torch.equal(results[0][0].view(torch.int16), results[1][0].view(torch.int16))
    assert (results[0][1] - results[1][1]).abs().max().item() <= 1e-5 * results[0][1].abs().max().item()
