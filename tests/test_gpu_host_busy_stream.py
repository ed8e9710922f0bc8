"""Host entry called while the caller's stream is still filling the pinned inputs."""
import pytest
import torch

from test_operator_b200.inputs import Workload, make_sequence
from tests.metrics import assert_backward_close

pytestmark = pytest.mark.gpu
KEYS = ("q", "kv", "dO", "lse", "O", "indices")


@pytest.mark.parametrize("delta_on_the_host", [False, True])
def test_inputs_that_arrive_on_the_stream(delta_on_the_host, monkeypatch):
    from oracle.sparse_mla_ref import sparse_mla_bwd_ref
    from test_operator_b200 import op
    if delta_on_the_host:
        monkeypatch.setattr(op, "_HOST_DELTA_BYTES", 0)
        monkeypatch.setattr(op, "_idle_cores", lambda: 64)
        monkeypatch.setattr(torch, "get_num_threads", lambda: 64)
    s = make_sequence(Workload("busy", 1, 130, 512, 64, 128, "uniform", invalid_frac=0.1), device="cuda:0", seed=23)
    dev = [s[k] for k in KEYS]
    host = [torch.zeros(t.shape, dtype=t.dtype, pin_memory=True) for t in dev]
    big = torch.zeros(1 << 28, device="cuda:0")
    torch.cuda.synchronize()
    for _ in range(20):                 # some 6 ms in front of the copies
        big.add_(1.0)
    for h, d in zip(host, dev):
        h.copy_(d, non_blocking=True)
    dq, dkv = op.mla_bwd_host(*host, device="cuda:0", q_start_index_s=None)
    assert_backward_close(dq, dkv, *sparse_mla_bwd_ref(*(t.cpu() for t in dev), q_start_index_s=None))
