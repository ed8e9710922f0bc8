"""Host-buffer entry point (pipelined copies) against the device entry point."""
import pytest
import torch

from test_operator_b200.inputs import Workload, make_sequence

pytestmark = pytest.mark.gpu
KEYS = ("q", "kv", "dO", "lse", "O", "indices")


@pytest.mark.parametrize("q_start", [None, 40])
def test_host_entry_matches_device_entry(q_start, monkeypatch):
    from test_operator_b200 import op
    w = Workload("host", 1, 130, 512, 64, 128, "uniform", invalid_frac=0.1)       # 27 MB of inputs: blocks are of 4 MB at least
    s = make_sequence(w, device="cpu", seed=19)
    host = [s[k].pin_memory() for k in ("q", "kv", "dO", "lse", "O", "indices")]
    real, blocks = op.mla_bwd, []
    monkeypatch.setattr(op, "mla_bwd", lambda *a, **k: (blocks.append(a[0].shape[0]), real(*a, **k))[1])
    dq_h, dkv_h = op.mla_bwd_host(*host, device="cuda:0", q_start_index_s=q_start, n_chunks=5)
    assert len(blocks) == 5 and sum(blocks) == 130
    dev = [t.to("cuda:0") for t in host]
    dq_d, dkv_d = op.mla_bwd(*dev, q_start_index_s=q_start, check_device_status=True)
    from oracle.sparse_mla_ref import sparse_mla_bwd_ref
    from tests.metrics import assert_backward_close
    assert_backward_close(dq_d.cpu(), dkv_d.cpu(), *sparse_mla_bwd_ref(*host, q_start_index_s=q_start))
    assert not dq_h.is_cuda and not dkv_h.is_cuda
    assert torch.equal(dq_h.view(torch.int16), dq_d.cpu().view(torch.int16))
    assert (dkv_h - dkv_d.cpu()).abs().max().item() <= 1e-5 * dkv_d.abs().max().item()


@pytest.mark.parametrize("s_q,n_chunks", [(1, 8), (2, 2), (5, 8), (11, 7), (30, 30)])
def test_host_entry_with_fewer_rows_than_parts(s_q, n_chunks, monkeypatch):
    """Blocks of a few rows and of none."""
    from test_operator_b200 import op
    monkeypatch.setattr(op, "_HOST_BLOCK_BYTES", 1)
    s = make_sequence(Workload("rows", 1, s_q, 300, 16, 100, "uniform", invalid_frac=0.1), device="cuda:0", seed=20)
    dev = [s[k] for k in KEYS]
    host = [t.cpu().pin_memory() for t in dev]
    dq_h, dkv_h = op.mla_bwd_host(*host, device="cuda:0", q_start_index_s=None, n_chunks=n_chunks)
    dq_d, dkv_d = op.mla_bwd(*dev, q_start_index_s=None, check_device_status=True)
    assert torch.equal(dq_h.view(torch.int16), dq_d.cpu().view(torch.int16))
    assert (dkv_h - dkv_d.cpu()).abs().max().item() <= 1e-5 * dkv_d.abs().max().item()


def test_host_entry_takes_strided_and_longer_inputs():
    from test_operator_b200 import op
    s = make_sequence(Workload("strided", 1, 40, 300, 16, 100, "uniform", invalid_frac=0.1), device="cpu", seed=21)
    host = [s[k] for k in KEYS]
    want = op.mla_bwd_host(*host, device="cuda:0", q_start_index_s=None)
    q, kv, dO, lse, O, idx = host
    wide = torch.zeros(40, 16, 600, dtype=torch.bfloat16)
    wide[:, :, :576] = q
    got = op.mla_bwd_host(wide[:, :, :576], kv, torch.cat([dO, dO]), torch.cat([lse, lse]), O, idx.repeat(2, 1), device="cuda:0",
                          q_start_index_s=None)
    assert torch.equal(got[0].view(torch.int16), want[0].view(torch.int16))
    assert (got[1] - want[1]).abs().max().item() <= 1e-5 * want[1].abs().max().item()


@pytest.mark.parametrize("bad", ["lse_dtype", "dO_width", "heads", "indices_dtype", "transposed_q", "short_O", "kv_width"])
def test_host_entry_refuses_before_anything_is_copied(bad, monkeypatch):
    from test_operator_b200 import op
    s = make_sequence(Workload("bad", 1, 24, 300, 16, 100, "uniform"), device="cpu", seed=22)
    q, kv, dO, lse, O, idx = (s[k] for k in KEYS)
    if bad == "lse_dtype":
        lse = lse.double()
    elif bad == "dO_width":
        dO = dO[:, :, :256].contiguous()
    elif bad == "heads":
        q, dO, O, lse = (t[:, :12].contiguous() for t in (q, dO, O, lse))
    elif bad == "indices_dtype":
        idx = idx.long()
    elif bad == "transposed_q":
        q = q.transpose(0, 1).contiguous().transpose(0, 1)
    elif bad == "short_O":
        O = O[:20]
    else:
        kv = kv[:, :512].contiguous()
    copies = []
    real = torch.Tensor.copy_
    monkeypatch.setattr(torch.Tensor, "copy_", lambda self, *a, **k: (copies.append(1), real(self, *a, **k))[1])
    with pytest.raises(RuntimeError):
        op.mla_bwd_host(q, kv, dO, lse, O, idx, device="cuda:0", q_start_index_s=None)
    assert not copies


def test_reduction_rate_probe_adds_what_it_claims():
    """The probe's figure is bytes / time, so the bytes must be real: every launch adds exactly one to
    n_ctas x rows_per_cta x row_floats elements (whole rows, so every row holds one integer value)."""
    import ctypes
    from test_operator_b200 import op
    lib = op.load_library()
    n_rows, row_floats, rows_per_cta, n_ctas = 512, 576, 64, 7
    buf = torch.zeros(n_rows, row_floats, dtype=torch.float32, device="cuda:0")
    rc = lib.smla_reduction_rate_probe(ctypes.c_void_p(buf.data_ptr()), n_rows, row_floats, rows_per_cta, n_ctas,
                                       ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    torch.cuda.synchronize()
    assert buf.sum(dtype=torch.float64).item() == n_ctas * rows_per_cta * row_floats
    assert torch.equal(buf, buf[:, :1].expand_as(buf))
    assert lib.smla_reduction_rate_probe(None, n_rows, row_floats, rows_per_cta, n_ctas, None) == 1      # bad argument
    assert op.reduction_rate_gbs(4096, torch.device("cuda:0"), rows_per_cta=512) > 100.0
