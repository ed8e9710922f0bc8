"""NaN and infinities through the forward: what is not a number stays none, whether a query is worked on whole or spread over
several clusters whose parts are added up.  Against plain fp32 torch on the valid slots."""
import pytest
import torch

from test_operator_b200.inputs import LOG2E, Workload, make_sequence

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _reference(q, kv, idx):
    o = torch.empty(*q.shape[:2], 512, device=DEV)
    lse = torch.empty(q.shape[:2], device=DEV)
    for r in range(q.shape[0]):
        k = kv[idx[r][idx[r] >= 0].long()].float()
        p = q[r].float() @ k.T / 24.0
        lse[r] = torch.logsumexp(p, 1) * LOG2E
        o[r] = torch.softmax(p, 1) @ k[:, :512]
    return o, lse


@pytest.mark.parametrize("h_q", [16, 64, 128])
@pytest.mark.parametrize("s_q", [2, 300])         # every query in parts; most queries whole, some cut between two clusters
@pytest.mark.parametrize("kind", ["kv_nan", "kv_inf", "q_nan", "one_head_nan", "all_minus_inf"])
def test_nonfinite_values_are_kept(kind, s_q, h_q):
    from test_operator_b200 import op
    s = make_sequence(Workload(kind, 1, s_q, 4096, h_q, 1500, "uniform", invalid_frac=0.1), device=DEV, seed=63, with_forward=False)
    q, kv, idx = s["q"], s["kv"], s["indices"]
    idx[:, 1100] = torch.arange(s_q, device=DEV, dtype=torch.int32) * 7 % 4096
    if kind in ("kv_nan", "kv_inf"):        # every second query meets it, in one of its six tiles
        kv[idx[::2, 1100].long(), 3] = float("nan" if kind == "kv_nan" else "inf")
    elif kind == "q_nan":
        q[1::2, :, 5] = float("nan")
    elif kind == "one_head_nan":
        q[:, 3, 570] = float("nan")
    else:                                   # products beyond the range of fp32
        q[:, :, 575], kv[:, 575] = 3e38, -3e38
    o_ref, lse_ref = _reference(q, kv, idx)
    o, lse = op.mla_fwd(q, kv, idx, q_start_index_s=None, check_device_status=True)
    assert torch.equal(torch.isnan(lse), torch.isnan(lse_ref))
    assert torch.equal(torch.isposinf(lse), torch.isposinf(lse_ref)) and torch.equal(torch.isneginf(lse), torch.isneginf(lse_ref))
    bad = ~torch.isfinite(o_ref)
    assert bad.any() and torch.equal(~torch.isfinite(o), bad)
    if not bad.all():                       # the tolerance of the other forward tests
        assert (o.float() - o_ref)[~bad].abs().max().item() <= 2 ** -6 * o_ref[~bad].abs().max().item()
