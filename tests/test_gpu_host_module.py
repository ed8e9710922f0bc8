"""The compiled host module against the Python way it stands in front of: every form of a call gives the same outputs or the same
error through both, and the form that nearly every call has is taken by the module."""
import numpy
import pytest
import torch

from test_operator_b200.inputs import Workload, make_sequence

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


class Sub(torch.Tensor):
    pass


def _strided(t):
    return t.transpose(0, 1).contiguous().transpose(0, 1)


# name, taken by the module, changes to the arguments (a dict of replacements made from the plain ones)
FORMS = [
    ("plain", True, lambda a: {}),
    ("three_dims", True, lambda a: {"kv": a["kv"][:, None], "indices": a["indices"][:, None]}),
    ("parameter", True, lambda a: {"q": torch.nn.Parameter(a["q"])}),
    ("scale_and_start", True, lambda a: {"sm_scale": 0.07, "q_start_index_s": 150}),
    ("no_start", True, lambda a: {"q_start_index_s": None}),
    ("numpy_scalars", False, lambda a: {"sm_scale": numpy.float32(0.07), "q_start_index_s": numpy.int64(150)}),
    ("int_scale", False, lambda a: {"sm_scale": 1}),
    ("bool_start", False, lambda a: {"q_start_index_s": True}),
    ("start_beyond_32_bits", False, lambda a: {"q_start_index_s": 2 ** 40 + 150}),
    ("subclass", False, lambda a: {"q": a["q"].as_subclass(Sub)}),
    ("strided", False, lambda a: {"q": _strided(a["q"])}),
    ("wrong_dtype", False, lambda a: {"kv": a["kv"].float()}),
    ("host_tensor", False, lambda a: {"indices": a["indices"].cpu()}),
    ("no_tensor", False, lambda a: {"kv": None}),
    ("wrong_heads", False, lambda a: {k: a[k][:, :12].contiguous() for k in ("q", "dO", "O", "lse")}),
    ("wrong_rows", False, lambda a: {"indices": a["indices"][1:].contiguous()}),
    ("wrong_dims", False, lambda a: {"kv": a["kv"][None]}),
    ("no_query", False, lambda a: {k: a[k][:0].contiguous() for k in ("q", "dO", "O", "lse", "indices")}),
    ("no_slot", False, lambda a: {"indices": a["indices"][:, :0].contiguous()}),
    ("misaligned", True, lambda a: {"kv": torch.cat([a["kv"].reshape(-1), a["kv"][0]])[1:1 + a["kv"].numel()].view_as(a["kv"])}),
]


def _outcome(f):
    try:
        return f()
    except Exception as e:
        return type(e), str(e)


def _same(a, b):
    if isinstance(a[0], torch.Tensor) and isinstance(b[0], torch.Tensor):
        return all(x.shape == y.shape and x.dtype == y.dtype and torch.equal(x, y) for x, y in zip(a, b))
    return a == b


@pytest.mark.parametrize("form", FORMS, ids=[f[0] for f in FORMS])
def test_both_ways_agree(form, monkeypatch):
    from test_operator_b200 import op
    _, taken, change = form
    s = make_sequence(Workload("host", 1, 5, 300, 16, 70, "uniform", invalid_frac=0.1), device=DEV, seed=3)
    a = {k: s[k] for k in ("q", "kv", "dO", "lse", "O", "indices")}
    a.update(sm_scale=None, q_start_index_s=0)
    a.update(change(a))
    scal = {k: a.pop(k) for k in ("sm_scale", "q_start_index_s")}
    native = op._host()
    if native is op._NoNativeHost:
        pytest.skip("the host module is not built")
    bwd = lambda **kw: op.mla_bwd(*a.values(), **scal, **kw)                               # noqa: E731
    fwd = lambda: op.mla_fwd(a["q"], a["kv"], a["indices"], **scal)                        # noqa: E731
    # (the kernels' order of additions into dKV varies: one query per row of dKV would be needed to compare it bit for bit; here its
    # shape and type)
    calls = [fwd, lambda: bwd()[:1], lambda: (torch.zeros_like(bwd()[1]),), lambda: bwd(accumulate=True),
             lambda: (bwd(out_dq=torch.empty_like(a["q"]), out_dkv=torch.empty(a["kv"].shape, device=DEV))[0],)]
    got = [_outcome(c) for c in calls]
    assert (native.fwd(a["q"], a["kv"], a["indices"], scal["sm_scale"], scal["q_start_index_s"], 1) is not None) == taken
    monkeypatch.setattr(op, "_native", op._NoNativeHost)
    for g, c in zip(got, calls):
        want = _outcome(c)
        assert _same(g, want), (g, want)


def test_wrapped_tensors_are_not_taken():
    from test_operator_b200 import op
    s = make_sequence(Workload("host", 1, 4, 300, 16, 70, "uniform"), device=DEV, seed=4)
    with pytest.raises(Exception):
        torch.func.vmap(lambda q: op.mla_fwd(q, s["kv"], s["indices"])[0])(torch.stack([s["q"], s["q"]]))
    seen = []

    def f(q):
        seen.append(op._host().fwd(q, s["kv"], s["indices"], None, 0, 1))
        return q.sum()
    torch.func.grad(f)(s["q"])
    assert seen == [None]
