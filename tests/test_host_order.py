"""The host entry reads its inputs behind what the caller's stream holds when it is called, on the CPU: streams are stood in for by objects
that do their work when they are waited for."""
import contextlib

import pytest
import torch

from test_operator_b200 import op


class _Stream:
    """Work runs when the stream, or an event recorded behind it, is waited for by the host."""

    def __init__(self):
        self.pending = []

    def synchronize(self):
        while self.pending:
            self.pending.pop(0)()

    def query(self):
        return not self.pending

    def record_event(self):
        return self

    def wait_stream(self, other):
        pass

    wait_event = wait_stream


@pytest.fixture
def caller(monkeypatch):
    """The caller's stream of calls that are long enough for Delta on the host; `mla_bwd` only keeps the Delta that it is given."""
    stream = _Stream()
    empty = torch.empty
    monkeypatch.setattr(torch, "empty", lambda *a, **k: empty(*a, **{n: v for n, v in k.items() if n != "pin_memory"}))
    monkeypatch.setattr(torch, "get_num_threads", lambda: 64)
    monkeypatch.setattr(op, "_HOST_DELTA_BYTES", 0)
    monkeypatch.setattr(op, "_idle_cores", lambda: 64)
    monkeypatch.setattr(torch.Tensor, "record_stream", lambda *_: None)
    for name, value in (("device", lambda _: contextlib.nullcontext()), ("stream", lambda _: contextlib.nullcontext()),
                        ("Stream", _Stream), ("current_stream", lambda *_: stream)):
        monkeypatch.setattr(torch.cuda, name, value)
    monkeypatch.setattr(op, "_validate", lambda *_: None)
    stream.given, stream.args = [], []

    def mla_bwd(*args, delta=None, **_):
        stream.given.append(delta if delta is None else delta.clone())
        stream.args.append(args)
    monkeypatch.setattr(op, "mla_bwd", mla_bwd)
    return stream


def _call(O, dO):
    rows, heads = O.shape[:2]
    q, kv = torch.zeros(rows, heads, 576).bfloat16(), torch.zeros(300, 576).bfloat16()
    op.mla_bwd_host(q, kv, dO, torch.zeros(rows, heads), O, torch.zeros(rows, 100, dtype=torch.int32), device="cpu")


def test_delta_is_of_what_the_stream_has_written(caller):
    heads, rows = 64, 130
    old, new = (torch.full((rows, heads, 512), v).bfloat16() for v in (1.0, 2.0))
    O, dO = old.clone(), old.clone()
    caller.pending += [lambda: O.copy_(new), lambda: dO.copy_(new)]
    _call(O, dO)
    got = torch.cat(caller.given)
    assert got.shape == (rows, heads) and bool((got == 4 * 512).all())


@pytest.mark.parametrize("what", ["short", "busy", "one thread", "neither"])
def test_who_finds_delta(caller, monkeypatch, what):
    """The host where the call is long and cores are idle; O is copied otherwise, as these calls take longer with threads beside them."""
    O = torch.ones(130, 64, 512).bfloat16()
    if what == "short":
        monkeypatch.setattr(op, "_HOST_DELTA_BYTES", 28 << 20)
    elif what == "busy":
        monkeypatch.setattr(op, "_idle_cores", lambda: 5)
    elif what == "one thread":
        monkeypatch.setattr(torch, "get_num_threads", lambda: 1)
    _call(O, O)
    assert [d is None for d in caller.given] == [what != "neither"] * len(caller.given) and len(caller.given) > 1


@pytest.mark.parametrize("by", ["host", "device"])
def test_o_is_on_the_device_only_where_it_is_read(caller, monkeypatch, by):
    O, dO = (torch.randn(130, 64, 512, generator=torch.Generator().manual_seed(n)).bfloat16() for n in (1, 2))
    if by == "device":              # no compiled host module
        monkeypatch.setattr(op, "_host", lambda: op._NoNativeHost)
    _call(O, dO)
    given, o, g = caller.given, [a[4] for a in caller.args], [a[2] for a in caller.args]
    assert torch.equal(torch.cat(g), dO) and [d is None for d in given] == [by == "device"] * len(given)
    if by == "device":
        assert torch.equal(torch.cat(o), O)
    else:
        assert [t.data_ptr() for t in o] == [t.data_ptr() for t in g]
    rows = 130 * 64
    of_o = rows * (1024 if by == "device" else 4)       # O, or Delta
    assert op.last_host_copy_bytes() == (300 * 1152 + rows * (1152 + 1024 + 4) + of_o + 130 * 400, rows * 1152 + 300 * 2304)


def test_the_limit_and_the_idle_cores():
    assert op._HOST_DELTA_BYTES >= 256 << 20
    assert 0 <= op._idle_cores() <= len(op.os.sched_getaffinity(0))
