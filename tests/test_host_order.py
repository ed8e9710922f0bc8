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
    """The caller's stream; `mla_bwd` only keeps the Delta that it is given."""
    stream = _Stream()
    empty = torch.empty
    monkeypatch.setattr(torch, "empty", lambda *a, **k: empty(*a, **{n: v for n, v in k.items() if n != "pin_memory"}))
    monkeypatch.setattr(torch, "get_num_threads", lambda: 64)
    monkeypatch.setattr(torch.Tensor, "record_stream", lambda *_: None)
    for name, value in (("device", lambda _: contextlib.nullcontext()), ("stream", lambda _: contextlib.nullcontext()),
                        ("Stream", _Stream), ("current_stream", lambda *_: stream)):
        monkeypatch.setattr(torch.cuda, name, value)
    monkeypatch.setattr(op, "_validate", lambda *_: None)
    stream.given = []
    monkeypatch.setattr(op, "mla_bwd", lambda *a, **k: stream.given.append(k["delta"].clone()))
    return stream


def test_delta_is_of_what_the_stream_has_written(caller):
    heads, rows = 64, 130
    old, new = (torch.full((rows, heads, 512), v).bfloat16() for v in (1.0, 2.0))
    O, dO = old.clone(), old.clone()
    caller.pending += [lambda: O.copy_(new), lambda: dO.copy_(new)]
    q, kv = torch.zeros(rows, heads, 576).bfloat16(), torch.zeros(300, 576).bfloat16()
    op.mla_bwd_host(q, kv, dO, torch.zeros(rows, heads), O, torch.zeros(rows, 100, dtype=torch.int32), device="cpu")
    got = torch.cat(caller.given)
    assert got.shape == (rows, heads) and bool((got == 4 * 512).all())
