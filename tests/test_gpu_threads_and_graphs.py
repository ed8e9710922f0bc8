"""Calls without a workspace of their own: from several host threads on one stream, and recorded in a CUDA graph that outlives
larger calls on the stream it was recorded on."""
import threading

import pytest
import torch

from test_operator_b200.inputs import Workload, make_sequence

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
KEYS = ("q", "kv", "dO", "lse", "O", "indices")


def _calls(op, s):
    """Entry points that repeat bit for bit, by name (of the plain backward dQ does)."""
    from tests.conftest import import_extension
    q, kv, idx = s["q"], s["kv"], s["indices"]
    args = [s[k] for k in KEYS]
    return {
        "bwd": lambda: op.mla_bwd(*args, q_start_index_s=None)[:1],
        "repeatable": lambda: op.mla_bwd(*args, q_start_index_s=None, deterministic=True),
        "module": lambda: import_extension().mla_bwd(*args, q_start_index_s=None)[:1],
        "fwd": lambda: op.mla_fwd(q, kv, idx, q_start_index_s=None),
        "inverse": lambda: op.index_inverse(idx, kv.shape[0]),
    }


def _sequence(s_q, s_kv, h_q, topk, seed):
    return make_sequence(Workload("tg", 1, s_q, s_kv, h_q, topk, "uniform", invalid_frac=0.1), device=DEV, seed=seed)


def _same(a, b):
    return all(torch.equal(x.view(torch.int16), y.view(torch.int16)) for x, y in zip(a, b))


SMALL, LARGE = (5, 700, 64, 300, 81), (300, 2000, 128, 600, 82)


@pytest.mark.parametrize("names", [("fwd", "fwd"), ("inverse", "inverse"), ("fwd", "inverse"), ("bwd", "bwd"), ("bwd", "fwd"),
                                   ("repeatable", "repeatable"), ("repeatable", "bwd"), ("module", "module")])
def test_two_threads_on_one_stream(names):
    from test_operator_b200 import op
    jobs = [_calls(op, _sequence(*shape))[n] for n, shape in zip(names, (SMALL, LARGE))]
    want = [j() for j in jobs]
    torch.cuda.synchronize()
    wrong = [0, 0]
    start = threading.Barrier(2)

    def work(i):
        torch.cuda.set_device(0)
        start.wait()
        for _ in range(10):                 # a few results at a time, compared afterwards: the launches come in quick succession
            got = [jobs[i]() for _ in range(20)]
            wrong[i] += sum(not _same(g, want[i]) for g in got)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert wrong == [0, 0]


@pytest.mark.parametrize("name", ["fwd", "inverse", "bwd", "repeatable", "module"])
def test_a_graph_outlives_a_larger_call_on_its_stream(name):
    from test_operator_b200 import op
    small, large = (_calls(op, _sequence(*shape))[name] for shape in (SMALL, LARGE))
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(side):
        want = [t.clone() for t in small()]             # the warm-up, on the stream that is recorded
        with torch.cuda.graph(graph, stream=side):
            got = small()
        large()
        # what a buffer given up meanwhile would now belong to
        others = [torch.full((n,), 77, dtype=torch.uint8, device=DEV) for n in (1 << 12, 1 << 16, 1 << 20, 1 << 22, 1 << 24, 1 << 25)]
        for _ in range(2):
            for t in got:
                t.zero_()
            graph.replay()
            side.synchronize()
            assert _same(got, want)
        assert all(bool((t == 77).all()) for t in others)


def test_a_backward_after_one_that_was_only_recorded():
    """The first backward on a stream is recorded and not run; calls behind it on that stream get a workspace of their own."""
    from test_operator_b200 import op
    s = _sequence(*SMALL)
    small = _calls(op, s)["bwd"]
    want = small()
    torch.cuda.synchronize()
    op.release_cached_workspaces()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(side):
        with torch.cuda.graph(graph, stream=side):
            recorded = small()
        got = op.mla_bwd(*[s[k] for k in KEYS], q_start_index_s=None, check_device_status=True)
        assert _same(got[:1], want)
        graph.replay()
        side.synchronize()
        assert _same(recorded, want)
