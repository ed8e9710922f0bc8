"""Delta = rowsum(O * dO) found on the host: the order of the device's sums, whatever the number of threads and rows."""
import ctypes
import shutil
import subprocess

import numpy as np
import pytest
import torch


def _job(o, g, threads):
    from test_operator_b200 import op
    out = torch.full(o.shape[:2], -1.0)
    job = op._host().delta_start(o, g, out, threads)
    return op._host(), job, out


@pytest.mark.parametrize("rows,heads,threads", [(1, 8, 1), (16, 8, 3), (43, 24, 2), (129, 128, 6)])
def test_sums_in_the_order_of_a_warp(rows, heads, threads):
    gen = torch.Generator().manual_seed(rows)
    o, g = (torch.randn(rows, heads, 512, generator=gen).bfloat16() for _ in range(2))
    host, job, out = _job(o, g, threads)
    assert host.delta_wait(job, out.numel(), True)
    p = (o.float() * g.float()).numpy().reshape(-1, 2, 32, 8)      # exact products
    acc = np.zeros((len(p), 32), np.float32)
    for half in range(2):
        for k in range(8):
            acc += p[:, half, :, k]
    n = 32
    while n > 1:
        n //= 2
        acc = acc[:, :n] + acc[:, n:2 * n]
    assert np.array_equal(acc[:, 0], out.numpy().reshape(-1))


def test_a_part_of_the_rows_can_be_waited_for_and_a_job_dropped():
    o = torch.ones(600, 128, 512).bfloat16()
    host, job, out = _job(o, o, 4)
    assert host.delta_wait(job, 1000, True) and bool((out.view(-1)[:1000] == 512).all())
    del job                                     # ends its threads; the rows that are done stay
    assert set(out.view(-1).tolist()) <= {512.0, -1.0}


@pytest.mark.parametrize("case", ["strided", "short", "type", "negated"])
def test_other_inputs_are_left_to_the_device(case):
    o = torch.ones(8, 8, 512).bfloat16()
    other = {"strided": torch.ones(8, 8, 520).bfloat16()[:, :, :512], "short": o[:7], "type": o.half(),
             "negated": torch._neg_view(o)}[case]
    host, job, _ = _job(o, other, 2)
    assert job is None


@pytest.mark.parametrize("flags", [[], ["-DSMLA_PLAIN_DELTA"]])
def test_every_way_the_sum_is_compiled(flags, tmp_path):
    """With vectors, and as the plain loop that other compilers and processors get."""
    from test_operator_b200 import build
    compiler = shutil.which("g++")
    if compiler is None:
        pytest.skip("no g++")
    source, lib = tmp_path / "sum.cpp", tmp_path / "sum.so"
    source.write_text(f'#include "{build.HOST_DELTA}"\nextern "C" void sums(const uint16_t* o, const uint16_t* g, float* out, int64_t n) '
                      "{ delta_rows_host(o, g, out, n); }\n")
    subprocess.run([compiler, "-O2", "-std=c++17", "-shared", "-fPIC", *flags, str(source), "-o", str(lib)], check=True)
    o, g = (torch.randn(16, 8, 512, generator=torch.Generator().manual_seed(n)).bfloat16() for n in (1, 2))
    got = torch.empty(16, 8)
    ctypes.CDLL(str(lib)).sums(*(ctypes.c_void_p(t.data_ptr()) for t in (o, g, got)), ctypes.c_int64(128))
    host, job, want = _job(o, g, 1)
    assert host.delta_wait(job, want.numel(), True) and torch.equal(got, want)


def test_the_module_is_named_by_the_sum_too(monkeypatch, tmp_path):
    from test_operator_b200 import build
    here, other = build.host_path(), tmp_path / "smla_host_delta.h"
    with open(build.HOST_DELTA) as f:
        other.write_text(f.read() + "// another one\n")
    monkeypatch.setattr(build, "HOST_DELTA", str(other))
    assert build.host_path() != here
