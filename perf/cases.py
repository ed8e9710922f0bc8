"""The work whose speed this framework is judged by: calls of its public entry points over the sizes they are used at.

A case is a dict of plain values:
  path    the entry point, see `run`: "bwd" (op.mla_bwd), "module" (mla_bwd_cuda.mla_bwd, the drop-in extension),
          "varlen" (op.mla_bwd_varlen), "repro" (op.mla_bwd with deterministic=True), "host" (op.mla_bwd_host on pinned
          host buffers), "fwd" (op.mla_fwd), "train" (op.sparse_mla, forward and backward through autograd),
          "inverse" (op.index_inverse)
  s_q, s_kv, h_q, topk    queries, kv rows, heads, top-k slots per query (d_qk = 576, d_v = 512 throughout)
  pattern how the indices are drawn:
          "uniform"  distinct rows anywhere in kv
          "offset"   the queries are the last s_q tokens of the s_kv; distinct rows below the query's own position
          "prefix"   token t attends to min(t + 1, topk) of the rows 0 .. t, the other slots hold an out-of-range value
                     (the reference script's pattern; with "varlen" inside every sequence)
          "skewed"   half of the slots among the last 4096 rows, half among the rest (long context)
  unused  share of the slots that are -1 on top of that
  n_seq, split   "varlen" only: number of packed sequences and the seed of their lengths
"""
import math
import random

import torch

from test_operator_b200 import op
from test_operator_b200.inputs import forward_o_lse

D_QK, D_V = 576, 512
RECENT = 4096          # "skewed": rows that half of the slots come from
BWD_FLOPS, FWD_FLOPS = 5504, 2176   # per (query, head, slot in use): multiply-adds of the five / two contractions


def _case(name, path, s_q, s_kv, h_q, topk, pattern, unused=0.0, n_seq=1, split=0):
    c = dict(path=path, s_q=s_q, s_kv=s_kv, h_q=h_q, topk=topk, pattern=pattern, unused=unused, n_seq=n_seq, split=split)
    return dict(c, name=name) if name else c


def listed():
    return [
        # decoding: the next tokens of a request (a few speculative ones at a time) against a long kv cache.  Pure latency.
        _case("decode_8_tokens", "fwd", 8, 16384, 128, 2048, "offset"),
        # the smallest configuration of the benchmark: a unit test's or a toy model's step, host path and launches only
        _case("bwd_tiny_16_heads", "bwd", 64, 256, 16, 64, "uniform", unused=0.10),
        # training on packed documents of different lengths, each with its own causal prefix
        _case("bwd_packed_documents", "varlen", 1531, 1531, 128, 1000, "prefix", n_seq=6, split=3),
        # a training step of a small 64-head layer through autograd, with sizes that fit no tile
        _case("train_step_64_heads", "train", 777, 3001, 64, 600, "offset"),
        # prefill of a long prompt's last block, the forward of the headline configuration
        _case("prefill_128_heads", "fwd", 4096, 32768, 128, 2048, "offset", unused=0.05),
        # the 64-head configuration of the benchmark: every kv row is chosen by a quarter of the queries
        _case("bwd_64_heads", "bwd", 4096, 8192, 64, 2048, "uniform"),
        # what the reference's own script runs, through the module of its name and with its default arguments
        _case("module_reference_script", "module", 4096, 8192, 128, 2048, "prefix"),
        # the headline configuration
        _case("bwd_128_heads", "bwd", 4096, 32768, 128, 2048, "offset", unused=0.05),
        # one sequence of the batch-sharded configuration: what a GPU of an eight-GPU node works on
        _case("bwd_128_heads_8192_queries", "bwd", 8192, 16384, 128, 2048, "uniform"),
        # a debugging or regression run that has to repeat bit for bit
        _case("bwd_repeatable", "repro", 1024, 8192, 128, 2048, "uniform", unused=0.10),
        # the operator on host buffers: inputs come over PCIe and gradients go back with every call
        _case("bwd_host_buffers", "host", 1024, 32768, 128, 2048, "offset", unused=0.05),
        # the pre-pass that turns the headline configuration's pattern into a list of slots per kv row
        _case("inverse_of_the_pattern", "inverse", 4096, 32768, 128, 2048, "offset", unused=0.05),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    path = rng.choices(["bwd", "module", "varlen", "repro", "host", "fwd", "train", "inverse"],
                       weights=[5, 3, 3, 1, 1, 5, 4, 2])[0]
    h_q = rng.choices([16, 64, 128, 8 * rng.randint(1, 16)], weights=[2, 3, 4, 2])[0]
    topk = rng.choice([2048, 1024, 512, _log_int(rng, 16, 2048), _log_int(rng, 16, 2048)])
    most = {"repro": 1024, "host": 1024, "train": 3072}.get(path, 8192)
    s_q = _log_int(rng, 16 if path == "varlen" else 1, most)
    pattern = "prefix" if path == "varlen" else rng.choice(["uniform", "offset", "offset", "skewed", "prefix"])
    if path == "varlen":
        s_kv = s_q
    elif pattern == "prefix":
        s_kv = s_q + rng.choice([0, rng.randint(0, s_q)])
    else:       # rows for distinct slots, and every query's own position inside the kv
        s_kv = _log_int(rng, max(64, s_q + topk), 65536)
    unused = rng.choice([0.0, 0.05, 0.10])
    n_seq = rng.randint(2, 8) if path == "varlen" else 1
    return _case(None, path, s_q, s_kv, h_q, topk, pattern, 0.0 if path == "varlen" else unused, n_seq,
                 rng.randint(1, 999) if path == "varlen" else 0)


def _lengths(case):
    """Lengths of the packed sequences, at least one token each."""
    n, total = case["n_seq"], case["s_q"]
    r = random.Random(case["split"])
    cuts = sorted(r.sample(range(1, total), n - 1)) if n > 1 else []
    return [b - a for a, b in zip([0] + cuts, cuts + [total])]


def _distinct(limits, k, width, gen, device):
    """Row i: min(k, limits[i]) distinct integers below limits[i] in random order, then -1."""
    n = limits.numel()
    out = torch.full((n, k), -1, dtype=torch.int32, device=device)
    kk = min(k, width)
    step = max(1, (1 << 26) // max(width, 1))
    col = torch.arange(width, device=device)
    for r0 in range(0, n, step):
        lim = limits[r0:r0 + step].unsqueeze(1)
        keys = torch.rand(lim.shape[0], width, generator=gen, device=device).masked_fill_(col >= lim, -1.0)
        val, idx = keys.topk(kk, dim=1)
        out[r0:r0 + step, :kk] = torch.where(val >= 0, idx, -1).to(torch.int32)
    return out


def _indices(pattern, s_q, s_kv, topk, unused, gen, device):
    rows = torch.arange(s_q, device=device)
    if pattern == "skewed":
        half, recent = topk // 2, min(RECENT, s_kv // 2)
        a = _distinct(torch.full_like(rows, recent), half, recent, gen, device)
        b = _distinct(torch.full_like(rows, s_kv - recent), topk - half, s_kv - recent, gen, device)
        idx = torch.cat([torch.where(a >= 0, a + (s_kv - recent), a), b], dim=1)
        idx = idx.gather(1, torch.rand(idx.shape, generator=gen, device=device).argsort(dim=1))
    else:
        limits = {"uniform": torch.full_like(rows, s_kv), "offset": s_kv - s_q + rows, "prefix": rows + 1}[pattern]
        idx = _distinct(limits, topk, min(s_kv, int(limits.max())), gen, device)
        if pattern == "prefix":
            idx = torch.where(idx >= 0, idx, s_kv)
    if unused:
        idx = torch.where(torch.rand(idx.shape, generator=gen, device=device) < unused, -1, idx)
    return idx.to(torch.int32).contiguous()


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    path, s_q, s_kv, h_q, topk = (case[k] for k in ("path", "s_q", "s_kv", "h_q", "topk"))
    start = 0 if case["pattern"] == "prefix" else None      # causal rule: from the query's own row, or range check only
    st = {"path": path, "start": start, "s_kv": s_kv}
    if path == "varlen":
        lens = _lengths(case)
        st["cu"] = [sum(lens[:i]) for i in range(len(lens) + 1)]
        st["idx"] = torch.cat([_indices("prefix", n, n, topk, 0.0, gen, dev) for n in lens])
    else:
        st["idx"] = _indices(case["pattern"], s_q, s_kv, topk, case["unused"], gen, dev)
    if path == "inverse":
        return st
    new = lambda *shape: torch.randn(*shape, generator=gen, device=dev).to(torch.bfloat16)  # noqa: E731
    q, kv = new(s_q, h_q, D_QK), new(s_kv, D_QK)
    st.update(q=q, kv=kv)
    if path == "fwd":
        return st
    st["dO"] = new(s_q, h_q, D_V)
    if path == "train":
        q.requires_grad_()
        kv.requires_grad_()
        return st
    if path == "varlen":
        parts = [forward_o_lse(q[a:b], kv[a:b], st["idx"][a:b], q_start_index_s=0) for a, b in zip(st["cu"], st["cu"][1:])]
        st["O"], st["lse"] = (torch.cat(p) for p in zip(*parts))
        st["lse"] *= math.log(2.0)          # this caller keeps natural logarithms
    else:
        st["O"], st["lse"] = forward_o_lse(q, kv, st["idx"], q_start_index_s=start)
    if path == "module":
        import mla_bwd_cuda
        st["call"] = mla_bwd_cuda.mla_bwd
    if path == "host":
        st["dev"] = dev
        for k in ("q", "kv", "dO", "lse", "O", "idx"):
            st[k] = st[k].cpu().pin_memory()
        st["dq"] = torch.empty(q.shape, dtype=torch.bfloat16, pin_memory=True)
        st["dkv"] = torch.empty(kv.shape, dtype=torch.float32, pin_memory=True)
    return st


def run(st):
    path = st["path"]
    if path == "inverse":
        return op.index_inverse(st["idx"], st["s_kv"], st["start"])
    q, kv, idx, start = st["q"], st["kv"], st["idx"], st["start"]
    if path == "fwd":
        return op.mla_fwd(q, kv, idx, q_start_index_s=start)
    if path == "train":
        o = op.sparse_mla(q, kv, idx, q_start_index_s=start)
        return (o.detach(),) + torch.autograd.grad(o, (q, kv), st["dO"])
    args = (q, kv, st["dO"], st["lse"], st["O"], idx)
    if path == "bwd":
        return op.mla_bwd(*args, q_start_index_s=start)
    if path == "module":
        return st["call"](*args) if start == 0 else st["call"](*args, q_start_index_s=start)
    if path == "varlen":
        return op.mla_bwd_varlen(*args, st["cu"], st["cu"], lse_is_base2=False)
    if path == "repro":
        return op.mla_bwd(*args, q_start_index_s=start, deterministic=True)
    return op.mla_bwd_host(*args, st["dev"], q_start_index_s=start, out_dq=st["dq"], out_dkv=st["dkv"])


def work(case):
    path, s_q, s_kv, h_q, topk = (case[k] for k in ("path", "s_q", "s_kv", "h_q", "topk"))
    if path == "varlen":
        used = sum(min(t + 1, topk) for n in _lengths(case) for t in range(n))
    elif case["pattern"] == "prefix":
        used = sum(min(t + 1, topk) for t in range(s_q))
    elif case["pattern"] == "skewed":
        recent = min(RECENT, s_kv // 2)
        used = s_q * (min(topk // 2, recent) + min(topk - topk // 2, s_kv - recent))
    else:
        used = s_q * min(topk, s_kv)
    used *= 1.0 - case["unused"]
    idx = 4 * s_q * topk
    if path == "inverse":
        return {"bytes": 2 * idx + 4 * (s_kv + 1), "flops": 0}
    kv = min(s_kv, used)                            # rows that have to be read
    rows = s_q * h_q
    fwd_in, fwd_out = 2 * D_QK * (rows + kv) + idx, 2 * D_V * rows
    if path == "fwd":
        return {"bytes": fwd_in + fwd_out + 4 * rows, "flops": FWD_FLOPS * used * h_q}
    if path == "train":
        return {"bytes": fwd_in + fwd_out + 2 * D_V * rows + 2 * D_QK * (rows + s_kv),
                "flops": (FWD_FLOPS + BWD_FLOPS) * used * h_q}
    return {"bytes": fwd_in + 2 * 2 * D_V * rows + 4 * rows + 2 * D_QK * rows + 4 * D_QK * s_kv, "flops": BWD_FLOPS * used * h_q}


def tolerance(case):
    # whole numbers are exact; everything else passes through bf16 (o and dQ are bf16, and the probabilities and their
    # gradients are rounded to bf16 before the products that make dKV)
    return "exact" if case["path"] == "inverse" else {"rel": 0.01}
