"""The attention work this library is timed on: what its users have it do, through its public entry points.

Kinds of case:
  bwd     ops.fa3_bwd on tensors that are on the GPU already (the call behind shaobo_fa3_bwd_v2)
  fwd     ops.fa3_fwd, the forward that produces O and the log-sum-exp
  step    torch_binding.attention forward and its gradients through autograd: one layer of a training step
  packed  ops.fa3_fwd_varlen and ops.fa3_bwd_varlen over sequences of different lengths laid end to end
  host    ops.HostBackwardC: the backward of tensors that live in pinned host memory, copies included
"""
import math

import numpy as np
import torch

from flash_attention3_b200 import ops, torch_binding

DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}


def _case(name, kind, b, hq, hkv, sq, sk, d, dtype, causal, layout="bhsd", window=(-1, -1), softcap=0.0,
          deterministic=False, lengths=""):
    c = {"kind": kind, "b": b, "hq": hq, "hkv": hkv, "sq": sq, "sk": sk, "d": d, "dtype": dtype, "causal": causal,
         "layout": layout, "window_left": window[0], "window_right": window[1], "softcap": softcap,
         "deterministic": deterministic, "lengths": lengths}
    return dict(c, name=name) if name else c


def listed():
    return [
        # a single head: the smallest call, bound by launches and host work
        _case("bwd_1head_1k", "bwd", 1, 1, 1, 1024, 1024, 128, "fp16", True),
        # the default benchmark shape: fewer key tiles than SMs
        _case("bwd_4heads_2k", "bwd", 1, 4, 4, 2048, 2048, 128, "fp16", True),
        # full attention over whole tiles (encoders), both head dimensions
        _case("bwd_full_4k_d128", "bwd", 4, 16, 16, 4096, 4096, 128, "bf16", False),
        _case("bwd_full_4k_d64", "bwd", 4, 16, 16, 4096, 4096, 64, "bf16", False),
        # long causal sequences with four query heads per key head: the largest call
        _case("bwd_gqa_8k", "bwd", 2, 32, 8, 8192, 8192, 128, "bf16", True),
        # bitwise reproducible gradients (debugging, regression runs)
        _case("bwd_deterministic_2k", "bwd", 2, 16, 16, 2048, 2048, 128, "bf16", True, deterministic=True),
        # forward alone (evaluation, activation recomputation): small and long
        _case("fwd_4heads_2k", "fwd", 1, 4, 4, 2048, 2048, 128, "fp16", True),
        _case("fwd_gqa_8k", "fwd", 2, 32, 8, 8192, 8192, 128, "bf16", True),
        # one layer of a training step, token-major tensors, ragged and unequal lengths
        _case("step_ragged_1k_d64", "step", 2, 16, 8, 1111, 1300, 64, "bf16", True, layout="bshd"),
        # one layer with local attention and capped scores
        _case("step_window_softcap_4k", "step", 1, 16, 8, 4096, 4096, 128, "bf16", True, layout="bshd",
              window=(1023, 0), softcap=30.0),
        # a batch of documents of different lengths, packed
        _case("packed_documents", "packed", 9, 16, 4, 2048, 2048, 128, "bf16", True,
              lengths="2048,77,1500,300,1024,513,129,900,1701"),
        # gradients of host-resident tensors, the default benchmark shape
        _case("host_4heads_2k", "host", 1, 4, 4, 2048, 2048, 128, "fp16", True),
    ]


# A drawn case does at most the arithmetic of the largest listed one, in the time of that one: forms that do
# more work than `work` counts (the reproducible path computes the scores twice, narrow heads and capped scores
# take longer per product) get a smaller share.
_MOST_FLOPS = 2.7e12
_MOST_HOST_BYTES = 96e6


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["bwd", "fwd", "step", "packed", "host"], [35, 20, 20, 15, 10])[0]
    while True:
        d = rng.choice([64, 128])
        dtype = rng.choice(["fp16", "bf16", "bf16"])
        causal = rng.random() < 0.7
        group = rng.choice([1, 1, 2, 4, 8])
        sq = _log_int(rng, 64, 8192)
        if rng.random() < 0.4:
            sq = max(128, sq // 128 * 128)
        sk = sq if rng.random() < 0.8 else max(sq, _log_int(rng, 64, 8192))
        layout = rng.choice(["bhsd", "bshd"])
        window, softcap, deterministic, lengths = (-1, -1), 0.0, False, ""
        b = _log_int(rng, 1, 16)
        if kind == "packed":
            seqs = [_log_int(rng, 16, max(64, sq)) for _ in range(_log_int(rng, 2, 24))]
            lengths, b, sq, layout = ",".join(map(str, seqs)), len(seqs), max(seqs), "bshd"
            sk = sq
        elif kind == "host":
            sk, layout = sq, "bhsd"
        elif rng.random() < 0.2:
            window = (_log_int(rng, 64, 4096), 0 if causal else _log_int(rng, 64, 4096))
        if kind in ("fwd", "step") and rng.random() < 0.15:
            softcap = rng.choice([15.0, 30.0, 50.0])
        if kind == "bwd" and rng.random() < 0.2:
            deterministic = True
        hkv = _log_int(rng, 1, 32)
        case = _case("", kind, b, hkv * group, hkv, sq, sk, d, dtype, causal, layout, window, softcap, deterministic, lengths)
        w = work(case)
        share = (0.4 if deterministic else 1.0) * (0.5 if d == 64 else 1.0) * (0.5 if softcap else 1.0)
        if w["flops"] <= share * _MOST_FLOPS and w["bytes"] <= (_MOST_HOST_BYTES if kind == "host" else 1.5e9):
            return case


def _shapes(case):
    q = (case["b"], case["sq"], case["hq"], case["d"]) if case["layout"] == "bshd" else (case["b"], case["hq"], case["sq"], case["d"])
    k = (case["b"], case["sk"], case["hkv"], case["d"]) if case["layout"] == "bshd" else (case["b"], case["hkv"], case["sk"], case["d"])
    return q, k


def prepare(case, seed):
    dtype, kind = DTYPES[case["dtype"]], case["kind"]
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(shape):
        return torch.randn(shape, device="cuda", generator=gen).to(dtype)

    state = {"case": case, "window": (case["window_left"], case["window_right"])}
    if kind == "packed":
        lengths = [int(x) for x in case["lengths"].split(",")]
        total = sum(lengths)
        state["cu"] = torch.tensor(np.concatenate([[0], np.cumsum(lengths)]), dtype=torch.int32, device="cuda")
        state["max"] = max(lengths)
        q, k = (total, case["hq"], case["d"]), (total, case["hkv"], case["d"])
    else:
        q, k = _shapes(case)
    state["q"], state["k"], state["v"] = normal(q), normal(k), normal(k)
    if kind != "fwd":
        state["dout"] = normal(q)
    if kind == "step":
        for n in ("q", "k", "v"):
            state[n].requires_grad_(True)
    if kind in ("bwd", "host"):
        # what the forward pass left behind
        state["out"], state["lse"] = ops.fa3_fwd(state["q"], state["k"], state["v"], case["causal"], layout=case["layout"],
                                                 window=state["window"], softcap=case["softcap"])
    if kind == "host":
        names = ("dout", "q", "k", "v", "out", "lse")
        on_host = [state.pop(n).cpu().pin_memory() for n in names]
        grads = [torch.empty_like(on_host[i]).pin_memory() for i in (1, 2, 3)]
        state["host"] = on_host + grads
        state["call"] = ops.HostBackwardC(case["b"], case["hq"], case["hkv"], case["sq"], case["d"], dtype, case["causal"])
    return state


def run(state):
    case = state["case"]
    kind, causal = case["kind"], case["causal"]
    if kind == "bwd":
        return ops.fa3_bwd(state["dout"], state["q"], state["k"], state["v"], state["out"], state["lse"], causal,
                           deterministic=case["deterministic"], layout=case["layout"], window=state["window"],
                           softcap=case["softcap"])
    if kind == "fwd":
        return ops.fa3_fwd(state["q"], state["k"], state["v"], causal, layout=case["layout"], window=state["window"],
                           softcap=case["softcap"])
    if kind == "step":
        out = torch_binding.attention(state["q"], state["k"], state["v"], causal=causal, window=state["window"],
                                      softcap=case["softcap"], layout=case["layout"])
        dq, dk, dv = torch.autograd.grad(out, (state["q"], state["k"], state["v"]), state["dout"])
        return out.detach(), dq, dk, dv
    if kind == "packed":
        cu, longest = state["cu"], state["max"]
        out, lse = ops.fa3_fwd_varlen(state["q"], state["k"], state["v"], cu, cu, longest, longest, causal)
        dq, dk, dv = ops.fa3_bwd_varlen(state["dout"], state["q"], state["k"], state["v"], out, lse, cu, cu, longest,
                                        longest, causal)
        return out, lse, dq, dk, dv
    state["call"](*state["host"])
    return state["host"][6:]


def _visible_pairs(sq, sk, causal, window):
    """(query, key) pairs that attend: query i sees keys i+off-left .. i+off+right, off = sk - sq."""
    left, right = window
    if causal:
        right = 0
    i = np.arange(sq, dtype=np.int64) + (sk - sq)
    lo = np.maximum(i - left, 0) if left >= 0 else np.zeros_like(i)
    hi = np.minimum(i + right, sk - 1) if right >= 0 else np.full_like(i, sk - 1)
    return float(np.maximum(hi - lo + 1, 0).sum())


def work(case):
    kind, d, hq, hkv = case["kind"], case["d"], case["hq"], case["hkv"]
    window = (case["window_left"], case["window_right"])
    if kind == "packed":
        lengths = [int(x) for x in case["lengths"].split(",")]
        pairs = sum(_visible_pairs(n, n, case["causal"], window) for n in lengths)
        rows_q = rows_k = sum(lengths)
    else:
        pairs = case["b"] * _visible_pairs(case["sq"], case["sk"], case["causal"], window)
        rows_q, rows_k = case["b"] * case["sq"], case["b"] * case["sk"]
    q_bytes, kv_bytes, lse_bytes = 2.0 * rows_q * hq * d, 2.0 * rows_k * hkv * d, 4.0 * rows_q * hq
    forward = {"flops": 4.0 * pairs * hq * d, "bytes": 2 * q_bytes + 2 * kv_bytes + lse_bytes}    # q, k, v in; out, lse out
    backward = {"flops": 10.0 * pairs * hq * d, "bytes": 4 * q_bytes + 4 * kv_bytes + lse_bytes}  # q, k, v, out, dout, lse in; dq, dk, dv out
    if kind == "fwd":
        return forward
    if kind in ("bwd", "host"):
        return backward
    # both directions: q, k, v, dout in; out, lse, dq, dk, dv out
    return {"flops": forward["flops"] + backward["flops"], "bytes": 4 * q_bytes + 4 * kv_bytes + lse_bytes}


def tolerance(case):
    # 16-bit storage of the results and of P and dS inside: 8 significant bits for bf16, 11 for fp16
    return {"rel": 1e-2} if case["dtype"] == "bf16" else {"rel": 2e-3}

