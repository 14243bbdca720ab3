"""The five-GEMM kernel where CTAs take over the tiles of blocks that have not started (more tiles than SMs): one tile more than
the SMs of a B200, tiles of one step, many tiles per CTA, key tiles that nobody sees, packed sequences with blocks without rows.
dK and dV do not depend on which CTA had a tile: repeated calls agree bit for bit."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# (b, hq, hkv, sq, sk, d, dtype, causal, layout, window)
CASES = [
    (1, 149, 149, 128, 128, 128, "bf16", True, "bhsd", (-1, -1)),
    (1, 149, 149, 128, 128, 64, "fp16", False, "bshd", (-1, -1)),
    (2, 160, 160, 128, 256, 128, "fp16", False, "bhsd", (-1, -1)),
    (4, 48, 48, 256, 384, 64, "bf16", False, "bhsd", (-1, -1)),
    (2, 60, 30, 300, 900, 128, "bf16", True, "bshd", (-1, -1)),
    (1, 40, 40, 700, 700, 128, "fp16", True, "bhsd", (-1, -1)),
    (1, 64, 64, 256, 1024, 128, "bf16", False, "bhsd", (8, 64)),   # key tiles without queries
    (1, 80, 80, 515, 300, 128, "fp16", True, "bshd", (100, -1)),   # queries without keys
]


@pytest.mark.parametrize("deterministic", [False, True])
@pytest.mark.parametrize("b,hq,hkv,sq,sk,d,dtype,causal,layout,window", CASES)
def test_tiles_taken_over(b, hq, hkv, sq, sk, d, dtype, causal, layout, window, deterministic):
    from tests.helpers import Problem, assert_parity, run_v2
    prob = Problem(b, hq, hkv, sq, d, dtype, causal, seed=31 + sq + sk, sk=sk, layout=layout, window=window)
    first = run_v2(prob, deterministic=deterministic)
    assert_parity(first, prob, label=f"{(b, hq, hkv, sq, sk, d, dtype, causal, layout, window)}")
    for _ in range(3):
        again = run_v2(prob, deterministic=deterministic)
        assert not deterministic or np.array_equal(again["dq"], first["dq"])
        assert np.array_equal(again["dk"], first["dk"]) and np.array_equal(again["dv"], first["dv"])


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("causal", [False, True])
def test_packed_tiles_taken_over(causal, d):
    from flash_attention3_b200 import ops
    from oracle import golden
    from tests.helpers import dev, host
    from tests.test_gpu_varlen import packed_problem
    seqs = [(900, 900)] + [(5, 7), (130, 130), (1, 9), (257, 300), (64, 129)] * 4
    packed, refs, cu_q, cu_k = packed_problem(seqs, 4, 2, d, "bf16", causal, (-1, -1), seed=91)
    t = {n: dev(packed[n], "bf16") for n in ("q", "k", "v", "dout", "out")}
    cu = [torch.from_numpy(c).cuda() for c in (cu_q, cu_k)]
    call = lambda: ops.fa3_bwd_varlen(t["dout"], t["q"], t["k"], t["v"], t["out"], dev(packed["lse"]), *cu, 900, 900, causal, sync=True)
    got = [host(g) for g in call()]
    for i, ref in enumerate(refs):
        for name, g, c in zip(("dq", "dk", "dv"), got, (cu_q, cu_k, cu_k)):
            assert golden.check_gradient(g[c[i]:c[i + 1]].transpose(1, 0, 2)[None], ref[name], "bf16")["pass"], (i, name)
    again = [host(g) for g in call()]
    assert np.array_equal(got[1], again[1]) and np.array_equal(got[2], again[2])


# (b, hq, hkv, s, d, layout, used queries, used keys): entries without queries, without keys, with one query, whole ones
USED = [
    (7, 24, 12, 384, 64, "bhsd", [0, 384, 100, 257, 0, 1, 384], [384, 0, 384, 129, 0, 300, 200]),
    (7, 24, 24, 384, 128, "bshd", [384, 130, 0, 384, 5, 256, 0], [20, 384, 128, 0, 260, 384, 7]),
]


@pytest.mark.parametrize("b,hq,hkv,s,d,layout,used_q,used_k", USED)
def test_used_lengths(b, hq, hkv, s, d, layout, used_q, used_k):
    """Tiles without work, and rows behind a used length, between tiles that CTAs take over, forward and both backwards: every entry is
    the oracle's on the truncated sequences, exact zeros (-inf for the log-sum-exp) behind them."""
    from flash_attention3_b200 import ops
    from oracle import golden
    from tests.helpers import dev, host, poison
    dtype, scale = "bf16", 1.0 / float(np.sqrt(d))
    q, k, v, do = golden.seeded_inputs(61, b, hq, hkv, s, d, dtype)
    to = lambda x: dev(np.ascontiguousarray(x.transpose(0, 2, 1, 3)) if layout == "bshd" else x, dtype)
    back = lambda t: host(t).transpose(0, 2, 1, 3) if layout == "bshd" else host(t)
    tq, tk, tv, tdo = (to(x) for x in (q, k, v, do))
    used = [torch.tensor(u, dtype=torch.int32, device="cuda") for u in (used_q, used_k)]
    out, lse = ops.fa3_fwd(tq, tk, tv, True, layout=layout, seqused_q=used[0], seqused_k=used[1], sync=True)
    grads = [[back(g) for g in ops.fa3_bwd(tdo, tq, tk, tv, out, lse, True, layout=layout, seqused_q=used[0], seqused_k=used[1], sync=True,
                                           outputs=tuple(poison(t.shape, t.dtype) for t in (tq, tk, tv)), deterministic=deterministic)]
             for deterministic in (False, True)]
    out, lse = back(out), host(lse)
    for i in range(b):
        uq, uk = used_q[i], used_k[i]
        assert (out[i, :, uq:] == 0).all() and np.isneginf(lse[i, :, uq:]).all(), (i, "forward")
        for dq, dk, dv in grads:
            assert (dq[i, :, uq:] == 0).all() and (dk[i, :, uk:] == 0).all() and (dv[i, :, uk:] == 0).all(), (i, "behind")
        if uq == 0 or uk == 0:
            assert (out[i] == 0).all() and np.isneginf(lse[i]).all() and all((g[i] == 0).all() for gs in grads for g in gs), i
            continue
        ref = golden.backward(q[i:i + 1, :, :uq], k[i:i + 1, :, :uk], v[i:i + 1, :, :uk], do[i:i + 1, :, :uq], True, scale, dtype)
        assert golden.check_gradient(out[i:i + 1, :, :uq], ref["out"], dtype)["pass"], (i, "out")
        finite = np.isfinite(ref["lse"])
        assert np.array_equal(np.isfinite(lse[i:i + 1, :, :uq]), finite)
        assert np.abs(lse[i:i + 1, :, :uq][finite] - ref["lse"][finite]).max() <= 2e-3, (i, "lse")
        for gs in grads:
            for name, g, n in zip(("dq", "dk", "dv"), gs, (uq, uk, uk)):
                assert golden.check_gradient(g[i:i + 1, :, :n], ref[name], dtype)["pass"], (i, name)


@pytest.mark.parametrize("d,causal", [(64, False), (128, True)])
def test_streams_and_graphs(d, causal):
    """Calls whose CTAs take over tiles, on four streams at once and replayed from a graph: what one call alone gives, bit for bit (dQ of
    the five-GEMM kernel, whose order of addition is free, left out)."""
    from flash_attention3_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(8)
    q, k, v, do = (torch.randn((2, 160, 384, d), device="cuda", generator=gen).bfloat16() for _ in range(4))

    def call():
        out, lse = ops.fa3_fwd(q, k, v, causal)
        _, dk, dv = ops.fa3_bwd(do, q, k, v, out, lse, causal)
        return out, lse, dk, dv, *ops.fa3_bwd(do, q, k, v, out, lse, causal, deterministic=True)

    alone = call()
    torch.cuda.synchronize()
    streams, results = [torch.cuda.Stream() for _ in range(4)], []
    for i in range(8):
        with torch.cuda.stream(streams[i % 4]):
            results.append(call())
    torch.cuda.synchronize()
    with torch.cuda.stream(streams[0]):
        call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        replayed = call()
    for _ in range(3):
        for t in replayed:
            t.fill_(float("nan"))
        graph.replay()
    torch.cuda.synchronize()
    for got in (*results, replayed):
        assert all(torch.equal(a, b) for a, b in zip(got, alone))
