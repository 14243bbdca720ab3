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


# (rows of the slot, rows used) of queries and keys
USED_PACKED = [((384, 0), (384, 384)), ((130, 130), (260, 200)), ((5, 5), (7, 0)), ((256, 100), (128, 128)), ((300, 300), (300, 150)),
               ((64, 64), (500, 333)), ((384, 384), (384, 77)), ((130, 1), (260, 260)), ((5, 0), (7, 7)), ((256, 256), (128, 100)),
               ((300, 17), (300, 300)), ((64, 60), (500, 64))]
USED_PACKED_HEADS = (24, 12)


@pytest.mark.parametrize("d", [64, 128])
def test_used_lengths_of_packed_sequences(d):
    """The same with the entries' slots laid end to end (C ABI)."""
    import ctypes
    from flash_attention3_b200 import capi
    from oracle import golden
    from tests.helpers import dev, host, poison
    (hq, hkv), scale, lib = USED_PACKED_HEADS, 1.0 / float(np.sqrt(d)), capi.load()
    slots = [np.concatenate([[0], np.cumsum([e[i][0] for e in USED_PACKED])]).astype(np.int32) for i in (0, 1)]
    total_q, total_k = int(slots[0][-1]), int(slots[1][-1])
    q, k, v, do = (x[0] for x in golden.seeded_inputs(77, 1, hq, hkv, total_q, d, "bf16", sk=total_k))
    rows_first = lambda x: dev(np.ascontiguousarray(x.transpose(1, 0, 2)), "bf16")
    tq, tk, tv, tdo = (rows_first(x) for x in (q, k, v, do))
    ints = lambda x: torch.tensor(np.asarray(x), dtype=torch.int32, device="cuda")
    cu, used = [ints(s) for s in slots], [ints([e[i][1] for e in USED_PACKED]) for i in (0, 1)]
    longest = [max(e[i][0] for e in USED_PACKED) for i in (0, 1)]
    params = capi.new_params(batch=len(USED_PACKED), num_heads_q=hq, num_heads_kv=hkv, head_dim_qk=d, head_dim_v=d, causal=1,
                             dtype=capi.DTYPE_BF16, cu_seqlens_q=cu[0].data_ptr(), cu_seqlens_k=cu[1].data_ptr(), total_q=total_q,
                             total_k=total_k, seqlen_q=longest[0], seqlen_k=longest[1], max_seqlen_q=longest[0],
                             max_seqlen_k=longest[1], seqused_q=used[0].data_ptr(), seqused_k=used[1].data_ptr(), sync_after_launch=1)
    vp = lambda t: ctypes.c_void_p(t.data_ptr())
    out, lse = poison(tq.shape, tq.dtype), poison((hq, total_q), torch.float32)
    assert lib.shaobo_fa3_b200_fwd(vp(tq), vp(tk), vp(tv), vp(out), vp(lse), ctypes.byref(params)) == capi.STATUS_SUCCESS
    results = []
    for deterministic in (0, 1):
        params.deterministic = deterministic
        need = lib.shaobo_fa3_bwd_v2_workspace_bytes(ctypes.byref(params))
        workspace = torch.full((need,), 0xFF, dtype=torch.uint8, device="cuda")
        params.workspace, params.workspace_bytes = workspace.data_ptr(), need
        grads, delta = [poison(t.shape, t.dtype) for t in (tq, tk, tv)], poison(lse.shape, torch.float32)
        torch.cuda.synchronize()
        assert lib.shaobo_fa3_bwd_v2(vp(tdo), vp(tq), vp(tk), vp(tv), vp(out), vp(lse), *map(vp, grads), vp(delta),
                                     ctypes.byref(params)) == capi.STATUS_SUCCESS
        torch.cuda.synchronize()
        assert lib.shaobo_fa3_b200_device_error(1) == 0
        results.append([host(g).transpose(1, 0, 2) for g in grads])
    out, lse = host(out).transpose(1, 0, 2), host(lse)
    for i, ((slot_q, uq), (slot_k, uk)) in enumerate(USED_PACKED):
        q0, k0 = slots[0][i], slots[1][i]
        assert (out[:, q0 + uq:q0 + slot_q] == 0).all() and np.isneginf(lse[:, q0 + uq:q0 + slot_q]).all(), (i, "forward")
        ref = None if uq == 0 or uk == 0 else golden.backward(q[None, :, q0:q0 + uq], k[None, :, k0:k0 + uk], v[None, :, k0:k0 + uk],
                                                              do[None, :, q0:q0 + uq], True, scale, "bf16")
        if ref is None:
            assert (out[:, q0:q0 + slot_q] == 0).all() and np.isneginf(lse[:, q0:q0 + slot_q]).all(), i
        else:
            assert golden.check_gradient(out[None, :, q0:q0 + uq], ref["out"], "bf16")["pass"], (i, "out")
        for grads in results:
            for name, g, first, n, slot in zip(("dq", "dk", "dv"), grads, (q0, k0, k0), (uq, uk, uk), (slot_q, slot_k, slot_k)):
                assert (g[:, first + n:first + slot] == 0).all(), (i, name, "behind")
                if ref is None:
                    assert (g[:, first:first + slot] == 0).all(), (i, name)
                else:
                    assert golden.check_gradient(g[None, :, first:first + n], ref[name], "bf16")["pass"], (i, name)
