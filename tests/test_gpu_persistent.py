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
