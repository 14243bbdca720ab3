"""The forward where CTAs take over the pairs of query tiles of CTAs that have not started (twice as many pairs as SMs): pairs
with one tile, tiles of one key tile, queries without keys, blocks without rows.  A tile's result does not depend on which CTA had
it: repeated calls agree bit for bit."""
import numpy as np
import pytest
import torch

from oracle import golden

pytestmark = pytest.mark.gpu

# (b, hq, hkv, sq, sk, d, dtype, causal, layout, window)
CASES = [
    (1, 300, 300, 128, 128, 64, "bf16", True, "bhsd", (-1, -1)),
    (1, 300, 300, 128, 128, 128, "fp16", False, "bshd", (-1, -1)),
    (1, 150, 150, 512, 512, 64, "fp16", True, "bshd", (-1, -1)),     # one and two steps, then three and four
    (2, 80, 40, 512, 384, 128, "bf16", False, "bhsd", (-1, -1)),
    (1, 100, 100, 700, 300, 64, "fp16", True, "bhsd", (-1, -1)),     # queries without keys
    (1, 100, 50, 600, 900, 128, "bf16", True, "bshd", (200, -1)),
    (1, 160, 160, 300, 300, 64, "bf16", True, "bhsd", (-1, -1)),
]


@pytest.mark.parametrize("b,hq,hkv,sq,sk,d,dtype,causal,layout,window", CASES)
def test_tiles_taken_over(b, hq, hkv, sq, sk, d, dtype, causal, layout, window):
    from flash_attention3_b200 import ops
    from tests.helpers import dev, host
    q, k, v, _ = golden.seeded_inputs(41 + sq, b, hq, hkv, sq, d, dtype, sk=sk)
    scale = 1.0 / float(np.sqrt(d))
    ref = golden.backward(q, k, v, np.zeros_like(q), causal, scale, dtype, window)
    f = (lambda x: np.ascontiguousarray(x.transpose(0, 2, 1, 3))) if layout == "bshd" else (lambda x: x)
    t = [dev(f(x), dtype) for x in (q, k, v)]
    call = lambda: ops.fa3_fwd(*t, causal, scale, layout=layout, window=window, sync=True)
    out, lse = call()
    assert golden.check_gradient(f(host(out)) if layout == "bshd" else host(out), ref["out"], dtype)["pass"]
    finite = np.isfinite(ref["lse"])
    assert np.array_equal(np.isfinite(host(lse)), finite)
    assert np.abs(host(lse)[finite] - ref["lse"][finite]).max() <= 3e-3
    for _ in range(5):
        again, lse2 = call()
        assert torch.equal(again, out) and torch.equal(lse2, lse)


PACKED = [(700, 700)] + [(5, 7), (130, 130), (1, 9), (257, 300), (64, 129)] * 5
PACKED_HEADS = [8, 24]  # 8: too few pairs with rows, one per CTA; 24: taken over


@pytest.mark.parametrize("heads", PACKED_HEADS)
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("causal", [False, True])
def test_packed_tiles_taken_over(causal, d, heads):
    from flash_attention3_b200 import ops
    from tests.helpers import dev, host
    from tests.test_gpu_varlen import packed_problem
    packed, refs, cu_q, cu_k = packed_problem(PACKED, heads, heads // 2, d, "bf16", causal, (-1, -1), seed=17)
    t = {n: dev(packed[n], "bf16") for n in ("q", "k", "v")}
    cu = [torch.from_numpy(c).cuda() for c in (cu_q, cu_k)]
    call = lambda: ops.fa3_fwd_varlen(t["q"], t["k"], t["v"], *cu, 700, 700, causal, sync=True)
    out, lse = call()
    for i, ref in enumerate(refs):
        rows = slice(cu_q[i], cu_q[i + 1])
        assert golden.check_gradient(host(out)[rows].transpose(1, 0, 2)[None], ref["out"], "bf16")["pass"], i
        finite = np.isfinite(ref["lse"][0])
        assert np.abs(host(lse)[:, rows][finite] - ref["lse"][0][finite]).max() <= 3e-3, i
    again, lse2 = call()
    assert torch.equal(again, out) and torch.equal(lse2, lse)
