"""GPU parity of the forward where a cluster of CTAs shares the key tiles of a pair of query tiles: every
cluster size, key tiles that do not divide evenly, a ragged last pair, masks that leave a CTA without keys."""
import numpy as np
import pytest
import torch

from flash_attention3_b200 import ops
from oracle import golden
from tests.helpers import Problem, dev, host
from tests.test_gpu_forward import check_forward

pytestmark = pytest.mark.gpu

# (b, hq, hkv, sq, sk, d, dtype, causal, layout, window)
CASES = [
    (1, 1, 1, 1024, 1024, 128, "bf16", True, "bhsd", (-1, -1)),    # clusters of 8, early pairs with fewer keys than CTAs
    (1, 4, 2, 2048, 2048, 64, "fp16", True, "bshd", (-1, -1)),     # clusters of 4
    (1, 9, 9, 2048, 2048, 128, "bf16", False, "bhsd", (-1, -1)),   # clusters of 2
    (1, 2, 1, 130, 2000, 64, "bf16", False, "bshd", (-1, -1)),     # 16 key tiles, ragged; a pair with two rows in tile B
    (1, 1, 1, 129, 1153, 128, "fp16", True, "bhsd", (-1, -1)),     # 10 key tiles over 8 CTAs: the last ones get none
    (1, 2, 2, 1500, 1500, 128, "bf16", True, "bhsd", (700, -1)),   # a window: pairs see a part of the keys
    (1, 2, 2, 1700, 1100, 64, "fp16", True, "bhsd", (-1, -1)),     # leading queries without a key
    # CTAs that take the last and the first query tile, the last but one and the second, ... (no split)
    (1, 2, 1, 449, 449, 128, "bf16", True, "bhsd", (-1, -1)),      # four tiles, the last one ragged
    (2, 1, 1, 833, 333, 64, "fp16", True, "bshd", (-1, -1)),       # seven tiles: the middle one is alone; tiles without a key
    (1, 12, 4, 449, 449, 64, "bf16", True, "bhsd", (-1, -1)),      # with groups of query heads
    (1, 20, 5, 897, 897, 64, "bf16", True, "bshd", (-1, -1)),
    # neighbours, whole
    (1, 12, 4, 769, 769, 64, "bf16", True, "bshd", (-1, -1)),
]


@pytest.mark.parametrize("b,hq,hkv,sq,sk,d,dtype,causal,layout,window", CASES)
def test_split_keys(b, hq, hkv, sq, sk, d, dtype, causal, layout, window):
    prob = Problem(b, hq, hkv, sq, d, dtype, causal, seed=700 + sq + sk, sk=sk, layout=layout, window=window)
    x = prob.device_inputs()
    out, lse = ops.fa3_fwd(x["q"], x["k"], x["v"], causal, prob.scale, layout=layout, window=window, sync=True)
    check_forward(prob.from_layout(host(out)), host(lse), prob.ref["out"], prob.ref["lse"], dtype, (sq, sk, d, causal, window))


def test_used_lengths_with_split_keys():
    """Rows behind the used length are zero and do not disturb the merge."""
    b, h, s, d, dtype = 1, 2, 1280, 64, "bf16"
    used_q, used_k = 1000, 1111
    q, k, v, do = golden.seeded_inputs(41, b, h, h, s, d, dtype)
    ref = golden.backward(q[:, :, :used_q], k[:, :, :used_k], v[:, :, :used_k], do[:, :, :used_q], False, 1.0 / np.sqrt(d), dtype)
    used = [torch.tensor([n], dtype=torch.int32, device="cuda") for n in (used_q, used_k)]
    out, lse = ops.fa3_fwd(dev(q, dtype), dev(k, dtype), dev(v, dtype), False, seqused_q=used[0], seqused_k=used[1], sync=True)
    out, lse = host(out), host(lse)
    check_forward(out[:, :, :used_q], lse[:, :, :used_q], ref["out"], ref["lse"], dtype, "used lengths")
    assert (out[:, :, used_q:] == 0).all() and np.isneginf(lse[:, :, used_q:]).all()


@pytest.mark.parametrize("used_q,used_k", [(500, 500), (130, 500), (500, 260), (60, 1)])
def test_used_lengths_with_folded_pairs(used_q, used_k):
    b, h, s, d, dtype = 1, 3, 500, 128, "fp16"
    q, k, v, do = golden.seeded_inputs(43, b, h, h, s, d, dtype)
    ref = golden.backward(q[:, :, :used_q], k[:, :, :used_k], v[:, :, :used_k], do[:, :, :used_q], True, 1.0 / np.sqrt(d), dtype)
    used = [torch.tensor([n], dtype=torch.int32, device="cuda") for n in (used_q, used_k)]
    out, lse = ops.fa3_fwd(dev(q, dtype), dev(k, dtype), dev(v, dtype), True, seqused_q=used[0], seqused_k=used[1], sync=True)
    out, lse = host(out), host(lse)
    check_forward(out[:, :, :used_q], lse[:, :, :used_q], ref["out"], ref["lse"], dtype, "used lengths")
    assert (out[:, :, used_q:] == 0).all() and np.isneginf(lse[:, :, used_q:]).all()


@pytest.mark.parametrize("d", [64, 128])
def test_exponentials_far_below_the_maximum(d):
    """One key dominates every row: the other scores are hundreds of log2 units below it."""
    s = 384
    rng = np.random.default_rng(3)
    q = golden.round_to("fp16", np.abs(rng.standard_normal((1, 2, s, d), dtype=np.float32)) + 1.0)
    k = golden.round_to("fp16", -np.abs(rng.standard_normal((1, 2, s, d), dtype=np.float32)) * 8.0)
    k[:, :, 200] = 8.0
    v = golden.round_to("fp16", rng.standard_normal((1, 2, s, d), dtype=np.float32))
    ref = golden.backward(q, k, v, v * 0, False, 1.0, "fp16")
    out, lse = ops.fa3_fwd(dev(q, "fp16"), dev(k, "fp16"), dev(v, "fp16"), False, 1.0, sync=True)
    # the log-sum-exp is the dominant score, a sum of D exact products of one sign in 32 bits: at most D truncations to 24
    # bits, and three roundings in its conversion to and from log2 units
    score = np.matmul(q.astype(np.float64), k.astype(np.float64).transpose(0, 1, 3, 2))
    top = score.max(axis=-1)
    exact = top + np.log(np.exp(score - top[..., None]).sum(axis=-1))
    assert exact.min() > 512.0 and (np.abs(host(lse) - exact) <= exact * (d + 3) * 2.0 ** -23).all()
    check_forward(host(out), np.zeros(1), ref["out"], np.zeros(1), "fp16", "far below")
