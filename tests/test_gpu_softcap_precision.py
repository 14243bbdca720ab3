"""Capped gradients whose scores lie far above the cap, against 64-bit results.  The slope of the cap is nearly zero for most
(query, key) pairs there, and P times the slope lies below the normal range of fp16 in long rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def exact_gradients(q, k, v, dout, softcap, scale):
    """[S, D] tensors of one head, causal: O, log-sum-exp, dQ, dK, dV in 64 bits."""
    q, k, v, dout = (x.double() for x in (q, k, v, dout))
    t = torch.tanh(q @ k.T * (scale / softcap))
    s = (softcap * t).masked_fill(torch.ones_like(t, dtype=torch.bool).triu(1), float("-inf"))
    lse = torch.logsumexp(s, -1)
    p = torch.exp(s - lse[:, None])
    out = p @ v
    ds = p * (dout @ v.T - (dout * out).sum(-1, keepdim=True)) * (1 - t * t)
    return out, lse, ds @ k * scale, ds.T @ q * scale, p.T @ dout


@pytest.mark.parametrize("deterministic", [False, True])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("s,d,softcap,spread", [(8192, 128, 15.0, 40.0), (8192, 64, 5.0, 40.0), (2048, 64, 5.0, 5.0)])
def test_slope_of_scores_above_the_cap(s, d, softcap, spread, dtype, deterministic):
    """dS and the result are rounded to 16 bits, at most 2^-11 (fp16) or 2^-8 / 2 (bf16) of the value each and 0.42 of that in the
    root mean square; O, and by it delta, has the same share.  Together they stay below one such step."""
    from flash_attention3_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(7)
    q, k, v, dout = (torch.randn((1, 1, s, d), device="cuda", generator=gen) for _ in range(4))
    q, k, v, dout = (x.to(dtype) for x in (q * spread, k, v, dout))
    out, lse, *expected = exact_gradients(*(x[0, 0] for x in (q, k, v, dout)), softcap, d ** -0.5)
    got = ops.fa3_bwd(dout, q, k, v, out[None, None].to(dtype), lse[None, None].float(), True, softcap=softcap,
                      deterministic=deterministic, sync=True)
    for name, g, e in zip(("dq", "dk", "dv"), got, expected):
        error = ((g[0, 0].double() - e).norm() / e.norm()).item()
        assert error <= torch.finfo(dtype).eps / 2, (name, error)
