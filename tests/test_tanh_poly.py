"""tanh of capped scores on the FMA pipe (ptx::tanh_pair_fma, csrc/ptx.cuh): its error in emulated 32-bit arithmetic with the
coefficients of the source (no GPU), and capped scores of all magnitudes (GPU)."""
import re

import numpy as np
import pytest

from tests.conftest import ROOT


def test_error_of_the_polynomial():
    source = (ROOT / "flash_attention3_b200/csrc/ptx.cuh").read_text()
    body = source[source.index("uint64_t tanh_pair_fma("):]
    body = body[:body.index("\n}\n")]
    coefficients = [float.fromhex(c) for c in re.findall(r"f2_pack\((-?0x1\.[0-9a-f]+p[+-]\d+)f,", body)]
    assert len(coefficients) == 4
    fma = lambda a, b, c: (np.asarray(a, np.float64) * b + c).astype(np.float32)  # (the product is exact in 64 bits)
    x = np.concatenate([np.linspace(0, 12, 2000001), np.logspace(-8, 0, 100001)])
    worst = 0.0
    for error_of_z in (-2.0 ** -22, 0.0, 2.0 ** -22):  # ex2.approx: two units in the last place
        z = (np.exp(-2 * x) * (1 + error_of_z)).astype(np.float32)
        r = np.full(z.shape, coefficients[0], np.float32)
        for c in coefficients[1:]:
            r = fma(r, z, c)
        e = fma(fma(z, -1, -1), r, 1)
        r = fma(r, fma(e, e, e), r)
        error = np.abs(fma(fma(z, -1, 1), r, 0).astype(np.float64) - np.tanh(x))
        worst = max(worst, error.max())
    assert worst <= 1.9e-7  # what the source states


def _capped_lse(score, softcap, d, keys=128):
    from flash_attention3_b200 import ops
    from tests.helpers import dev, host
    q, k = np.zeros((1, 1, len(score), d), np.float32), np.zeros((1, 1, keys, d), np.float32)
    q[0, 0, :, 0], k[..., 0] = score, 1.0
    out, lse = ops.fa3_fwd(dev(q, "fp16"), dev(k, "fp16"), dev(k, "fp16"), False, 1.0, softcap=softcap, sync=True)
    return host(out)[0, 0], host(lse)[0, 0]


@pytest.mark.gpu
@pytest.mark.parametrize("spread", [0.05, 0.999, 1.001, 8.0])
@pytest.mark.parametrize("d", [64, 128])
def test_capped_scores_on_both_sides_of_the_range(d, spread):
    """Equal keys: the log-sum-exp is the capped score plus log(number of keys), 1.31 caps at most.  tanh is good to 2.3e-7;
    the cap in log2 units, the product with it, the sum and the product with ln 2 (and ln 2 itself) round once each."""
    softcap = 16.0
    score = np.random.default_rng(3).uniform(-spread * softcap, spread * softcap, 1024).astype(np.float16)
    _, lse = _capped_lse(score, softcap, d)
    expected = softcap * np.tanh(score.astype(np.float64) / softcap) + np.log(128)
    assert np.abs(lse - expected).max() / softcap <= 2.3e-7 + 5 * 1.31 * 2.0 ** -24


@pytest.mark.gpu
@pytest.mark.parametrize("d", [64, 128])
def test_a_small_score_does_not_depend_on_its_neighbours(d):
    score = np.random.default_rng(4).uniform(-8, 8, 256).astype(np.float16)
    out, lse = _capped_lse(score, 16.0, d)
    large = score.copy()
    large[::7] = 100.0
    out2, lse2 = _capped_lse(large, 16.0, d)
    rest = np.arange(256) % 7 != 0
    assert np.array_equal(lse[rest], lse2[rest]) and np.array_equal(out[rest], out2[rest])


@pytest.mark.gpu
@pytest.mark.parametrize("d", [64, 128])
def test_time_of_the_gradients_does_not_depend_on_the_scores(d):
    """Scores far below the cap, and one in a thousand above it.  Two runs differ by under a tenth; a form chosen by the scores of a
    tile made the second 1.24 to 1.5 times as long."""
    import torch
    from flash_attention3_b200 import ops
    times = []
    for spread in (1.0, 0.304 * 30.0):
        gen = torch.Generator(device="cuda").manual_seed(3)
        q, k, v, dout = (torch.randn((4, 16, 1024, d), device="cuda", generator=gen) for _ in range(4))
        q, k, v, dout = (x.bfloat16() for x in (q * spread, k, v, dout))
        out, lse = ops.fa3_fwd(q, k, v, True, softcap=30.0)
        call = lambda: ops.fa3_bwd(dout, q, k, v, out, lse, True, softcap=30.0)
        events = [torch.cuda.Event(enable_timing=True) for _ in range(12)]
        for _ in range(20):
            call()
        for e in events:
            for _ in range(10):
                call()
            e.record()
        torch.cuda.synchronize()
        times.append(sorted(a.elapsed_time(b) for a, b in zip(events, events[1:]))[5])
    assert times[1] <= 1.15 * times[0], times
