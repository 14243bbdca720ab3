"""The polynomial of ptx::tanh_poly (csrc/ptx.cuh): its error in emulated 32-bit arithmetic with the coefficients of the
source (no GPU), and capped scores on both sides of its range (GPU)."""
import re

import numpy as np
import pytest

from tests.conftest import ROOT


def test_error_of_the_polynomial():
    source = (ROOT / "flash_attention3_b200/csrc/ptx.cuh").read_text()
    body = source[source.index("uint64_t tanh_poly("):]
    body = body[:body.index("\n}\n")]
    coefficients = [float.fromhex(c) for c in re.findall(r"f2_pack\((-?0x1\.[0-9a-f]+p[+-]\d+)f,", body)]
    assert len(coefficients) == 7
    x = np.linspace(-1, 1, 2000001).astype(np.float32)
    u = x * x
    p = np.full(x.shape, coefficients[0], np.float32)
    for c in coefficients[1:]:
        p = (p.astype(np.float64) * u + c).astype(np.float32)  # (the product is exact in 64 bits)
    error = np.abs((x * p).astype(np.float64) - np.tanh(x.astype(np.float64)))
    assert error.max() <= 1.3e-7  # what the source states


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
