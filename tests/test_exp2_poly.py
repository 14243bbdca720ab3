"""The polynomial of ptx::exp2_poly (csrc/ptx.cuh), evaluated in emulated 32-bit arithmetic with the coefficients of the
source (no GPU)."""
import re

import numpy as np

from tests.conftest import ROOT


def test_error_of_the_polynomial():
    source = (ROOT / "flash_attention3_b200/csrc/ptx.cuh").read_text()
    body = source[source.index("float2 exp2_poly("):]
    body = body[:body.index("\n}\n")]
    coefficients = [float.fromhex(c) for c in re.findall(r"f2_pack\((0x1\.[0-9a-f]+p[+-]\d+)f,", body)]
    assert len(coefficients) == 6
    x = np.concatenate([np.linspace(-126, 8, 2000003), np.linspace(-0.5, 0.5, 200001)]).astype(np.float32)
    magic = np.float32(12582912.0)
    t = x + magic                      # the nearest integer, in the low bits
    n = t - magic
    f = (x - n).astype(np.float64)     # exact
    p = np.full(x.shape, coefficients[0], np.float32)
    for c in coefficients[1:]:
        p = (p.astype(np.float64) * f + c).astype(np.float32)  # (the product is exact in 64 bits)
    bits = p.view(np.uint32) + (t.view(np.uint32) << np.uint32(23))
    value = bits.view(np.float32).astype(np.float64)
    exact = np.exp2(x.astype(np.float64))
    error = np.abs(value / exact - 1.0)
    assert error.max() <= 2.2e-7  # what the source states
    assert np.abs(f).max() <= 0.5
