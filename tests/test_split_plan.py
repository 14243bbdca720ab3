"""How the backward splits key tiles (csrc/fa3_api.cpp), seen through the workspace it asks for (no GPU)."""
import ctypes

import pytest

from flash_attention3_b200 import capi


def params(b, hq, hkv, s, d, dtype, causal, sk=None, **extra):
    return capi.new_params(batch=b, seqlen_q=s, seqlen_k=s if sk is None else sk, num_heads_q=hq, num_heads_kv=hkv,
                           head_dim_qk=d, head_dim_v=d, causal=int(causal),
                           dtype=capi.DTYPE_FP16 if dtype == "fp16" else capi.DTYPE_BF16, **extra)


def partial_sum_bytes(p):
    """Workspace beyond the fp32 dQ accumulator, delta and the row statistics."""
    rows = p.batch * p.num_heads_q * p.seqlen_q
    up = lambda n: (n + 255) // 256 * 256
    need = capi.load(build_if_missing=False).shaobo_fa3_bwd_v2_workspace_bytes(ctypes.byref(p))
    return need - (up(up(rows * p.head_dim_qk * 4) + rows * 4) + rows * 12)


@pytest.mark.parametrize("shape", [(1, 40, 10, 2000, 128, False), (1, 64, 8, 2560, 64, False), (1, 200, 25, 700, 128, True)])
def test_partial_sums_are_fp32_where_every_sm_has_a_tile(shape):
    """With at least 148 key tiles the unsplit kernel would keep the whole sum in 32 bits."""
    b, hq, hkv, s, d, causal = shape
    assert -(-s // 128) * hkv * b >= 148
    chunks = partial_sum_bytes(params(b, hq, hkv, s, d, "fp16", causal)) / (2 * 128 * d * 4)
    assert chunks == int(chunks) and chunks >= 148
    assert partial_sum_bytes(params(b, hq, hkv, s, d, "bf16", causal)) == chunks * 2 * 128 * d * 4
