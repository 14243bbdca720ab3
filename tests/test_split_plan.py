"""How the backward splits key tiles (csrc/fa3_api.cpp, host code compiled with g++), and the workspace it asks for."""
import ctypes
import subprocess

import pytest

from flash_attention3_b200 import capi
from tests.conftest import ROOT

SRC = r'''
#include "fa3_host.h"
using namespace fa3b200;
extern "C" void plan(const ShaoboFa3Params* p, int* out) {
    const SplitPlan s = split_plan(p);
    out[0] = s.chunk_steps; out[1] = s.chunks_per_head; out[2] = s.slab_elem_bytes;
    for (int kt = 0; kt < tiles_of(p->seqlen_k) && kt < 148; ++kt) {
        const int steps = p->num_heads_q / p->num_heads_kv * q_tiles_of_k_tile(kt, band_of(p));
        out[3 + kt] = s.chunk_steps > 0 ? (steps + s.chunk_steps - 1) / s.chunk_steps : 0;
    }
}
'''


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("split")
    (d / "s.cpp").write_text(SRC)
    so = d / "libsplit.so"
    csrc = ROOT / "flash_attention3_b200/csrc"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I", str(csrc), "-I", str(ROOT / "include"),
                    str(d / "s.cpp"), str(csrc / "fa3_api.cpp"), "-o", str(so)], check=True)
    lib = ctypes.CDLL(str(so))

    def call(p):
        """(chunks per (batch, KV head), bytes per element of the partial sums, chunks of every key tile)"""
        out = (ctypes.c_int * 151)()
        lib.plan(ctypes.byref(p), out)
        return out[1], out[2], list(out[3:3 + -(-p.seqlen_k // 128)])

    return call


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


def test_partial_sums_of_fp16_problems_with_few_tiles_are_fp16(plan):
    assert plan(params(1, 4, 4, 2048, 128, "fp16", True))[1] == 2 and plan(params(1, 4, 4, 2048, 128, "bf16", True))[1] == 4


def test_gpu_cases_reach_the_form_they_name(plan):
    from tests.test_gpu_shapes import MANY_CHUNKS, MANY_TILES_SPLIT
    # launch_convert: eight lanes share a vector's partial sums where a tile has many of them on average
    shared = []
    for b, hq, hkv, sq, sk, d, dtype, causal, _ in MANY_CHUNKS:
        chunks, elem, per_tile = plan(params(b, hq, hkv, sq, d, dtype, causal, sk=sk))
        assert sum(per_tile) == chunks and elem == (2 if dtype == "fp16" else 4)
        if chunks >= 16 * len(per_tile) if elem == 2 else chunks > 8 * len(per_tile):
            shared.append((per_tile, b * hq * sq * d // 8 % 32, elem))
    assert len(shared) == 5
    assert {elem for *_, elem in shared} == {2, 4}
    assert any(min(n) != max(n) for n, _, _ in shared) and any(any(c % 8 for c in n) for n, _, _ in shared)
    assert any(rest != 0 for _, rest, _ in shared)  # dQ vectors that are no multiple of a warp
    split = [plan(params(b, hq, hkv, s, d, dtype, causal))[0] * b * hkv for b, hq, hkv, s, d, dtype, causal in MANY_TILES_SPLIT]
    assert split == [300, 0, 200]
