"""Where CTAs take over the work of CTAs that have not started (csrc/cta_order.h, host code compiled with g++)."""
import ctypes
import subprocess

import pytest

from tests.conftest import ROOT
from tests.test_split_plan import params, plan  # noqa: F401  (a fixture)

SRC = r'''
#include "cta_order.h"
using namespace fa3b200;
extern "C" int forward(int longest, int causal, long long pairs, long long heads, int batch, long long rows) {
    return fwd_takes_over(make_band(longest, longest, causal != 0, -1, -1), pairs, heads, batch, rows, 148);
}
extern "C" int clusters(int sq, int sk, int causal, int left, int right, long long heads) {
    return plan_fwd(make_band(sq, sk, causal != 0, left, right), heads, FwdGangs{148, 74, 33, 15}, false).splits;
}
extern "C" int backward(int sq, int sk, long long blocks, int group) { return bwd_takes_over(make_band(sq, sk, false, -1, -1), blocks, group, 148); }
'''


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("takeover")
    (d / "t.cpp").write_text(SRC)
    so = d / "libt.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", str(ROOT / "flash_attention3_b200/csrc"), str(d / "t.cpp"),
                    "-o", str(so)], check=True)
    lib = ctypes.CDLL(str(so))
    lib.forward.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_longlong, ctypes.c_longlong, ctypes.c_int, ctypes.c_longlong]
    lib.clusters.argtypes = [ctypes.c_int] * 5 + [ctypes.c_longlong]
    lib.backward.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_longlong, ctypes.c_int]
    return lib


def packed(lib, heads, lengths, causal):
    pairs = (max(lengths) + 255) // 256 * len(lengths) * heads
    return bool(lib.forward(max(lengths), causal, pairs, heads, len(lengths), sum(lengths)))


@pytest.mark.parametrize("pairs,expected", [(295, False), (296, True), (1 << 31, True)])
def test_forward_line(lib, pairs, expected):
    assert bool(lib.forward(1024, 0, pairs, 8, 4, 0)) == bool(lib.forward(1024, 1, pairs, 8, 4, 0)) == expected


@pytest.mark.parametrize("heads,lengths,full,causal", [
    (8, [1000] + [40] * 20, False, False),     # 192 pairs with rows in 672 blocks
    (4, [4096] + [100] * 15, False, False),    # 124 in 1024
    (1, [4096] + [30] * 40, False, False),     # 56 in 656
    (2, [8192] + [500] * 8, False, False),     # 96 in 576
    (16, [2048] + [128] * 20, False, True),    # 448 in 2688
    (32, [2048] + [128] * 20, True, True),     # 896 in 5376
    (16, [1024] + [30] * 50, True, True),      # 864 in 3264
    (16, [2048, 77, 1500, 300, 1024, 513, 129, 900, 1701], True, True),
    (40, [1024, 1024], False, True),           # every block has rows
    (36, [1024, 1024], False, False),
])
def test_forward_of_packed_sequences_counts_the_pairs_with_rows(lib, heads, lengths, full, causal):
    assert packed(lib, heads, lengths, False) == full and packed(lib, heads, lengths, True) == causal


@pytest.mark.parametrize("blocks,expected", [(148, False), (149, True)])
def test_backward_line(lib, blocks, expected):
    assert bool(lib.backward(1024, 1024, blocks, 4)) == expected


def test_no_wait_spans_a_tile_of_a_second(lib):
    """Warps that wait from the start of a tile to its end give up after 2e9 cycles, about 500000 steps: 64 query heads on one key
    head with a million queries, or as many keys."""
    most = 1 << 16
    assert 8 * 4000 * most > 2e9 >= 7 * 4000 * most  # with this much in hand
    assert lib.backward(most * 128 // 64, 1 << 20, 8192, 64) and not lib.backward(most * 128 // 64 + 1, 1 << 20, 8192, 64)
    assert not lib.backward(1 << 20, 1 << 20, 8192, 64)
    assert lib.forward(most * 128, 0, 1 << 16, 1, 1, 0) and not lib.forward(most * 128 + 1, 0, 1 << 16, 1, 1, 0)
    assert not lib.forward(most * 128 + 1, 1, 1 << 16, 1, 1, most * 128 + 1)


def test_gpu_cases_reach_the_form_they_name(lib, plan):
    """Enough tiles, no clusters (forward), no split key tiles (backward)."""
    from tests import test_gpu_forward_persistent as forward, test_gpu_persistent as backward
    for b, hq, _, sq, sk, _, _, causal, _, window in forward.CASES:
        assert lib.forward(sq, causal, (sq + 255) // 256 * b * hq, hq, b, 0), (b, hq, sq)
        assert lib.clusters(sq, sk, causal, *window, b * hq) == 1
    for causal in (False, True):
        assert [packed(lib, heads, [q for q, _ in forward.PACKED], causal) for heads in forward.PACKED_HEADS] == [False, True]
    for b, hq, hkv, sq, sk, d, dtype, causal, _, window in backward.CASES:
        assert lib.backward(sq, sk, (sk + 127) // 128 * b * hkv, hq // hkv), (b, hkv, sk)
        assert plan(params(b, hq, hkv, sq, d, dtype, causal, sk=sk, window_left=window[0], window_right=window[1]))[0] == 0
    for b, hq, hkv, s, *_ in backward.USED:
        assert lib.backward(s, s, (s + 127) // 128 * b * hkv, hq // hkv)
        assert lib.forward(s, 1, (s + 255) // 256 * b * hq, hq, b, 0) and lib.clusters(s, s, 1, -1, -1, b * hq) == 1
    heads, heads_kv = backward.USED_PACKED_HEADS
    assert packed(lib, heads, [slot for (slot, _), _ in backward.USED_PACKED], True)
    longest = max(slot for _, (slot, _) in backward.USED_PACKED)
    assert lib.backward(384, longest, (longest + 127) // 128 * len(backward.USED_PACKED) * heads_kv, heads // heads_kv)
