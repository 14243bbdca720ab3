"""How the forward hands out its query tiles (csrc/cta_order.h, host code compiled with g++)."""
import ctypes
import subprocess

import pytest

from tests.conftest import ROOT

SRC = r'''
#include "cta_order.h"
using namespace fa3b200;
extern "C" int plan(int sq, int sk, int causal, int wl, int wr, long long heads, const int* gangs, int packed) {
    const FwdPlan p = plan_fwd(make_band(sq, sk, causal != 0, wl, wr), heads, FwdGangs{gangs[0], gangs[1], gangs[2], gangs[3]}, packed != 0);
    return p.fold ? -p.splits : p.splits;
}
'''
B200 = (148, 74, 33, 15)  # clusters of 1, 2, 4 and 8 CTAs (fewer than SMs / CTAs: a cluster stays inside a GPC)


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("fwdplan")
    (d / "p.cpp").write_text(SRC)
    so = d / "libplan.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", str(ROOT / "flash_attention3_b200/csrc"),
                    str(d / "p.cpp"), "-o", str(so)], check=True)
    lib = ctypes.CDLL(str(so))
    lib.plan.argtypes = [ctypes.c_int] * 5 + [ctypes.c_longlong, ctypes.POINTER(ctypes.c_int), ctypes.c_int]

    def call(sq, sk, causal, heads, window=(-1, -1), gangs=B200, packed=False):
        """CTAs that share the keys of a pair of query tiles; -1: pairs of the last and the first tile"""
        return lib.plan(sq, sk, int(causal), window[0], window[1], heads, (ctypes.c_int * 4)(*gangs), int(packed))

    return call


@pytest.mark.parametrize("sq,sk,causal,heads", [(300, 8000, False, 1), (1024, 1024, True, 1), (2048, 2048, True, 4), (2048, 2048, False, 9)])
def test_clusters_that_the_device_does_not_run_are_not_planned(plan, sq, sk, causal, heads):
    splits = plan(sq, sk, causal, heads)
    assert splits in (2, 4, 8)
    assert abs(plan(sq, sk, causal, heads, gangs=(148, 0, 0, 0))) == 1
    for size, gangs in ((2, (148, 74, 0, 0)), (4, (148, 0, 36, 0)), (8, (148, 0, 0, 16))):
        assert plan(sq, sk, causal, heads, gangs=gangs) in (-1, 1, size)


def test_gpu_cases_reach_the_form_they_name(plan):
    """Clusters of 8, 4 and 2, folded pairs and neighbours, on devices with more or fewer clusters per GPC."""
    from tests.test_gpu_forward_split import CASES
    expected = [8, 4, 2, 8, 8, 8, 8, -1, -1, -1, -1, 1]
    for gangs in (B200, (148, 74, 36, 18)):
        assert [plan(sq, sk, causal, b * hq, window, gangs) for b, hq, _, sq, sk, _, _, causal, _, window in CASES] == expected
        assert plan(1280, 1280, False, 2, gangs=gangs) == 8  # (used lengths)
    assert plan(500, 500, True, 3) == -1  # (used lengths, folded)


def test_non_finite_problems_cover_the_forms(plan):
    from tests.test_gpu_nonfinite import PROBLEMS
    assert [plan(s, s, True, heads) for heads, s in PROBLEMS] == [8, -1, 1]


def test_only_causal_masks_fold_and_packed_sequences_do_not(plan):
    assert plan(449, 449, True, 12) == -1
    assert plan(449, 449, True, 12, packed=True) > 0 and plan(449, 449, False, 12) > 0
    assert plan(449, 449, True, 12, window=(200, -1)) > 0
    assert plan(8192, 8192, True, 64) == 1  # many waves
