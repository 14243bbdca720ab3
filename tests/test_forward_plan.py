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
