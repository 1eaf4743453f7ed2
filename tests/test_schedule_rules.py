"""The host rules that pick the schedule of a props round (csrc/schedule.h).  No GPU."""
import ctypes as C
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "scft_string_b200", "csrc")
SRC = """#include "schedule.h"
extern "C" int default_groups(int pair, long long M, int nb) { return scft::default_groups(pair, M, nb); }
extern "C" int effective_groups(int ng, int nb) { return scft::effective_groups(ng, nb); }
extern "C" int wide_tiles(int w, int m0, int ncol, int n, int nslots) { return scft::wide_tiles(w, m0, ncol, 32, n, nslots); }
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("needs g++")
    d = tmp_path_factory.mktemp("rules")
    (d / "r.cpp").write_text(SRC)
    out = str(d / "librules.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I" + CSRC, "-o", out, str(d / "r.cpp")], check=True)
    L = C.CDLL(out)
    L.default_groups.argtypes = [C.c_int, C.c_longlong, C.c_int]
    return L


@pytest.mark.parametrize("pair", [0, 1])
def test_default_groups_are_of_some_size(rules, pair):
    for m in (2, 8, 16, 24, 32, 40, 48, 64, 80, 96, 112, 128, 200):
        for nb in range(1, 65):
            ng = rules.default_groups(pair, m ** 3, nb)
            assert ng in ((1, 2, 4, 8) if pair else (1, 2))
            assert nb >= {1: 1, 2: 4, 4: 12, 8: 24}[ng], (m, nb, ng)
            if ng == 1:
                assert nb < 4


def test_default_groups_where_measured(rules):
    """The fastest count, or one within half a per cent of it."""
    fastest = {(48, 8): 2, (48, 16): 2, (48, 24): 4, (48, 32): 4, (64, 8): 2, (64, 10): 2, (64, 11): 2, (64, 12): 4,
               (64, 14): 4, (64, 16): 4, (64, 20): 4, (64, 24): 8, (80, 8): 2, (80, 12): 2, (80, 16): 2, (96, 8): 2,
               (96, 12): 2, (96, 16): 2, (128, 4): 2}
    for (m, nb), ng in fastest.items():
        assert rules.default_groups(1, m ** 3, nb) == ng, (m, nb)


def test_tile_width_asked_for_is_taken(rules):
    for m in (32, 48, 64, 96, 128):
        for spectra in (2, 4):
            for nslots in (1, 4, 16, 48):
                ncol = m * (m // 2 + 1)
                assert rules.wide_tiles(0, m, ncol, spectra, nslots) == 0
                assert rules.wide_tiles(1, m, ncol, spectra, nslots) == 1
    assert rules.wide_tiles(-1, 64, 64 * 33, 4, 16) == 1 and rules.wide_tiles(-1, 64, 64 * 33, 4, 1) == 0
    assert rules.wide_tiles(-1, 128, 128 * 65, 4, 8) == 0
