"""Compensated sums taken in parts and joined (kahan_add, kahan_join of
scft_string_b200/csrc/common.cuh; the density pass of small grids), built for the host:
the total is the exact sum to one rounding, whatever the order of the parts' sizes."""
import ctypes as C
import math
import os
import shutil
import subprocess

import numpy as np
import pytest

from test_reg64_host import _cuda_include

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "scft_string_b200", "csrc")
SRC = """#include "common.cuh"
extern "C" double total(const double *v, int n, int parts)
{
    double sum = 0, c = 0;
    for (int p = 0; p < parts; p++) {
        double s = 0, d = 0;
        for (int i = n * p / parts; i < n * (p + 1) / parts; i++) scft::kahan_add(s, d, v[i]);
        if (p == 0)
            sum = s, c = d;
        else
            scft::kahan_join(sum, c, s, d);
    }
    return sum - c;
}
"""


@pytest.mark.parametrize("parts", [1, 2, 4])
@pytest.mark.parametrize("n", [3, 4, 9, 127])
def test_parts_join_exactly(tmp_path, parts, n):
    inc = _cuda_include()
    if inc is None or shutil.which("g++") is None:
        pytest.skip("needs g++ and the CUDA headers")
    (tmp_path / "k.cpp").write_text(SRC)
    out = str(tmp_path / "libk.so")
    subprocess.run(["g++", "-O2", "-w", "-std=c++17", "-shared", "-fPIC", "-I" + inc, "-I" + CSRC, "-o", out,
                    str(tmp_path / "k.cpp")], check=True)
    L = C.CDLL(out)
    L.total.restype = C.c_double
    L.total.argtypes = [np.ctypeslib.ndpointer(np.float64, flags="C_CONTIGUOUS"), C.c_int, C.c_int]
    rng = np.random.default_rng(7)
    for _ in range(5000):
        # positive terms, as products of propagators are, that grow or fall over the contour
        v = np.exp(rng.normal(size=n) + rng.uniform(-6, 6) * np.linspace(-1, 1, n))
        ref = math.fsum(v)
        # the exact sum rounded once, and an error of order n eps^2 that may tip the rounding
        assert abs(L.total(v, n, parts) - ref) <= np.spacing(ref)
