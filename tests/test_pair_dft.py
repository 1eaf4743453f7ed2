"""The register DFTs of the pair-packed step kernels (scft_string_b200/csrc/dft.cuh),
built for the host and checked against numpy's FFT for every length they have,
both signs, in double precision.  No GPU."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from test_reg64_host import _cuda_include

HERE = os.path.dirname(os.path.abspath(__file__))
LENGTHS = [1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 12, 14, 15, 16, 20, 24]

SRC = r"""
#include <cmath>
#include <cuda_runtime.h>
using std::fma;
using std::fabs;
#include "dft.cuh"
using namespace scft;
template <int R> static void go(int sign, cplx<double> *v)
{
    if (sign < 0) Reg<double, R, -1>::run(v); else Reg<double, R, 1>::run(v);
}
extern "C" void h_third(int n, double *v)
{
    for (int i = 0; i < n; i++) v[i] = third(v[i]);
}
extern "C" void h_dft(int n, int sign, double *v)
{
    cplx<double> *c = reinterpret_cast<cplx<double> *>(v);
    switch (n) {
%s
    }
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    inc = _cuda_include()
    if inc is None or shutil.which("g++") is None:
        pytest.skip("needs g++ and the CUDA headers")
    d = tmp_path_factory.mktemp("dft")
    src = d / "dft_host.cpp"
    src.write_text(SRC % "\n".join(f"        case {n}: go<{n}>(sign, c); break;" for n in LENGTHS))
    out = str(d / "libdft_host.so")
    csrc = os.path.join(HERE, "..", "scft_string_b200", "csrc")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I" + inc, "-I" + csrc, "-o", out, str(src)],
                   check=True)
    L = C.CDLL(out)
    L.h_third.argtypes = [C.c_int, np.ctypeslib.ndpointer(np.float64, flags="C_CONTIGUOUS")]
    L.h_dft.argtypes = [C.c_int, C.c_int, np.ctypeslib.ndpointer(np.float64, flags="C_CONTIGUOUS")]
    return L


@pytest.mark.parametrize("n", LENGTHS)
@pytest.mark.parametrize("sign", [-1, 1])
def test_register_dft(lib, n, sign):
    rng = np.random.default_rng(n)
    x = rng.normal(size=n) + 1j * rng.normal(size=n)
    ref = np.fft.fft(x) if sign < 0 else np.fft.ifft(x) * n
    v = np.ascontiguousarray(x.view(np.float64))
    lib.h_dft(n, sign, v)
    # a few roundings of n terms of size 1
    assert np.abs(v.view(np.complex128) - ref).max() <= 8 * n * np.finfo(float).eps


def test_third(lib):
    """third(x) is x / 3 correctly rounded wherever the quotient and the residual are
    normal, and x / 3 for infinities and NaN."""
    rng = np.random.default_rng(3)
    x = rng.normal(size=200000) * 2.0 ** rng.integers(-900, 900, 200000)
    top = np.finfo(float).max
    x = np.concatenate([x, np.arange(-3000.0, 3000.0), [top, -top, np.inf, -np.inf, np.nan]])
    v = x.copy()
    lib.h_third(v.size, v)
    np.testing.assert_array_equal(v, x / 3.0)


def test_quotients_by_reciprocal(tmp_path):
    """div_by with div_mag(n) is b // n for every divisor and range that the
    run-time sizes use (axes up to 510, butterfly and element counts below 2^16)."""
    inc = _cuda_include()
    if inc is None or shutil.which("g++") is None:
        pytest.skip("needs g++ and the CUDA headers")
    src, out = tmp_path / "div.cpp", str(tmp_path / "libdiv.so")
    src.write_text('#include "common.cuh"\nextern "C" int bad(int nmax, int bmax) { for (int n = 1; n <= nmax; n++) {'
                   " unsigned m = scft::div_mag(n); for (int b = 0; b < bmax; b++)"
                   " if (scft::div_by(b, m) != b / n) return n; } return 0; }\n")
    csrc = os.path.join(HERE, "..", "scft_string_b200", "csrc")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I" + inc, "-I" + csrc, "-o", out, str(src)],
                   check=True)
    assert C.CDLL(out).bad(2048, 65536) == 0
