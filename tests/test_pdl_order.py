"""What a step kernel reads before it waits for the kernel ahead of it on the stream.

The launches of a contour step overlap: a kernel may start while the one before it
runs, and sees that one's writes only after its wait.  Before the wait it may read
what was there when the chain began: twiddle factors, diffusion factors, the replica
list; and, from the second kernel on, the E tables.  The first combine of a chain
(modes 1 and 2) follows the kernel that writes the E tables.  One thread of each
kernel runs on the host and its reads are noted.  No GPU."""
import ctypes as C
import os
import shutil
import subprocess

import pytest

from test_reg64_host import _cuda_include

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "scft_string_b200", "csrc")
ARRAYS = ["W", "HIST", "ETAB", "JTAB", "SPEC", "PBUF", "SIZES", "CONST"]

PDL = """#pragma once
#include <cstring>
namespace scft {
inline void pdl_trigger() {}
inline void pdl_wait() { waited = true; }
inline bool pdl_early(int) { return false; }
inline void prefetch_l2(const void *, int) {}
inline void pair_arrive() {}
inline void pair_wait() {}
}
"""
TMA = """#pragma once
namespace scft {
inline void mbar_init(uint64_t *, int) {}
inline void mbar_fence_init() {}
inline void mbar_expect_tx(uint64_t *, uint32_t) {}
inline void mbar_wait(uint64_t *, uint32_t, int *) {}
inline void fence_proxy_async_smem() {}
inline void tma_store_wait_read() {}
inline void bulk_commit() {}
inline void bulk_g2s(void *d, const void *s, uint32_t n, uint64_t *)
{
    note((const char *)s);
    std::memcpy(d, s, n);
}
inline void bulk_s2g(void *d, const void *s, uint32_t n) { std::memcpy(d, s, n); }
}
"""


@pytest.fixture(scope="module")
def early(tmp_path_factory):
    inc = _cuda_include()
    if inc is None or shutil.which("g++") is None:
        pytest.skip("needs g++ and the CUDA headers")
    d = tmp_path_factory.mktemp("pdl")
    for f in ("real_slab.cuh", "pair.cuh", "common.cuh", "fft.cuh", "dft.cuh", "kernels.h"):
        shutil.copy(os.path.join(CSRC, f), d / f)
    (d / "pdl.cuh").write_text(PDL)
    (d / "tma.cuh").write_text(TMA)
    shutil.copy(os.path.join(HERE, "pdl_order_host.cpp"), d / "pdl_order_host.cpp")
    out = str(d / "libpdl.so")
    subprocess.run(["g++", "-O1", "-w", "-std=c++17", "-shared", "-fPIC", "-I" + inc, "-o", out,
                    str(d / "pdl_order_host.cpp")], check=True)
    L = C.CDLL(out)

    def run(fp32, which, s, mode):
        n = (C.c_int * 16)()
        assert L.h_early(fp32, which, s, mode, n) == 0, "no wait"
        return {a for a, k in zip(ARRAYS, n) if k}

    return run


@pytest.mark.parametrize("fp32", [0, 1])
@pytest.mark.parametrize("s,mode", [(-1, 1), (-1, 2), (3, 2)])
def test_first_combine_of_a_chain(early, fp32, s, mode):
    assert early(fp32, 0, s, mode) <= {"CONST"}


@pytest.mark.parametrize("fp32", [0, 1])
@pytest.mark.parametrize("which,s", [(0, 0), (0, 3), (0, 7), (1, 0), (1, 5), (2, 0)])
def test_later_kernels(early, fp32, which, s):
    assert early(fp32, which, s, 0) <= {"CONST", "ETAB", "JTAB"}
