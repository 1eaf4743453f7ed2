"""Parameter derivatives on grids whose general kernels need more than 256 threads per
CTA (csrc/stress_kernels_512.cu, _1024.cu): large slabs, long x axes, both precisions,
against the FP64 oracle and central differences in f."""
import numpy as np
import pytest

import oracle as O
import scft_string_b200 as S

pytestmark = pytest.mark.gpu


# slabs of 288, 448 and 544 threads, of which the second has no packed kernels in FP64
@pytest.mark.parametrize("m", [(2, 96, 96), (2, 120, 112), (2, 128, 128)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_derivatives(built_lib, m, precision):
    N, f, phic, alpha = 8, 0.43, 0.8, 0.1
    D = tuple(v / 12 for v in m)
    M = int(np.prod(m))
    rng = np.random.default_rng(21)
    wm, wp = rng.normal(0, 2.0, M), rng.normal(0, 0.5, M)

    def ctx(f, precision="fp64"):
        c = S.Context(m, D, N, chi=12, f=f, phidb=phic, ens=1, alpha=alpha, strn=1, dostring=0, fcont=1, precision=precision)
        c.set_fields(0, wm, wp)
        return c

    c = ctx(f, precision)
    # the tolerances of the same comparisons on small grids
    rtol, atol = (1e-10, 0) if precision == "fp64" else (2e-4, 2e-6)
    ref = O.Density(m, D, N).stress(np.concatenate([wm, wp]), N, alpha, phic, f, 1, fcont=True)
    for got in (c.stress(0)[0], c.stress_ckpt(0, 3)[0], -c.gradients(0)[0]):
        assert np.abs(got - ref).max() <= rtol * np.abs(ref).max() + atol
    h, lnQ = 1e-4, []
    for s in (1, -1):
        p = ctx(f + s * h)
        p.props(0)
        lnQ.append(p.get_conc(0)[1])
    fd = (lnQ[0] - lnQ[1]) / (2 * h)
    tol = (1e-6 if precision == "fp64" else 2e-4) * max(1.0, abs(fd))
    assert abs(c.dF_df(0)[0] - fd) <= tol and abs(-c.gradients(0)[2] - fd) <= tol
