"""The FP64 contour step on q + i q^dagger (csrc/pair.cuh) against the FP64
oracle, on every slab shape it has (merged and unmerged passes, run-time sizes)
and with an x axis of its own, and on shapes it leaves to the general kernels, as one replica (the combine of two CTAs per slab where the
batch is small) and in a batch of several (one CTA per slab)."""
import numpy as np
import pytest

import oracle as O
import scft_string_b200 as S

pytestmark = pytest.mark.gpu

GRIDS = [(16, 16, 16), (24, 24, 24), (40, 40, 40), (80, 80, 80), (16, 64, 64), (96, 24, 24), (80, 64, 96),
         (128, 16, 16), (24, 96, 96), (48, 48, 48), (8, 128, 128),
         # run-time sizes: every radix, prime axes, the smallest ones, one column left over
         (35, 54, 45), (2, 2, 2), (3, 5, 7), (9, 100, 98), (6, 15, 16), (112, 14, 12), (10, 3, 3),
         (30, 108, 112), (64, 25, 27), (1, 12, 10), (12, 1, 10), (12, 10, 1), (4, 125, 6)]


@pytest.mark.parametrize("m", GRIDS)
def test_step_and_densities(built_lib, m):
    M = int(np.prod(m))
    D = tuple(v / 12 for v in m)
    Ns, f = 10, 0.4
    rng = np.random.default_rng(11)
    wm, wp = rng.normal(0, 1.0, (9, M)), rng.normal(0, 0.5, (9, M))
    ctx = S.Context(m, D, Ns, chi=10, f=f, phidb=0.8, ens=2, strn=9, dostring=0, alpha=0.2)
    for ii in range(9):
        ctx.set_fields(ii, wm[ii], wp[ii])
    od = O.Density(m, D, Ns)
    od.prepare(1.0 / Ns, np.concatenate([wm[8], wp[8]]))
    qin = 1.0 + 0.3 * rng.normal(size=2 * M)
    for s in (0, 3, 4, 6, Ns - 1):  # A and B blocks of q and of q^dagger
        ref = od.do_step(qin, s, 4, 6)
        # the tolerance of the other FP64 step tests
        assert np.abs(ctx.do_step(8, qin, s) - ref).max() <= 1e-13 * np.abs(ref).max(), s
    ctx.props(8)  # alone
    one = ctx.get_conc(8)
    ctx.solve_field0_all(2, 0.0)  # one batched round at the same fields
    batch = ctx.get_conc(8)
    w = np.zeros(6 * M)
    w[:M], w[M:2 * M] = wm[8], wp[8]
    lnQ, phis = od.props(w, Ns, 0.2, 0.8, f, 2)
    for conc, q, ph in (one, batch):
        assert abs(q - lnQ) <= 1e-12 * abs(lnQ)
        assert np.abs(conc - w[2 * M:]).max() <= 1e-12 * np.abs(w[2 * M:]).max()
    np.testing.assert_array_equal(one[0], batch[0])
