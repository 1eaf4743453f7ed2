"""The FP32 slab and x kernels with in-place register passes (csrc/real_slab.cuh)
keep every rounding of the staged transforms, which the persistent step kernel
still runs: a props round gives the same densities, lnQ and propagators bit for
bit on every compile-time shape, with and without a junction step, with wide and
default x tiles, and the step entry matches the oracle at the FP32 tolerance."""
import numpy as np
import pytest

import oracle as O
import scft_string_b200 as S

pytestmark = pytest.mark.gpu

SHAPES = [(32, 32, 32), (48, 48, 48), (64, 64, 64), (64, 64, 96), (96, 96, 96), (128, 128, 128)]


@pytest.mark.parametrize("m", SHAPES)
@pytest.mark.parametrize("fcont", [0, 1])
def test_same_bits_as_staged_transforms(built_lib, monkeypatch, m, fcont):
    M, N = int(np.prod(m)), 10
    rng = np.random.default_rng(5)
    wm, wp = rng.normal(0, 3.0, (2, M)), rng.normal(0, 1.0, (2, M))

    def run(persist, wide):
        monkeypatch.setenv("SCFT_PERSIST", persist)
        monkeypatch.setenv("SCFT_PENCIL_TILE_WIDE", wide)
        ctx = S.Context(m, (4.0, 4.1, 4.2), N, chi=14, f=0.43, phidb=0.85, ens=2, strn=2, dostring=0, precision="fp32",
                        fcont=fcont)
        for ii in range(2):
            ctx.set_fields(ii, wm[ii], wp[ii])
        ctx.solve_field0_all(2, 0.0)
        conc, lnQ, _ = ctx.get_conc(1)
        return conc, lnQ, ctx.propagator(1, 0, N), ctx.propagator(1, 1, N)

    ref = run("1", "0")
    for wide in ("0", "1"):
        got = run("0", wide)
        for a, b in zip(ref, got):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("m", [(48, 48, 48), (64, 64, 96)])
def test_step_at_the_block_change(built_lib, m):
    """Steps before, at and after q's and q^dagger's change of blocks (the next
    step's table is then not the staged one)."""
    M, Ns = int(np.prod(m)), 12
    rng = np.random.default_rng(6)
    wm, wp = rng.normal(0, 1.0, M), rng.normal(0, 0.5, M)
    D = (3.0, 3.1, 4.2)
    ctx = S.Context(m, D, Ns, chi=10, f=1 / 3, phidb=0.8, ens=2, strn=1, dostring=0, precision="fp32")
    ctx.set_fields(0, wm, wp)
    od = O.Density(m, D, Ns)
    od.prepare(1.0 / Ns, np.concatenate([wm, wp]))
    q = 1.0 + 0.3 * rng.normal(size=2 * M)
    for s in (0, 3, 4, 7, 8, Ns - 1):
        ref = od.do_step(q, s, 4, 8)
        # the tolerance of the other FP32 step tests
        assert np.abs(ctx.do_step(0, q, s) - ref).max() <= 2e-6 * np.abs(ref).max(), s


@pytest.mark.parametrize("m,many", [((16, 12, 20), 24), ((35, 14, 45), 11), ((30, 28, 27), 13), ((9, 50, 21), 44)])
def test_run_time_sizes_same_bits_alone_and_in_a_batch(built_lib, m, many):
    """At sizes without compile-time kernels a small batch shares each slab between
    two CTAs; a replica gets the same bits there as in a batch that does not."""
    M, N = int(np.prod(m)), 11
    rng = np.random.default_rng(8)
    wm, wp = rng.normal(0, 3.0, M), rng.normal(0, 1.0, M)

    def run(n):
        ctx = S.Context(m, (4.0, 4.1, 4.2), N, chi=14, f=0.43, phidb=0.85, ens=2, strn=n, dostring=0, precision="fp32")
        for ii in range(n):
            ctx.set_fields(ii, wm, wp)
        ctx.solve_field0_all(2, 0.0)
        conc, lnQ, _ = ctx.get_conc(n - 1)
        return conc, lnQ, ctx.propagator(n - 1, 0, N), ctx.propagator(n - 1, 1, N)

    for a, b in zip(run(1), run(many)):
        np.testing.assert_array_equal(a, b)
