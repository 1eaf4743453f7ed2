"""The packed FP64 step (csrc/pair.cuh) carries q + i 2^k q^dagger with k chosen so that
both parts are of one size: each propagator keeps the precision of a transform of its
own, whatever the mean of W- makes of the other.  Chains and single steps against the
same scheme in 80-bit arithmetic on the host, the box stress against the FP64 oracle."""
import numpy as np
import pytest

import oracle as O
import scft_string_b200 as S

pytestmark = pytest.mark.gpu

LD = np.longdouble
PI = LD("3.14159265358979323846264338327950288")
EPS = np.finfo(float).eps


def _h(m, D, N):
    k2 = LD(0)
    for i in range(3):
        n = np.fft.fftfreq(m[i], 1.0 / m[i]) if i < 2 else np.arange(m[2] // 2 + 1)
        shape = [1, 1, 1]
        shape[i] = -1
        k2 = k2 + ((2 * PI * n.astype(LD) / LD(D[i])) ** 2).reshape(shape)
    return np.exp(-k2 / (12 * LD(N)))


def _step(q, e4, h):
    """One Richardson step in 80 bits (density.h:129-220); e4 = exp(-w ds/4)."""
    conv = lambda v, g: np.fft.irfftn(np.fft.rfftn(v) * g, s=v.shape, axes=(0, 1, 2))  # noqa: E731
    e2 = e4 * e4
    return (4 * e4 * conv(e2 * conv(e4 * q, h), h) - e2 * conv(e2 * q, h * h)) / 3


def _e4(wm, wp, m, N):
    wm, wp = wm.astype(LD).reshape(m), wp.astype(LD).reshape(m)
    return np.exp(-(wm + wp) / (4 * LD(N))), np.exp(-(wp - wm) / (4 * LD(N)))


def _err(got, ref):
    d = got.astype(LD).ravel() - ref.ravel()
    return float(np.sqrt((d * d).sum() / (ref * ref).sum()))


def _fields(m, mean):
    rng = np.random.default_rng(11)
    M = int(np.prod(m))
    return mean + rng.normal(0, 2.0, M), rng.normal(0, 0.5, M)


# a slab in one CTA, run-time sizes, one unmerged slab over two CTAs, the largest slab
# that a CTA's shared memory holds
@pytest.mark.parametrize("m", [(16, 16, 16), (10, 12, 25), (4, 128, 128), (2, 144, 98)])
@pytest.mark.parametrize("mean", [0.0, 6.0, -10.0, 20.0, 40.0])
def test_propagators_keep_their_precision(built_lib, m, mean):
    N, f = 48, 0.375
    D = tuple(v / 12 for v in m)
    n1 = round(N * f)
    wm, wp = _fields(m, mean)
    ctx = S.Context(m, D, N, chi=20, f=f, phidb=0.8, ens=2, strn=1, dostring=0, alpha=0.2)
    ctx.set_fields(0, wm, wp)
    ctx.props(0)
    eA, eB = _e4(wm, wp, m, N)
    h = _h(m, D, N)
    for fld, (e1, e2, n) in enumerate(((eA, eB, n1), (eB, eA, N - n1))):
        q = np.ones(m, LD)
        for s in range(N):
            q = _step(q, e1 if s < n else e2, h)
            if s + 1 in (n1, N // 2, N - n1, N):
                # one rounding unit per step, all of one sign
                assert _err(ctx.propagator(0, fld, s + 1), q) <= N * EPS, (fld, s + 1)


@pytest.mark.parametrize("m", [(16, 16, 16), (35, 6, 45)])
@pytest.mark.parametrize("size", [1e-9, 1e7, 1e-250, 1e250, "point"])
def test_step_of_slices_of_different_size(built_lib, m, size):
    N, s = 32, 9
    D = tuple(v / 12 for v in m)
    wm, wp = _fields(m, 0.0)
    M = wm.size
    rng = np.random.default_rng(12)
    q = 1.0 + 0.3 * rng.normal(size=2 * M)
    if size == "point":
        q[:M] = 0.0
        q[M // 3] = 1e-6
    else:
        q[M:] *= size
    ctx = S.Context(m, D, N, chi=20, f=0.5, phidb=0.8, ens=2, strn=1, dostring=0)
    ctx.set_fields(0, wm, wp)
    out = ctx.do_step(0, q, s)
    eA, eB = _e4(wm, wp, m, N)
    h = _h(m, D, N)
    # six transforms, each of a rounding unit per factor two of its length, and the
    # pointwise products
    tol = 6 * np.log2(M) * EPS
    assert _err(out[:M], _step(q[:M].astype(LD).reshape(m), eA, h)) <= tol
    assert _err(out[M:], _step(q[M:].astype(LD).reshape(m), eB, h)) <= tol


@pytest.mark.parametrize("m", [(16, 16, 16), (10, 12, 25), (48, 48, 48), (4, 128, 128)])
@pytest.mark.parametrize("mean", [0.0, 10.0, 40.0])
def test_checkpointed_chain_has_the_same_bits(built_lib, m, mean):
    """A chain that starts again from a checkpoint goes on with the sizes it had and
    rounds as the chain without a break does: the same lnQ, and the same densities up
    to the order of the density sums."""
    N = 48
    wm, wp = _fields(m, mean)
    ctx = S.Context(m, tuple(v / 12 for v in m), N, chi=20, f=0.375, phidb=0.8, ens=1, strn=1, dostring=0, alpha=0.2)
    ctx.set_fields(0, wm, wp)
    ctx.props(0)
    full, lnQ, _ = ctx.get_conc(0)
    q, _, _ = ctx.props_ckpt(0, 7)
    ck = ctx.get_conc(0)[0]
    assert q == lnQ
    assert np.abs(ck - full).max() <= 4 * N * EPS * np.abs(full).max()


# every kind of slab and x pass: odd axes, one column left over in the last x tile, x
# planes beyond the blocks of the sums, merged passes, a slab over two CTAs
@pytest.mark.parametrize("m,mean", [((8, 12, 10), 0.0), ((8, 12, 10), 10.0), ((8, 12, 10), 40.0), ((3, 5, 7), 0.0),
                                    ((9, 15, 14), 0.0), ((7, 9, 25), 3.0), ((14, 15, 15), 0.0), ((96, 24, 24), 5.0),
                                    ((8, 64, 96), 0.0), ((16, 48, 48), 0.0), ((4, 128, 128), 8.0)])
@pytest.mark.parametrize("fcont", [0, 1])
def test_stress_matches_oracle(built_lib, m, mean, fcont):
    N, f = 20, 0.43 if fcont else 0.45
    D = tuple(v / 12 for v in m)
    wm, wp = _fields(m, mean)
    ctx = S.Context(m, D, N, chi=12, f=f, phidb=0.8, ens=1, alpha=0.1, strn=1, dostring=0, fcont=fcont)
    ctx.set_fields(0, wm, wp)
    ref = O.Density(m, D, N).stress(np.concatenate([wm, wp]), N, 0.1, 0.8, f, 1, fcont=bool(fcont))
    tol = 1e-10 * np.abs(ref).max()
    assert np.abs(ctx.stress(0)[0] - ref).max() <= tol
    assert np.abs(ctx.stress_ckpt(0, 6)[0] - ref).max() <= tol


@pytest.mark.parametrize("m", [(16, 16, 16), (10, 12, 25)])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_step_keeps_a_nonfinite_slice_to_itself(built_lib, m, bad):
    N, s = 32, 9
    D = tuple(v / 12 for v in m)
    wm, wp = _fields(m, 0.0)
    M = wm.size
    ctx = S.Context(m, D, N, chi=20, f=0.5, phidb=0.8, ens=2, strn=1, dostring=0)
    ctx.set_fields(0, wm, wp)
    eA, eB = _e4(wm, wp, m, N)
    h = _h(m, D, N)
    q = 1.0 + 0.3 * np.random.default_rng(13).normal(size=2 * M)
    for fld, e4 in ((0, eB), (1, eA)):
        p = q.copy()
        p[fld * M + M // 2] = bad
        out = ctx.do_step(0, p, s).reshape(2, M)
        assert not np.isfinite(out[fld]).any()
        o = 1 - fld
        assert _err(out[o], _step(p[o * M:(o + 1) * M].astype(LD).reshape(m), e4, h)) <= 6 * np.log2(M) * EPS


@pytest.mark.parametrize("nostore", [0, 1])
def test_densities_where_one_propagator_overflows(built_lib, nostore):
    """Replica 1 of three has an A field in which q grows beyond a double at once; its
    homopolymer, which sees the B field alone, and the other replicas do not notice."""
    m, N, alpha = (16, 12, 10), 20, 0.2
    D = tuple(v / 12 for v in m)
    M = int(np.prod(m))
    W = [_fields(m, 0.0) for _ in range(3)]
    big = 5e3
    W[1] = (W[1][0] - big, W[1][1] - big)  # wA = W- + W+, wB = W+ - W-
    ctx = S.Context(m, D, N, chi=12, f=0.4, phidb=0.8, ens=1, strn=3, dostring=0, alpha=alpha, nostore=nostore, ckpt_K=6)
    for ii in range(3):
        ctx.set_fields(ii, *W[ii])
    with pytest.raises(S.ScftError, match="replica 1"):
        ctx.solve_field0_all(2, 0.0)  # one round, which then finds the residual of replica 1 to be NaN
    for ii in (0, 2):
        conc, lnQ, phis = ctx.get_conc(ii)
        w = np.concatenate([*W[ii], np.zeros(4 * M)])
        ref_lnQ, ref = O.Density(m, D, N).props(w, N, alpha, 0.8, 0.4, 1)
        assert np.abs(conc - w[2 * M:]).max() <= 1e-12 * np.abs(w[2 * M:]).max()
        assert abs(lnQ - ref_lnQ) <= 1e-12 * abs(ref_lnQ) and abs(phis[4] - ref[4]) <= 1e-12 * abs(ref[4])
    # q^dagger of replica 1 in the B block, and the homopolymer's Simpson sum (density.h:404-422)
    eB, h, Nh = _e4(*W[1], m, N)[1], _h(m, D, N), int(alpha * N)
    q = [np.ones(m, LD)]
    for s in range(Nh):
        q.append(_step(q[-1], eB, h))
    rh = 2 * q[Nh] + sum((2 if (s - 1) % 2 else 4) * q[s] * q[Nh - s] for s in range(1, Nh))
    rh = rh * (1 - 0.8) / (q[Nh].mean() * alpha) / (3 * LD(N))
    conc, lnQ, phis = ctx.get_conc(1)
    assert not np.isfinite(lnQ) and not np.isfinite(conc[:2 * M]).any()
    assert _err(conc[2 * M:3 * M], rh) <= N * EPS
    assert abs(phis[4] - float(rh.mean())) <= N * EPS * abs(phis[4])
    if not nostore:
        assert _err(ctx.propagator(1, 1, Nh), q[Nh]) <= N * EPS
