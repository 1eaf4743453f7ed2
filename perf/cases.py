"""The work that users of this field solver have it do, as timed cases.

Every case goes through the public Python entry points of scft_string_b200
(the C ABI underneath).  A case's ``kind`` is the call a program makes:

* ``step``       one Richardson contour step of a host slice (``do_step``);
* ``density``    ``Density.props`` with the reference's host-array signature,
                 the call the reference's own main loop makes;
* ``relax``      the W+ relaxation of all replicas (``solve_field0_all``);
* ``string``     one iteration of the solver loop (``string_step``): the W+
                 relaxation, the densities, and for a string its arc length,
                 projection, mixing and redistribution; a single replica
                 (strn = 1) runs the same loop without the string coupling;
* ``anderson``   a few iterations of the Anderson solver;
* ``gradients``  dF/dL, dF/dchiN and dF/df by the adjoint (the backward
                 direction);
* ``ckpt``       the densities from propagators kept at checkpoints.

Grids, chain lengths and field patterns are those of ``configs`` and of the
tests.  An FP32 context computes to single precision, so a program that asks
for one keeps what it returns in single precision; so does ``run``.
"""
import math

import numpy as np
import torch
import torch.utils.checkpoint

import scft_string_b200 as S
from scft_string_b200.configs import ADJOINT_96, MIXED_128, PLAIN_32, STRING_64

LAM0 = 0.05  # mixing parameter of both reference loops at their start


def _problem(c, **over):
    """A configuration dictionary as plain values (m0, m1, m2 and D0, D1, D2)."""
    out = dict(chi=c["chi"], f=c["f"], ens=c["ens"], phidb=c["phidb"], N=c["N"], alpha=c["alpha"], strn=c["strn"],
               fix=int(c["fix"][0]), dostring=c["dostring"], precision="fp64", fcont=0)
    for i in range(3):
        out["m%d" % i], out["D%d" % i] = int(c["m"][i]), float(c["D"][i])
    out.update(over)
    return out


def _grid(m, spacing=16.0):
    m = (m, m, m) if isinstance(m, int) else m
    return {**{"m%d" % i: int(m[i]) for i in range(3)}, **{"D%d" % i: m[i] / spacing for i in range(3)}}


def listed():
    single = dict(strn=1, fix=0, dostring=0)
    return [
        # the smallest call there is: one contour step on a small grid with three
        # different axes, a host slice in and out
        _problem(PLAIN_32, name="step_16x12x20", kind="step", pattern="noise", N=24, **_grid((16, 12, 20))),
        # the canonical single-replica blend: one density evaluation per call,
        # host arrays as the reference's main loop passes them
        _problem(PLAIN_32, name="density_32", kind="density", pattern="lam"),
        # odd axes with factors 3, 5 and 7 and an odd number of steps
        _problem(PLAIN_32, name="density_35x54x45", kind="density", pattern="lam", N=75, ens=2, **_grid((35, 54, 45))),
        # one 64^3 replica in FP32
        _problem(STRING_64, name="density_64_fp32", kind="density", pattern="lam", precision="fp32", **single),
        # one solver iteration of a small independent solve
        _problem(PLAIN_32, name="solve_48", kind="string", pattern="noise", N=96, ens=2, chi=18.0, f=0.4, **_grid(48)),
        # the headline workload: one iteration of the 16-replica 64^3 string, in
        # the reference's arithmetic and in FP32
        _problem(STRING_64, name="string16_64", kind="string", pattern="string"),
        _problem(STRING_64, name="string16_64_fp32", kind="string", pattern="string", precision="fp32"),
        # a large independent solve by Anderson mixing
        _problem(STRING_64, name="anderson_96", kind="anderson", pattern="noise", N=192, chi=18.0, iters=4, **single,
                 **_grid(96)),
        # eight 128^3 replicas in FP32 and two in FP64: one relaxation iteration,
        # the largest fields
        _problem(MIXED_128, name="relax8_128_fp32", kind="relax", pattern="gyroid", precision="fp32", iters=1),
        _problem(MIXED_128, name="relax2_128", kind="relax", pattern="gyroid", iters=1, strn=2),
        # the adjoint workload: all parameter derivatives of one replica
        _problem(ADJOINT_96, name="gradients_64x64x96", kind="gradients", pattern="lam", fcont=1, f=0.403),
        # the densities in little memory
        _problem(ADJOINT_96, name="ckpt_64x64x96", kind="ckpt", pattern="lam", K=13),
    ]


SMOOTH = [n for n in range(8, 129) if not [p for p in range(11, n + 1) if n % p == 0 and all(p % q for q in range(2, p))]]
CUBES = [16, 24, 32, 40, 48, 64, 80, 96, 128]
MOST = 16 * 20 * 128 * 64 ** 3  # grid points times contour steps of the largest listed case
MEMORY = 20e9                   # bytes of one context's propagator store


def _props(c):
    """Density evaluations of one pass."""
    per = {"step": 1.0 / c["N"], "density": 1, "ckpt": 2, "gradients": 2, "string": 20}
    return c["strn"] * (per[c["kind"]] if c["kind"] in per else c["iters"])


def draw(rng):
    while True:
        kind = rng.choice(["step", "density", "density", "relax", "string", "string", "anderson", "gradients", "ckpt"])
        if rng.random() < 0.5:  # most grids in use are cubes of a few sizes
            m = (rng.choice(CUBES),) * 3
        else:
            base = math.exp(rng.uniform(math.log(10), math.log(110)))
            m = tuple(rng.choice([n for n in SMOOTH if 0.6 * base <= n <= 1.6 * base]) for _ in range(3))
        strn = 1 if kind not in ("relax", "string") else int(round(math.exp(rng.uniform(0, math.log(16)))))
        dostring = int(kind == "string" and strn >= 3)
        c = dict(kind=kind, chi=round(rng.uniform(12, 22), 3), f=round(rng.uniform(0.3, 0.5), 3), ens=rng.choice([1, 2]),
                 phidb=round(rng.uniform(0.7, 1.0), 3), N=int(round(math.exp(rng.uniform(math.log(16), math.log(256))))),
                 alpha=0.1, strn=strn, fix=dostring * rng.randint(0, 1), dostring=dostring, fcont=int(kind == "gradients"),
                 precision="fp32" if kind in ("density", "relax", "string") and rng.random() < 0.35 else "fp64",
                 pattern="string" if dostring else rng.choice(["lam", "noise", "gyroid"]), **_grid(m, rng.choice([12.0, 16.0])))
        if kind in ("relax", "anderson"):
            c["iters"] = rng.randint(2, 6)
        if kind == "ckpt":
            c["K"] = rng.randint(5, 20)
        M = m[0] * m[1] * m[2]
        n1 = int(c["N"] * c["f"])
        if c["fcont"] and int(0.1 * c["N"]) > c["N"] - n1 - 1:
            continue
        if _props(c) * c["N"] * M <= MOST and (kind == "ckpt" or 16.0 * M * (c["N"] + 1) * strn <= MEMORY):
            return c


def _dims(c):
    return tuple(c["m%d" % i] for i in range(3)), tuple(c["D%d" % i] for i in range(3))


def _fields(c, seed):
    """W- and W+ of every replica, (strn, 2, M): the patterns of ``configs``, and
    a W+ of the size that a relaxation has reached after some iterations."""
    m, D = _dims(c)
    rng = np.random.default_rng([seed, 77])
    chi, strn = c["chi"], c["strn"]
    X, Y, Z = (2 * np.pi * np.arange(n) / n for n in m)
    X, Y, Z = X[:, None, None], Y[None, :, None], Z[None, None, :]
    noise = lambda s: rng.normal(0.0, s * chi, m)  # noqa: E731
    W = np.zeros((strn, 2) + m)
    if c["pattern"] == "string":
        lam = 0.6 * chi * np.cos(Z) + np.zeros(m)
        end = noise(0.02)
        for ii in range(strn):
            t = ii / (strn - 1.0)
            W[ii, 0] = (1 - t) * lam + t * end + (noise(0.01) if 0 < ii < strn - 1 else 0.0)
    else:
        for ii in range(strn):
            if c["pattern"] == "lam":
                W[ii, 0] = 0.4 * chi * np.cos(Z if c["strn"] % 2 else X) + noise(0.02)
            elif c["pattern"] == "gyroid":
                W[ii, 0] = 0.3 * chi * (np.sin(X) * np.cos(Y) + np.sin(Y) * np.cos(Z) + np.sin(Z) * np.cos(X)) + noise(0.03)
            else:
                W[ii, 0] = noise(0.1)
    W[:, 1] = 0.02 * W[:, 0] ** 2 / chi
    return W.reshape(strn, 2, -1)


def _context(c):
    m, D = _dims(c)
    return S.Context(m, D, c["N"], chi=c["chi"], f=c["f"], phidb=c["phidb"], ens=c["ens"], alpha=c["alpha"], strn=c["strn"],
                     fix=(c["fix"], c["fix"]), dostring=c["dostring"], precision=c["precision"], fcont=c["fcont"],
                     nostore=1 if c["kind"] == "ckpt" else 0, ckpt_K=c.get("K", 0))


def _pinned(*shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy()


def prepare(c, seed):
    W = _fields(c, seed)
    M = W.shape[-1]
    st = dict(c=c, M=M)
    if c["kind"] == "density":
        m, D = _dims(c)
        st["dens"] = S.Density(m, D, c["N"], c["ens"], c["alpha"], c["phidb"], c["f"], chi=c["chi"], precision=c["precision"])
        st["w"] = np.zeros(6 * M)
        st["w"][: 2 * M] = W[0].ravel()
        return st
    st["ctx"] = _context(c)
    if c["kind"] in ("relax", "string", "anderson"):
        # the fields live in the program's pinned buffers, as a checkpointing
        # driver keeps them
        st["w"], st["out"] = _pinned(c["strn"], 2 * M), _pinned(c["strn"], 2 * M)
        st["w"][:] = W.reshape(c["strn"], 2 * M)
    else:
        st["ctx"].set_fields_2m(0, np.ascontiguousarray(W[0].ravel()))
    if c["kind"] == "step":
        rng = np.random.default_rng([seed, 78])
        st["q"] = 1.0 + 0.3 * rng.normal(size=2 * M)
        st["s"] = int(rng.integers(c["N"]))
    return st


def run(st):
    c, M = st["c"], st["M"]
    kind = c["kind"]
    keep = (lambda a: torch.from_numpy(np.asarray(a)).float()) if c["precision"] == "fp32" else (lambda a: a)
    if kind == "density":
        lnQ, phis = st["dens"].props(st["w"], c["N"], c["alpha"], c["phidb"], c["f"])
        return {"conc": keep(st["w"][2 * M:]), "scalars": keep(np.append(phis, lnQ))}
    ctx = st["ctx"]
    if kind == "step":
        return ctx.do_step(0, st["q"], st["s"])
    if kind == "gradients":
        dL, dchi, df = ctx.gradients(0)
        return {"dL": dL, "dchi": dchi, "df": df}
    if kind == "ckpt":
        lnQ, phis, _ = ctx.props_ckpt(0, c["K"])
        return {"conc": ctx.get_conc(0)[0], "scalars": np.append(phis, lnQ)}
    for ii in range(c["strn"]):
        ctx.set_fields_2m(ii, st["w"][ii])
    if kind == "relax":
        extra = {"k": ctx.solve_field0_all(c["iters"] + 1, 1e-4)}
    elif kind == "anderson":
        n, err = ctx.anderson_solve(0, c["iters"], 1e-10)
        extra = {"n": n, "err": err}
    else:
        # iteration 1: one without the free energies that every 50th adds
        ctx.string_resume(1, 4000, 1e-3)
        r = ctx.string_step()
        ctx.string_end()
        extra = {"errs": keep(r["errs"]), "errs3": keep(r["errs3"]), "errtot": keep(np.array([r["errtot"]]))}
    for ii in range(c["strn"]):
        ctx.get_fields(ii, out=st["out"][ii])
    return {"W": keep(st["out"]), **extra}


def work(c):
    """Fields in, densities or fields out, and the 30 M log2 M operations of the
    six real transforms of q and of its conjugate in every contour step."""
    m, _ = _dims(c)
    M = m[0] * m[1] * m[2]
    flops = 30.0 * M * math.log2(M) * c["N"] * _props(c)
    moved = {"step": 6, "density": 6, "ckpt": 6, "gradients": 2}.get(c["kind"], 4) * 8.0 * M * c["strn"]
    return {"bytes": moved, "flops": flops}


# ---------------------------------------------------------------- in 64 bits
def _tables(c, L=None):
    """Per-axis squared wave vectors summed on the half spectrum, (2 pi n / L)^2."""
    m, D = _dims(c)
    dev = torch.device("cuda")
    L = torch.tensor(D, dtype=torch.float64, device=dev) if L is None else L
    k2 = 0.0
    for i in range(3):
        n = torch.fft.fftfreq(m[i], 1.0 / m[i], dtype=torch.float64, device=dev) if i < 2 else \
            torch.arange(m[2] // 2 + 1, dtype=torch.float64, device=dev)
        shape = [1, 1, 1]
        shape[i] = -1
        k2 = k2 + ((2 * math.pi * n / L[i]) ** 2).reshape(shape)
    return k2


def _sizes(c):
    N = c["N"]
    n1 = int(math.floor(N * c["f"])) if c["fcont"] else int(round(N * (round(N * c["f"]) / N)))
    return N, n1, N - n1, int(c["alpha"] * N)


def _richardson(q, w, k2, ds, m):
    """(4 two half steps - one full step) / 3 of q in the field w."""
    e4 = torch.exp(-w * ds / 4)
    e2 = e4 * e4
    h = torch.exp(-k2 * ds / 12)
    back = lambda v, g: torch.fft.irfftn(torch.fft.rfftn(v, dim=(-3, -2, -1)) * g, s=m, dim=(-3, -2, -1))  # noqa: E731
    half = e4 * back(e2 * back(e4 * q, h), h)
    return (4 * half - e2 * back(e2 * q, h * h)) / 3


def _props64(c, W):
    """Densities (R, 4, M), lnQ and phis of fields W (R, 2, M)."""
    m, _ = _dims(c)
    N, n1, n2, Nh = _sizes(c)
    R, M, ds = W.shape[0], W.shape[-1], 1.0 / N
    most = max(1, int(30e9 // (16.0 * M * (N + 1))))
    if R > most:
        parts = [_props64(c, W[i:i + most]) for i in range(0, R, most)]
        return tuple(torch.cat([p[k] for p in parts]) for k in range(3))
    k2 = _tables(c)
    wA, wB = (W[:, 0] + W[:, 1]).reshape((R,) + m), (W[:, 1] - W[:, 0]).reshape((R,) + m)
    q = torch.ones((N + 1, R, 2) + m, dtype=torch.float64, device=W.device)
    for s in range(N):
        w = torch.stack([wA if s < n1 else wB, wB if s < n2 else wA], 1)
        q[s + 1] = _richardson(q[s], w, k2, ds, m)
    QC, Q2 = q[N, :, 0].mean((1, 2, 3)), q[Nh, :, 1].mean((1, 2, 3))

    def simpson(lo, hi, end, first):
        # the reference's weights 1, 4, 2, 4, ..., 1 without an odd-count correction
        t = q[lo, :, first] * q[end - lo, :, 1] + q[hi, :, first] * q[end - hi, :, 1]
        for s in range(lo + 1, hi):
            t = t + (2 if (s - lo - 1) % 2 else 4) * q[s, :, first] * q[end - s, :, 1]
        return t.reshape(R, M)

    if c["ens"] == 1:
        lnQ = c["phidb"] * torch.log(QC) + (1 - c["phidb"]) / c["alpha"] * torch.log(Q2)
        zB, zC = (1 - c["phidb"]) / (Q2 * c["alpha"]), c["phidb"] / QC
    else:
        lnQ = Q2 + c["phidb"] * QC
        zB, zC = torch.ones_like(Q2), torch.full_like(QC, c["phidb"])
    rA = simpson(0, n1, N, 0) * (zC * ds / 3)[:, None]
    rB = simpson(n1, N, N, 0) * (zC * ds / 3)[:, None]
    rh = simpson(0, Nh, Nh, 1) * (zB * ds / 3)[:, None]
    conc = torch.stack([rA, rB + rh, rh, rB], 1)
    phis = torch.stack([(rA + rB).mean(1), rA.mean(1), (rB + rh).mean(1), torch.zeros_like(lnQ), rh.mean(1)], 1)
    return conc, lnQ, phis


def _relax64(c, W, reps, maxIter, tol):
    """The W+ relaxation (each replica by its own mixing parameter), in place."""
    lam, err, errt, k = ({r: v for r in reps} for v in (LAM0, 1.0, 1.0, 1))
    cur = [r for r in reps if k[r] < maxIter and err[r] > tol]
    while cur:
        conc = _props64(c, W[cur])[0]
        nxt = []
        for j, r in enumerate(cur):
            d = c["chi"] * (conc[j, 0] + conc[j, 1] - 1.0)
            err[r] = float((d * d).mean().sqrt())
            W[r, 1] += lam[r] * d
            lam[r] = min(0.1, lam[r] * 1.09) if err[r] < errt[r] else max(0.005, lam[r] / 1.10)
            errt[r] = err[r]
            k[r] += 1
            if k[r] < maxIter and err[r] > tol:
                nxt.append(r)
        cur = nxt
    return k


def _spline64(x, a):
    """Natural cubic spline of a (n, M) over the knots x: coefficients b, c, d of
    every interval, (n - 1, M) each."""
    n = len(x)
    h = x[1:] - x[:-1]
    A = np.eye(n)
    for i in range(1, n - 1):
        A[i, i - 1:i + 2] = h[i - 1], 2 * (h[i - 1] + h[i]), h[i]
    ht = torch.tensor(h, device=a.device)[:, None]
    s = (a[1:] - a[:-1]) / ht
    rhs = torch.zeros_like(a)
    rhs[1:-1] = 3 * (s[1:] - s[:-1])
    cc = torch.linalg.solve(torch.tensor(A, device=a.device), rhs)
    return s - ht * (cc[1:] + 2 * cc[:-1]) / 3, cc, (cc[1:] - cc[:-1]) / (3 * ht)


def _arc64(W):
    d = (W[1:, 0] - W[:-1, 0]).square().sum(1).sqrt().cpu().numpy()
    x = np.concatenate([[0.0], np.cumsum(d / d.sum())])
    x[-1] = 1.0
    return x


def _interval(x, v):
    return max([i for i in range(len(x)) if x[i] < v], default=0)


def _string64(c, W):
    strn, M = W.shape[0], W.shape[-1]
    reps = [r for r in range(strn) if not (c["fix"] and r in (0, strn - 1))]
    _relax64(c, W, reps, 20, 1e-3)
    conc = _props64(c, W[reps])[0]
    dev = torch.zeros_like(W)
    for j, r in enumerate(reps):
        dev[r, 0] = c["chi"] * (conc[j, 1] - conc[j, 0]) - 2 * W[r, 0]
        dev[r, 1] = c["chi"] * (conc[j, 0] + conc[j, 1] - 1.0)
    rms = lambda: (dev.square().sum((1, 2)) / (2.0 * M)).sqrt().cpu().numpy()  # noqa: E731
    errs = rms()
    errs3 = errs.copy()
    if c["dostring"]:
        x = _arc64(W)
        b, cc, d = _spline64(x, W[:, 0])
        for r in range(1, strn - 1):
            # the derivative at a knot is taken at the end of the interval before it
            i = _interval(x, x[r])
            dx = x[r] - x[i]
            t = b[i] + 2 * dx * cc[i] + 3 * dx * dx * d[i]
            dev[r, 0] -= t * (dev[r, 0] * t).sum() / t.square().sum()
        errs3[1:-1] = rms()[1:-1]
    W += LAM0 * dev
    if c["dostring"]:
        x = _arc64(W)
        b, cc, d = _spline64(x, W[:, 0])
        a = W[:, 0].clone()
        for r in range(1, strn - 1):
            v = r / (strn - 1.0)
            i = _interval(x, v)
            dx = v - x[i]
            W[r, 0] += LAM0 * (a[i] + dx * (b[i] + dx * (cc[i] + dx * d[i])) - a[r])
    return errs, errs3, np.array([math.sqrt(float((errs3 ** 2).mean()))])


def _anderson64(c, W, iters, nhist=10, lam=0.1):
    xs, ds = [], []
    for _ in range(iters):
        conc = _props64(c, W)[0][0]
        d = torch.cat([c["chi"] * (conc[1] - conc[0]) - 2 * W[0, 0], c["chi"] * (conc[0] + conc[1] - 1.0)])
        x = W.reshape(-1).clone()
        y = x + lam * d
        new = y.clone()
        if xs:
            D = torch.stack([d - v for v in ds])
            U = D @ D.T
            U += 1e-12 * U.trace() * torch.eye(len(ds), dtype=U.dtype, device=U.device)
            th = torch.linalg.solve(U, D @ d)
            for t, xi, di in zip(th, xs, ds):
                new -= t * (y - (xi + lam * di))
        W.copy_(new.reshape(W.shape))
        xs, ds = ([x] + xs)[:nhist], ([d] + ds)[:nhist]
    return float((d * d).mean().sqrt())


def _gradients64(c, W):
    """lnQ as a function of the box and of the junction, differentiated by autograd."""
    m, D = _dims(c)
    N, n1, n2, Nh = _sizes(c)
    ds = 1.0 / N
    L = torch.tensor(D, dtype=torch.float64, device=W.device, requires_grad=True)
    th = torch.tensor(N * c["f"] - n1, dtype=torch.float64, device=W.device, requires_grad=True)
    wA, wB = (W[0, 0] + W[0, 1]).reshape(m), (W[0, 1] - W[0, 0]).reshape(m)
    k2 = _tables(c, L)
    step = lambda q, w: torch.utils.checkpoint.checkpoint(_richardson, q, w, k2, ds, m, use_reentrant=False)  # noqa: E731
    q = torch.ones(m, dtype=torch.float64, device=W.device)
    p = q
    for s in range(N):
        q = step(q, wA if s < n1 else th * wA + (1 - th) * wB if s == n1 else wB)
    for _ in range(Nh):
        p = step(p, wB)
    QC, Q2 = q.mean(), p.mean()
    lnQ = c["phidb"] * torch.log(QC) + (1 - c["phidb"]) / c["alpha"] * torch.log(Q2) if c["ens"] == 1 else Q2 + c["phidb"] * QC
    gL, gt = torch.autograd.grad(lnQ, (L, th))
    return {"dL": -gL, "dchi": 0.25 - float(W[0, 0].square().mean()) / c["chi"] ** 2, "df": -N * float(gt)}


def exact(c, seed):
    m, _ = _dims(c)
    if _props(c) * c["N"] * m[0] * m[1] * m[2] > 1.1 * MOST:
        return None
    W = torch.tensor(_fields(c, seed), device="cuda")
    kind, M = c["kind"], W.shape[-1]
    if kind == "step":
        rng = np.random.default_rng([seed, 78])
        q = torch.tensor(1.0 + 0.3 * rng.normal(size=2 * M), device="cuda").reshape((2,) + m)
        s = int(rng.integers(c["N"]))
        N, n1, n2, _ = _sizes(c)
        wA, wB = (W[0, 0] + W[0, 1]).reshape(m), (W[0, 1] - W[0, 0]).reshape(m)
        w = torch.stack([wA if s < n1 else wB, wB if s < n2 else wA])
        return _richardson(q, w, _tables(c), 1.0 / N, m).reshape(-1)
    if kind == "gradients":
        return _gradients64(c, W)
    if kind in ("density", "ckpt"):
        conc, lnQ, phis = _props64(c, W)
        return {"conc": conc[0].reshape(-1), "scalars": torch.cat([phis[0], lnQ])}
    if kind == "relax":
        k = _relax64(c, W, list(range(c["strn"])), c["iters"] + 1, 1e-4)
        extra = {"k": np.array([k[r] for r in range(c["strn"])], np.int32)}
    elif kind == "anderson":
        extra = {"n": c["iters"], "err": _anderson64(c, W, c["iters"])}
    else:
        errs, errs3, tot = _string64(c, W)
        extra = {"errs": errs, "errs3": errs3, "errtot": tot}
    return {"W": W.reshape(c["strn"], 2 * M), **extra}
