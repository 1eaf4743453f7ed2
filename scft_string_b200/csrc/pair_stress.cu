// pair_stress.cu -- the box derivative of lnQ (stress_kernels.cu) on pairs packed
// as one complex field, FP64.
//
// A pair <y, dS/dL x> needs the same pointwise products and x, y, z transforms of
// x and of y, so x and y (times the power of two that makes their sizes alike, taken
// back in the sums) travel as c = x + i y through the slab and x passes of
// pair.cuh: half the transforms, no packing passes.  The Parseval sums come back
// from the packed spectra: for real x, y and an even weight g,
//   sum_k g Re(X conj Y)                = 1/2 sum_k g Im(C(k) C(-k)),
//   sum_k g Re(Wx conj Uy + Ux conj Wy) =     sum_k g Im(Cw(k) Cu(-k)).
// Per chunk of pairs six launches: slab forward (E4 c, E2 c), x forward of both
// (the first also times K2/M and x inverse), slab mid (E2), x forward, the sums,
// the final sums.
#include <algorithm>

#include "pair.cuh"
#include "pair_shapes.h"

namespace scft {
namespace {

using T = double;

struct StressSlab {
    const T *x, *y, *E4;
};

// k of pair p: the packed field is x + i 2^k y (pair.cuh)
__device__ __forceinline__ int stress_shift(const StressArgs<T> &a, const StressPairs &P, int p)
{
    const int *e = a.pexp + (size_t)a.slot * (a.g.Ns + 1) * 2;
    return pair_shift(__ldg(e + P.xe[p]), __ldg(e + P.ye[p]));
}

// real slabs of pair p at x index xi
__device__ __forceinline__ StressSlab stress_slab(const StressArgs<T> &a, const StressPairs &P, int p, size_t off)
{
    const size_t M = a.g.M, base = (size_t)a.slot * (a.g.Ns + 1);
    const int sel = P.sel[p];
    StressSlab s;
    s.x = a.hist + ((base + P.xs[p]) * 2 + P.xf[p]) * M + off;
    s.y = a.hist + ((base + P.ys[p]) * 2 + P.yf[p]) * M + off;
    s.E4 = (sel == 2 ? a.jtab + (size_t)a.slot * M : a.etab + ((size_t)a.slot * 2 + sel) * M) + off;
    return s;
}

// spectra of E4 (x + i y) (full = 0) and E2 (x + i y) (full = 1), y and z transformed
template <class PS>
__device__ __forceinline__ void stress_fwd_body(const PS &B, const StressArgs<T> &a, const StressPairs &P, int xi, int full,
                                                int p)
{
    const int row = B.row();
    const size_t off = (size_t)xi * B.area();
    B.load_tables(a.tw, a.g.m0);
    const StressSlab s = stress_slab(a, P, p, off);
    const T up = pair_pow2(stress_shift(a, P, p));
    B.sync();
    B.template real_space<false, true>([&](cplxd *v, int o) {
#pragma unroll
        for (int r = 0; r < PS::RA; r++) {
            T e = __ldg(s.E4 + o + row * r);
            if (full) e *= e;
            v[r] = {__ldg(s.x + o + row * r) * e, __ldg(s.y + o + row * r) * e * up};
        }
    });
    B.forward_passes((full ? a.S2 : a.S4) + (size_t)p * a.g.M + off, false, false);
}

// E2 D2 E4 c: inverse slab, times E2, forward slab
template <class PS>
__device__ __forceinline__ void stress_mid_body(const PS &B, const StressArgs<T> &a, const StressPairs &P, int xi, int p)
{
    const int row = B.row();
    const size_t off = (size_t)xi * B.area();
    B.load_tables(a.tw, a.g.m0);
    const StressSlab s = stress_slab(a, P, p, off);
    cplxd *spec = a.S4p + (size_t)p * a.g.M + off;
    __syncthreads();
    B.inverse_passes(spec);
    B.template real_space<true, true>([&](cplxd *v, int o) {
#pragma unroll
        for (int r = 0; r < PS::RA; r++) {
            const T e = __ldg(s.E4 + o + row * r), e2 = e * e;
            v[r].x *= e2;
            v[r].y *= e2;
        }
    });
    B.forward_passes(spec, false, false);
}

template <int M1, int M2, int CL>
__global__ void __launch_bounds__(PairSlab<M1, M2, CL>::NT, PairSlab<M1, M2, CL>::MINB)
    k_pair_stress_fwd(StressArgs<T> a, StressPairs P)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    stress_fwd_body(PairSlab<M1, M2, CL>(smem_raw), a, P, blockIdx.x / CL, blockIdx.y, blockIdx.z);
}

template <int M1, int M2, int CL>
__global__ void __launch_bounds__(PairSlab<M1, M2, CL>::NT, PairSlab<M1, M2, CL>::MINB)
    k_pair_stress_mid(StressArgs<T> a, StressPairs P)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    stress_mid_body(PairSlab<M1, M2, CL>(smem_raw), a, P, blockIdx.x / CL, blockIdx.z);
}

template <int RA>
__global__ void __launch_bounds__(512, 1) k_pair_stress_fwd_any(StressArgs<T> a, StressPairs P, PairAny q)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    stress_fwd_body(PairSlabAny<RA>(smem_raw, q), a, P, blockIdx.x, blockIdx.y, blockIdx.z);
}

template <int RA>
__global__ void __launch_bounds__(512, 1) k_pair_stress_mid_any(StressArgs<T> a, StressPairs P, PairAny q)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    stress_mid_body(PairSlabAny<RA>(smem_raw, q), a, P, blockIdx.x, blockIdx.z);
}

// x pass of one tile of kPairTile columns, in x positions R2 k1 + t of frequency
// k1 + r1 t.  first: spectrum sp = 0 of S4 is stored transformed, and times K2/M
// and transformed back into S4p; sp = 1 of S2 is stored transformed.  Otherwise
// S4p is transformed in place.
template <int R2>
__global__ void __launch_bounds__(256, 2) k_pair_stress_pencil(StressArgs<T> a, int first, int ra, int rb)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    constexpr int TC = kPairTile;
    const Geo &g = a.g;
    const int m0 = g.m0, m1 = g.m1, m2 = g.m2, ncol = m1 * m2, c0 = blockIdx.x * TC, r1 = m0 / R2;
    const int nc = ncol - c0 < TC ? ncol - c0 : TC, sp = blockIdx.y, p = blockIdx.z;
    cplxd *buf = reinterpret_cast<cplxd *>(smem_raw), *tw = buf + m0 * TC;
    cplxd *spec = (first ? (sp ? a.S2 : a.S4) : a.S4p) + (size_t)p * g.M + c0;
    cplxd *back = first && sp == 0 ? a.S4p + (size_t)p * g.M + c0 : nullptr;
    T *gx = reinterpret_cast<T *>(tw + m0), *colf = gx + m0;
    for (int i = threadIdx.x; i < m0; i += blockDim.x) {
        stc(tw + i, ldc_ro(a.tw + i));
        gx[i] = __ldg(a.kfac + i);
    }
    for (int t = threadIdx.x; t < nc; t += blockDim.x) {
        const int c = c0 + t, kz = c / m1, q = c - kz * m1, ky = q / rb + ra * (q % rb);
        colf[t] = __ldg(a.kfac + m0 + ky) * __ldg(a.kfac + m0 + m1 + (2 * kz > m2 ? m2 - kz : kz));
    }
    const unsigned mag = div_mag(nc);
    if (nc > 1)
        pair_any<-1, false, true>(r1, spec, buf, tw, nc * R2, nc, mag, 1, ncol, R2 * ncol, 1, TC, R2 * TC);
    else
        pair_any<-1, false, true>(r1, spec, buf, tw, R2, 1 << 30, 0, ncol, 0, R2 * ncol, TC, 0, R2 * TC);
    __syncthreads();
#pragma unroll 1
    for (int b = threadIdx.x; b < r1 * nc; b += blockDim.x) {
        const int k1 = div_by(b, mag), t = b - k1 * nc;
        cplxd v[R2], *q = buf + R2 * k1 * TC + t, *o = spec + (size_t)(R2 * k1) * ncol + t;
        v[0] = ldc(q);
#pragma unroll
        for (int i = 1; i < R2; i++) v[i] = cmul(ldc(q + i * TC), ldc(tw + k1 * i));
        Reg<T, R2, -1>::run(v);
#pragma unroll
        for (int i = 0; i < R2; i++) stc(o + (size_t)i * ncol, v[i]);
        if (!back) continue;
        const T ct = colf[t];
#pragma unroll
        for (int i = 0; i < R2; i++) {
            const T f = gx[k1 + r1 * i] * ct * a.invM;
            v[i].x *= f;
            v[i].y *= f;
        }
        Reg<T, R2, 1>::run(v);
#pragma unroll
        for (int i = 1; i < R2; i++) v[i] = cmulc(v[i], ldc(tw + k1 * i));
#pragma unroll
        for (int i = 0; i < R2; i++) stc(q + i * TC, v[i]);
    }
    if (!back) return;
    __syncthreads();
    if (nc > 1)
        pair_any<1, false, false, true>(r1, buf, back, tw, nc * R2, nc, mag, 1, TC, R2 * TC, 1, ncol, R2 * ncol);
    else
        pair_any<1, false, false, true>(r1, buf, back, tw, R2, 1 << 30, 0, TC, 0, R2 * TC, ncol, 0, R2 * ncol);
}

// The Parseval sums of pair blockIdx.y: rows 0-2 of its partials the K2 term of
// dL_i, rows 6-8 the K1 term (the layout of k_stress_final).  r1, r2: x radices;
// ra, rb: y radices of the position order.
__global__ void __launch_bounds__(256) k_pair_stress_sums(StressArgs<T> a, StressPairs P, int r1, int r2, int ra, int rb)
{
    __shared__ double sh[6][8];
    const Geo &g = a.g;
    const int m0 = g.m0, m1 = g.m1, m2 = g.m2, ncol = m1 * m2, p = blockIdx.y;
    const cplxd *W = a.S4p + (size_t)p * g.M, *U = a.S4 + (size_t)p * g.M, *F = a.S2 + (size_t)p * g.M;
    const double ds = 1.0 / g.Ns, PI = 3.14159265358979323846;
    const unsigned magc = div_mag(m1), magx = div_mag(r2), magy = div_mag(rb), magr1 = div_mag(r1), magra = div_mag(ra);
    double acc[6] = {0, 0, 0, 0, 0, 0};
    // one x position per turn of the outer loop, columns across the threads
    for (int px = blockIdx.x; px < m0; px += gridDim.x) {
        const int k1 = div_by(px, magx), kx = k1 + r1 * (px - k1 * r2), mx = kx ? m0 - kx : 0;
        const int tx = div_by(mx, magr1), qx = r2 * (mx - tx * r1) + tx;
        const int n0 = 2 * kx > m0 ? m0 - kx : kx;
        const double gx = __ldg(a.kfac + kx);
        for (int c = threadIdx.x; c < ncol; c += 256) {
            const int kz = div_by(c, magc), q = c - kz * m1, y1 = div_by(q, magy), ky = y1 + ra * (q - y1 * rb);
            const int mz = kz ? m2 - kz : 0, my = ky ? m1 - ky : 0, ty = div_by(my, magra);
            const size_t at = (size_t)px * ncol + c, mir = (size_t)qx * ncol + mz * m1 + rb * (my - ty * ra) + ty;
            const int n1 = 2 * ky > m1 ? m1 - ky : ky, n2 = 2 * kz > m2 ? m2 - kz : kz;
            const double K2 = gx * __ldg(a.kfac + m0 + ky) * __ldg(a.kfac + m0 + m1 + n2);
            const cplxd w = ldc(W + at), u = ldc(U + mir), f = ldc(F + at), h = ldc(F + mir);
            const double s2 = K2 * (ds / 12.0) * (w.x * u.y + w.y * u.x);
            const double s1 = K2 * K2 * (ds / 6.0) * 0.5 * (f.x * h.y + f.y * h.x);
            const double w0 = (double)n0 * n0, w1 = (double)n1 * n1, w2 = (double)n2 * n2;
            acc[0] += s2 * w0;
            acc[1] += s2 * w1;
            acc[2] += s2 * w2;
            acc[3] += s1 * w0;
            acc[4] += s1 * w1;
            acc[5] += s1 * w2;
        }
    }
#pragma unroll
    for (int i = 0; i < 6; i++) {
        double t = acc[i];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if ((threadIdx.x & 31) == 0) sh[i][threadIdx.x >> 5] = t;
    }
    __syncthreads();
    if (threadIdx.x < 6) {
        const int i = threadIdx.x;
        double t = 0;
        for (int j = 0; j < 8; j++) t += sh[i][j];
        const double L = a.L[i % 3];
        a.part[((size_t)p * 9 + (i < 3 ? i : 3 + i)) * gridDim.x + blockIdx.x] =
            t * pair_pow2(-stress_shift(a, P, p)) * 8.0 * PI * PI / (L * L * L);
    }
}

__global__ void k_pair_stress_final(const double *part, int nblk, int npairs, double invM, double *out)
{
    const int row = threadIdx.x >> 5, p = blockIdx.x;  // six warps: K2 terms, K1 terms
    __shared__ double s[6];
    double t = 0;
    for (int i = threadIdx.x & 31; i < nblk; i += 32) t += part[((size_t)p * 9 + (row < 3 ? row : 3 + row)) * nblk + i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if ((threadIdx.x & 31) == 0) s[row] = t;
    __syncthreads();
    if (threadIdx.x < 3) out[p * 3 + threadIdx.x] = invM * (4.0 / 3.0 * s[threadIdx.x] - 1.0 / 3.0 * s[3 + threadIdx.x]);
}

}  // namespace

int pair_stress_setup(int m0, int m1, int m2)
{
    cudaError_t e = cudaSuccess;
    auto up = [&](auto *fn, int bytes) {
        if (e == cudaSuccess) e = raise_dyn_smem(fn, bytes);
    };
    PairAny q;
    int r1, r2;
#define X(A, B)                                                          \
    if (m1 == A && m2 == B) {                                            \
        constexpr int CL = kCl<A, B>;                                    \
        up(k_pair_stress_fwd<A, B, CL>, PairSlab<A, B, CL>::SMEM);       \
        up(k_pair_stress_mid<A, B, CL>, PairSlab<A, B, CL>::SMEM);       \
    }
    PAIR_SLABS(X)
#undef X
    if (!pair_slab_fixed(m1, m2) && pair_any_plan(m1, m2, q)) switch (q.ra) {
#define X(A)                                                \
    case A:                                                 \
        up(k_pair_stress_fwd_any<A>, pair_any_smem(q));     \
        up(k_pair_stress_mid_any<A>, pair_any_smem(q));     \
        break;
            PAIR_RADICES(X)
#undef X
        }
    if (pair_x_radices(m0, r1, r2)) switch (r2) {
#define X(A) \
    case A: up(k_pair_stress_pencil<A>, pair_any_pencil_smem(m0)); break;
            PAIR_RADICES(X)
#undef X
        }
    return e == cudaSuccess ? 0 : -1;
}

int pair_stress_chunk(const StressArgs<T> &a, const StressPairs &P, double *out, cudaStream_t st)
{
    const Geo &g = a.g;
    PairAny q{};
    int ra = 1, rb = 1, r1 = 1, r2 = 1;
    pair_y_radices(g.m1, g.m2, ra, rb);
    pair_x_radices(g.m0, r1, r2);
    const bool any = !pair_slab_fixed(g.m1, g.m2) && pair_any_plan(g.m1, g.m2, q);
    auto slab = [&](int mid) {
#define X(A, B)                                                                                                       \
    if (g.m1 == A && g.m2 == B) {                                                                                     \
        constexpr int CL = kCl<A, B>;                                                                                 \
        using S = PairSlab<A, B, CL>;                                                                                 \
        if (mid)                                                                                                      \
            launch_ex(false, k_pair_stress_mid<A, B, CL>, dim3(CL * g.m0, 1, P.n), S::NT, S::SMEM, CL, 1, st, a, P);        \
        else                                                                                                          \
            launch_ex(false, k_pair_stress_fwd<A, B, CL>, dim3(CL * g.m0, 2, P.n), S::NT, S::SMEM, CL, 1, st, a, P);        \
    }
        PAIR_SLABS(X)
#undef X
        if (any) switch (q.ra) {
#define X(A)                                                                                                           \
    case A:                                                                                                            \
        if (mid)                                                                                                       \
            k_pair_stress_mid_any<A><<<dim3(g.m0, 1, P.n), pair_any_threads(q, 2 * g.m0 * P.n), pair_any_smem(q), st>>>(a, P, q);       \
        else                                                                                                           \
            k_pair_stress_fwd_any<A><<<dim3(g.m0, 2, P.n), pair_any_threads(q, 2 * g.m0 * P.n), pair_any_smem(q), st>>>(a, P, q);       \
        break;
                PAIR_RADICES(X)
#undef X
            }
    };
    auto pencil = [&](int first) {
        const dim3 grid((g.m1 * g.m2 + kPairTile - 1) / kPairTile, first ? 2 : 1, P.n);
        switch (r2) {
#define X(A) \
    case A: k_pair_stress_pencil<A><<<grid, 256, pair_any_pencil_smem(g.m0), st>>>(a, first, ra, rb); break;
            PAIR_RADICES(X)
#undef X
        }
    };
    slab(0);
    pencil(1);
    slab(1);
    pencil(0);
    const int nblk = std::min(g.m0, kStressSumBlocks);
    k_pair_stress_sums<<<dim3(nblk, P.n), 256, 0, st>>>(a, P, r1, r2, ra, rb);
    k_pair_stress_final<<<P.n, 192, 0, st>>>(a.part, nblk, P.n, 1.0 / g.M, out);
    return 6;
}

}  // namespace scft
