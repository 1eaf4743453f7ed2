// pair.cuh -- the contour step on q + i q^dagger (density.h:129-220).
//
// Every operation of the Richardson step is either a pointwise product with a
// real table (E4, E2 of the field that q or q^dagger sees) or a convolution
// with a real, even kernel (K1, K2).  Both keep the real and the imaginary part
// of a complex field apart, so q and q^dagger of a replica travel as ONE complex
// field c = q + i q^dagger: one complex 3-D transform replaces two real ones
// with no packing, unpacking or Hermitian bookkeeping in between.
//
// The transforms round both parts relative to the larger one, and where W- has a mean
// q and q^dagger drift apart by exp(2 <W-> s).  So the field is c = q + i 2^k q^dagger,
// k per replica and step, from the root mean squares of the full-step result P (which
// mid has in registers and which is of the size of the next q): a power of two costs
// no rounding, and either propagator keeps the precision of a transform of its own.
//
// Each 1-D transform of length N = R1 R2 is done in place, in two register
// passes with one trip through shared memory between them:
//   forward  n = j + R2 r:  R1-point DFTs over r, for every j, written back to
//            j + R2 k1; then times w^(j k1) and R2-point DFTs over j, written to
//            R2 k1 + k2.  Position R2 k1 + k2 then holds frequency k1 + R1 k2.
//   inverse  the same passes backwards.
// A pass reads and writes the same positions, so a transform needs one barrier
// between its two passes and none inside them.  A slab (fixed x) transforms y
// (M1 = RA RB), then z (M2 = RZ RC); the small second y pass and first z pass
// share registers where both fit.  The outer passes meet global memory in
// registers: the RA-point y pass with lanes along z, so that tables, partial
// results and the propagator store move in whole rows, and the RC-point z pass
// with lanes along y positions, so that a spectrum slab is stored [kz][p] in
// whole rows (p the y position of ky = p/RB + RA (p mod RB)); only the diffusion
// factors need to know that order.
//
// Loops that load (tables, partial results, twiddle factors) and loops that store
// are kept apart: no load may pass a store that could touch the same memory, so a
// mixed loop over a butterfly waits for one load after the other.  One step of one
// replica with mixed loops and without: 16^3 11.4 and 8.7 us, 48^3 20.4 and 18.3,
// 64^3 35.3 and 32.9, 128^3 195 and 189; 16 replicas of 64^3 14.3 and 13.6 each.
#pragma once
#include "common.cuh"
#include "dft.cuh"
#include "kernels.h"
#include "pdl.cuh"

namespace scft {

using cplxd = cplx<double>;

// 16-byte accesses (cplx<double> itself is only 8-byte aligned)
__device__ __forceinline__ cplxd ldc(const cplxd *p)
{
    const double2 v = *reinterpret_cast<const double2 *>(p);
    return {v.x, v.y};
}
// through L2: spectra and partial results written by other CTAs of an earlier phase
__device__ __forceinline__ cplxd ldc_cg(const cplxd *p)
{
    const double2 v = __ldcg(reinterpret_cast<const double2 *>(p));
    return {v.x, v.y};
}
__device__ __forceinline__ cplxd ldc_ro(const cplxd *p)
{
    const double2 v = __ldg(reinterpret_cast<const double2 *>(p));
    return {v.x, v.y};
}
__device__ __forceinline__ void stc(cplxd *p, cplxd v)
{
    *reinterpret_cast<double2 *>(p) = make_double2(v.x, v.y);
}

__device__ __forceinline__ int cluster_rank()
{
    unsigned r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return (int)r;
}
// the same shared-memory object of CTA `rank` of the cluster, as a generic address
__device__ __forceinline__ cplxd *cluster_map(cplxd *p, int rank)
{
    unsigned long long o;
    asm("mapa.u64 %0, %1, %2;" : "=l"(o) : "l"((unsigned long long)p), "r"(rank));
    return reinterpret_cast<cplxd *>(o);
}

__device__ __forceinline__ const double *pair_etab(const PropsArgs<double> &a, int slot, int fld, int s)
{
    const Geo &g = a.g;
    if (g.jon && s == (fld == 0 ? g.jq : g.jqd)) return a.jtab + (size_t)slot * g.M;
    const int sel = fld == 0 ? (s < g.n1 ? 0 : 1) : (s < g.n2 ? 1 : 0);
    return a.etab + ((size_t)slot * 2 + sel) * g.M;
}

// Transform plan of an M1 x M2 slab: M1 = RA RB, M2 = RZ RC.  MERGE: the
// RB-point y pass and the RZ-point z pass share registers (RB RZ elements per
// thread), so a 2-D transform makes two trips through shared memory instead of
// three.  WANT: threads per SM the registers are budgeted for.
template <int M1, int M2>
struct PairPlan;
#define PAIR_PLAN(m1, m2, ra, rb, rz, rc, merge, nt, want)                                 \
    template <>                                                                             \
    struct PairPlan<m1, m2> {                                                                      \
        static constexpr int RA = ra, RB = rb, RZ = rz, RC = rc, NT = nt;                             \
        static constexpr bool MERGE = merge;                                                          \
        static constexpr int WANT = want;  \
    };
PAIR_PLAN(16, 16, 8, 2, 2, 8, true, 64, 768)
PAIR_PLAN(24, 24, 8, 3, 3, 8, true, 96, 768)
PAIR_PLAN(32, 32, 8, 4, 4, 8, true, 128, 512)
PAIR_PLAN(40, 40, 10, 4, 4, 10, true, 160, 480)
PAIR_PLAN(48, 48, 12, 4, 4, 12, true, 192, 576)
PAIR_PLAN(64, 64, 16, 4, 4, 16, true, 256, 512)
PAIR_PLAN(64, 96, 16, 4, 4, 24, true, 384, 384)
PAIR_PLAN(80, 80, 20, 4, 4, 20, true, 320, 320)
PAIR_PLAN(96, 96, 24, 4, 4, 24, true, 384, 384)
PAIR_PLAN(128, 128, 16, 8, 16, 8, false, 1024, 512)  // two CTAs per slab only
#undef PAIR_PLAN

// threads of one of CL CTAs
__host__ __device__ constexpr int pair_nt(int nt, int cl) { return cl == 1 ? nt : (nt / cl + 31) / 32 * 32; }

// CL CTAs of a cluster may share a slab: each holds M1/CL of its rows (y
// positions).  Every pass but the RA-point y pass stays within those rows; that
// one takes M2/CL columns per CTA and reads and writes the other CTAs' rows
// through distributed shared memory, in place, between two cluster barriers.
template <int M1, int M2, int CL>
struct PairSlab : PairPlan<M1, M2> {
    using T = double;
    using Plan = PairPlan<M1, M2>;
    using Plan::MERGE;
    using Plan::RA;
    using Plan::RB;
    using Plan::RC;
    using Plan::RZ;
    static_assert(RA * RB == M1 && RZ * RC == M2 && RA % CL == 0 && M2 % CL == 0, "plan");
    static constexpr int CTAS = CL;
    static constexpr int NT = pair_nt(Plan::NT, CL), L = M1 / CL, RAL = RA / CL, S = M2 | 1;
    static constexpr int SMEM = (L * S + M1 + M2) * (int)sizeof(cplx<T>);
    static constexpr int FIT = 227 * 1024 / (SMEM + 1024), REG = Plan::WANT / NT;
    static constexpr int MINB = FIT < 1 ? 1 : FIT < REG ? FIT : REG < 1 ? 1 : REG;

    cplx<T> *buf, *twy, *twz, *part[CL];
    int rank;

    // radices of the y transform that the spectrum order depends on
    static __host__ __device__ void radices(int &ra, int &rb)
    {
        ra = RA;
        rb = RB;
    }

    __device__ __forceinline__ PairSlab(unsigned char *smem)
    {
        buf = reinterpret_cast<cplx<T> *>(smem);
        twy = buf + L * S;
        twz = twy + M1;
        rank = 0;
        part[0] = buf;
        if constexpr (CL > 1) {
            rank = cluster_rank();
#pragma unroll
            for (int i = 0; i < CL; i++) part[i] = cluster_map(buf, i);
        }
    }

    __device__ __forceinline__ void load_tables(const cplx<T> *tw, int m0) const
    {
        for (int i = threadIdx.x; i < M1 + M2; i += NT) stc(twy + i, ldc_ro(tw + m0 + i));
    }

    // all of the slab's CTAs
    static __device__ __forceinline__ void sync()
    {
        if constexpr (CL > 1) {
            pair_arrive();
            pair_wait();
        } else {
            __syncthreads();
        }
    }
    // after the last access to another CTA's rows
    static __device__ __forceinline__ void finish()
    {
        if constexpr (CL > 1) sync();
    }

    // loop of a pass over COUNT butterflies
    template <int COUNT, class F>
    static __device__ __forceinline__ void each(F f)
    {
        if constexpr (COUNT <= NT) {
            if (COUNT == NT || (int)threadIdx.x < COUNT) f((int)threadIdx.x);
        } else {
#pragma unroll 1
            for (int b = threadIdx.x; b < COUNT; b += NT) f(b);
        }
    }

    // spectrum slab src -> buf, up to the last (RA-point y) pass
    __device__ __forceinline__ void inverse_passes(const cplx<T> *src, bool split = false) const
    {
        const cplx<T> *own = src + rank * L;
        each<L * RZ>([&](int b) {
            const int y = b % L, k1 = b / L;
            cplx<T> v[RC], *p = buf + y * S + RC * k1;
#pragma unroll
            for (int i = 0; i < RC; i++) v[i] = ldc_cg(own + (i * RZ + k1) * M1 + y);
            Reg<T, RC, 1>::run(v);
#pragma unroll
            for (int i = 1; i < RC; i++) v[i] = cmulc(v[i], ldc(twz + k1 * i));
#pragma unroll
            for (int i = 0; i < RC; i++) stc(p + i, v[i]);
        });
        __syncthreads();
        if (split) pair_arrive();
        if constexpr (MERGE) {
            each<RAL * RC>([&](int b) {
                const int j = b % RC, k1 = b / RC;
                cplx<T> v[RB][RZ], *p = buf + RB * k1 * S + j;
#pragma unroll
                for (int i = 0; i < RB; i++) {
#pragma unroll
                    for (int r = 0; r < RZ; r++) v[i][r] = ldc(p + i * S + RC * r);
                    Reg<T, RZ, 1>::run(v[i]);
                }
#pragma unroll
                for (int r = 0; r < RZ; r++) {
                    cplx<T> u[RB];
#pragma unroll
                    for (int i = 0; i < RB; i++) u[i] = v[i][r];
                    Reg<T, RB, 1>::run(u);
#pragma unroll
                    for (int i = 0; i < RB; i++) v[i][r] = u[i];
                }
#pragma unroll
                for (int i = 1; i < RB; i++) {
                    const cplx<T> w = ldc(twy + (rank * RAL + k1) * i);
#pragma unroll
                    for (int r = 0; r < RZ; r++) v[i][r] = cmulc(v[i][r], w);
                }
#pragma unroll
                for (int i = 0; i < RB; i++)
#pragma unroll
                    for (int r = 0; r < RZ; r++) stc(p + i * S + RC * r, v[i][r]);
            });
        } else {
            each<L * RC>([&](int b) {
                const int y = b % L, j = b / L;
                cplx<T> v[RZ], *p = buf + y * S + j;
#pragma unroll
                for (int r = 0; r < RZ; r++) v[r] = ldc(p + RC * r);
                Reg<T, RZ, 1>::run(v);
#pragma unroll
                for (int r = 0; r < RZ; r++) stc(p + RC * r, v[r]);
            });
            __syncthreads();
            each<RAL * M2>([&](int b) {
                const int z = b % M2, k1 = b / M2;
                cplx<T> v[RB], *p = buf + RB * k1 * S + z;
#pragma unroll
                for (int i = 0; i < RB; i++) v[i] = ldc(p + i * S);
                Reg<T, RB, 1>::run(v);
#pragma unroll
                for (int i = 1; i < RB; i++) v[i] = cmulc(v[i], ldc(twy + (rank * RAL + k1) * i));
#pragma unroll
                for (int i = 0; i < RB; i++) stc(p + i * S, v[i]);
            });
        }
        sync();
    }

    // The RA-point y passes around real space: butterfly (z, j) holds the points
    // y = j + RB r of column z, lanes along z.  f(v, offset of (j, z) in the
    // slab) changes them in place (or fills them: INV = false); element r is at
    // offset + row() r.  With FWD the first forward y pass follows in registers.
    static __device__ __forceinline__ int row() { return RB * M2; }
    static __device__ __forceinline__ int area() { return M1 * M2; }
    template <bool INV, bool FWD, class F>
    __device__ __forceinline__ void real_space(F f) const
    {
        each<RB * M2 / CL>([&](int b) {
            const int z = rank * (M2 / CL) + b % (M2 / CL), j = b / (M2 / CL), at = j * S + z;
            cplx<T> v[RA];
            if (INV) {
#pragma unroll
                for (int r = 0; r < RA; r++) v[r] = ldc(part[r / RAL] + at + RB * (r % RAL) * S);
                Reg<T, RA, 1>::run(v);
            }
            f(v, j * M2 + z);
            if (FWD) {
                Reg<T, RA, -1>::run(v);
#pragma unroll
                for (int r = 0; r < RA; r++) stc(part[r / RAL] + at + RB * (r % RAL) * S, v[r]);
            }
        });
    }

    // buf after the first forward y pass -> spectrum slab dst
    __device__ __forceinline__ void forward_passes(cplx<T> *dst, bool split, bool last) const
    {
        sync();
        if constexpr (MERGE) {
            each<RAL * RC>([&](int b) {
                const int j = b % RC, k1 = b / RC;
                cplx<T> v[RB][RZ], *p = buf + RB * k1 * S + j;
#pragma unroll
                for (int i = 0; i < RB; i++) {
                    const cplx<T> w = ldc(twy + (rank * RAL + k1) * i);
#pragma unroll
                    for (int r = 0; r < RZ; r++) {
                        v[i][r] = ldc(p + i * S + RC * r);
                        if (i > 0) v[i][r] = cmul(v[i][r], w);
                    }
                }
#pragma unroll
                for (int r = 0; r < RZ; r++) {
                    cplx<T> u[RB];
#pragma unroll
                    for (int i = 0; i < RB; i++) u[i] = v[i][r];
                    Reg<T, RB, -1>::run(u);
#pragma unroll
                    for (int i = 0; i < RB; i++) v[i][r] = u[i];
                }
#pragma unroll
                for (int i = 0; i < RB; i++) {
                    Reg<T, RZ, -1>::run(v[i]);
#pragma unroll
                    for (int r = 0; r < RZ; r++) stc(p + i * S + RC * r, v[i][r]);
                }
            });
        } else {
            each<RAL * M2>([&](int b) {
                const int z = b % M2, k1 = b / M2;
                cplx<T> v[RB], *p = buf + RB * k1 * S + z;
                v[0] = ldc(p);
#pragma unroll
                for (int i = 1; i < RB; i++) v[i] = cmul(ldc(p + i * S), ldc(twy + (rank * RAL + k1) * i));
                Reg<T, RB, -1>::run(v);
#pragma unroll
                for (int i = 0; i < RB; i++) stc(p + i * S, v[i]);
            });
            __syncthreads();
            each<L * RC>([&](int b) {
                const int y = b % L, j = b / L;
                cplx<T> v[RZ], *p = buf + y * S + j;
#pragma unroll
                for (int r = 0; r < RZ; r++) v[r] = ldc(p + RC * r);
                Reg<T, RZ, -1>::run(v);
#pragma unroll
                for (int r = 0; r < RZ; r++) stc(p + RC * r, v[r]);
            });
        }
        __syncthreads();
        if (split) pair_wait();
        if (last) pdl_trigger();
        cplx<T> *own = dst + rank * L;
        each<L * RZ>([&](int b) {
            const int y = b % L, k1 = b / L;
            cplx<T> v[RC], *p = buf + y * S + RC * k1;
            v[0] = ldc(p);
#pragma unroll
            for (int i = 1; i < RC; i++) v[i] = cmul(ldc(p + i), ldc(twz + k1 * i));
            Reg<T, RC, -1>::run(v);
#pragma unroll
            for (int i = 0; i < RC; i++) stc(own + (i * RZ + k1) * M1 + y, v[i]);
        });
    }
};

// ---------------------------------------------------------------- other slab shapes
// The same slab transforms with sizes and radices known at run time: every axis
// of a length R1 R2 with both radices among 1-10, 12, 14, 15, 16.  The passes are
// out-of-line functions of the radix, shared by all kernels; only the real-space
// radix RA is a template parameter of the slab.  The small y and z passes stay
// apart (no merged pass).
#define PAIR_RADICES(X) X(1) X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(12) X(14) X(15) X(16)

struct PairAny {
    int m1, m2, ra, rb, rz, rc, S;
    unsigned mag1, mag2;  // floor(2^32 / m) + 1: b / m = umulhi(b, mag), exact for b m < 2^32
};

// Butterfly b = i + n k reads src[i si + k sk + r sr] and writes
// dst[i di + k dk + r dr], r < R; TW: times w^(k r), before a forward DFT, after
// an inverse one.
template <int R, int SIGN, bool TW, bool FROM_GLOBAL, bool TO_GLOBAL>
__device__ __noinline__ void pair_any_pass(const cplxd *src, cplxd *dst, const cplxd *tw, int count, int n, unsigned mag,
                                           int si, int sk, int sr, int di, int dk, int dr)
{
    if (!FROM_GLOBAL) __builtin_assume(__isShared(src));
    if (!TO_GLOBAL) __builtin_assume(__isShared(dst));
    if (TW) __builtin_assume(__isShared(tw));
#pragma unroll 1
    for (int b = threadIdx.x; b < count; b += blockDim.x) {
        const int k = (int)__umulhi((unsigned)b, mag), i = b - k * n;
        const cplxd *p = src + i * si + k * sk;
        cplxd v[R];
#pragma unroll
        for (int r = 0; r < R; r++) {
            v[r] = FROM_GLOBAL ? ldc_cg(p + r * sr) : ldc(p + r * sr);
            if (TW && SIGN < 0 && r > 0) v[r] = cmul(v[r], ldc(tw + k * r));
        }
        Reg<double, R, SIGN>::run(v);
        if (TW && SIGN > 0) {
#pragma unroll
            for (int r = 1; r < R; r++) v[r] = cmulc(v[r], ldc(tw + k * r));
        }
        cplxd *o = dst + i * di + k * dk;
#pragma unroll
        for (int r = 0; r < R; r++) stc(o + r * dr, v[r]);
    }
}

template <int SIGN, bool TW, bool FROM_GLOBAL, bool TO_GLOBAL = false>
__device__ __forceinline__ void pair_any(int R, const cplxd *src, cplxd *dst, const cplxd *tw, int count, int n,
                                         unsigned mag, int si, int sk, int sr, int di, int dk, int dr)
{
    switch (R) {
#define X(Q) \
    case Q: pair_any_pass<Q, SIGN, TW, FROM_GLOBAL, TO_GLOBAL>(src, dst, tw, count, n, mag, si, sk, sr, di, dk, dr); break;
        PAIR_RADICES(X)
#undef X
    }
}

template <int RA_>
struct PairSlabAny {
    using T = double;
    static constexpr int RA = RA_, CTAS = 1, rank = 0;
    PairAny q;
    cplx<T> *buf, *twy, *twz;

    __device__ __forceinline__ PairSlabAny(unsigned char *smem, const PairAny &plan) : q(plan)
    {
        buf = reinterpret_cast<cplx<T> *>(smem);
        twy = buf + q.m1 * q.S;
        twz = twy + q.m1;
    }
    static __device__ __forceinline__ void sync() { __syncthreads(); }
    static __device__ __forceinline__ void finish() {}
    __device__ __forceinline__ int row() const { return q.rb * q.m2; }
    __device__ __forceinline__ int area() const { return q.m1 * q.m2; }

    __device__ __forceinline__ void load_tables(const cplx<T> *tw, int m0) const
    {
        for (int i = threadIdx.x; i < q.m1 + q.m2; i += blockDim.x) stc(twy + i, ldc_ro(tw + m0 + i));
    }

    __device__ __forceinline__ void inverse_passes(const cplx<T> *src, bool split = false) const
    {
        pair_any<1, true, true>(q.rc, src, buf, twz, q.m1 * q.rz, q.m1, q.mag1, 1, q.m1, q.rz * q.m1, q.S, q.rc, 1);
        __syncthreads();
        if (split) pair_arrive();
        if (q.rz > 1) {
            pair_any<1, false, false>(q.rz, buf, buf, twz, q.m1 * q.rc, q.m1, q.mag1, q.S, 1, q.rc, q.S, 1, q.rc);
            __syncthreads();
        }
        if (q.rb > 1) {
            pair_any<1, true, false>(q.rb, buf, buf, twy, q.ra * q.m2, q.m2, q.mag2, 1, q.rb * q.S, q.S, 1, q.rb * q.S, q.S);
            __syncthreads();
        }
    }

    template <bool INV, bool FWD, class F>
    __device__ __forceinline__ void real_space(F f) const
    {
#pragma unroll 1
        for (int b = threadIdx.x; b < q.rb * q.m2; b += blockDim.x) {
            const int j = (int)__umulhi((unsigned)b, q.mag2), z = b - j * q.m2, step = q.rb * q.S;
            cplx<T> v[RA], *p = buf + j * q.S + z;
            if (INV) {
#pragma unroll
                for (int r = 0; r < RA; r++) v[r] = ldc(p + step * r);
                Reg<T, RA, 1>::run(v);
            }
            f(v, b);
            if (FWD) {
                Reg<T, RA, -1>::run(v);
#pragma unroll
                for (int r = 0; r < RA; r++) stc(p + step * r, v[r]);
            }
        }
    }

    __device__ __forceinline__ void forward_passes(cplx<T> *dst, bool split, bool last) const
    {
        __syncthreads();
        if (q.rb > 1) {
            pair_any<-1, true, false>(q.rb, buf, buf, twy, q.ra * q.m2, q.m2, q.mag2, 1, q.rb * q.S, q.S, 1, q.rb * q.S, q.S);
            __syncthreads();
        }
        if (q.rz > 1) {
            pair_any<-1, false, false>(q.rz, buf, buf, twz, q.m1 * q.rc, q.m1, q.mag1, q.S, 1, q.rc, q.S, 1, q.rc);
            __syncthreads();
        }
        if (split) pair_wait();
        if (last) pdl_trigger();
        pair_any<-1, true, false, true>(q.rc, buf, dst, twz, q.m1 * q.rz, q.m1, q.mag1, q.S, q.rc, 1, 1, q.m1, q.rz * q.m1);
    }
};

// ---------------------------------------------------------------- sizes of q and q^dagger
// a.pexp[slot][s][field]: binary exponent of the root mean square of q(s) and
// q^dagger(s); 0 for q(0) = 1.

// k of a step whose exponents are e0, e1; bounded as the powers are, which stay normal
__device__ __forceinline__ int pair_shift(int e0, int e1) { return min(max(e0 - e1, -1000), 1000); }
__device__ __forceinline__ double pair_pow2(int k) { return __hiloint2double((1023 + min(max(k, -1000), 1000)) << 20, 0); }

// sums over the CTA's threads of x and y -> out[0], out[1]; sh: shared memory, a complex
// per warp, that no thread reads any more (no static memory: the largest slabs leave none)
__device__ __forceinline__ void pair_cta_sums(double x, double y, double *out, cplxd *sh)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        x += __shfl_xor_sync(0xffffffffu, x, o);
        y += __shfl_xor_sync(0xffffffffu, y, o);
    }
    if ((threadIdx.x & 31) == 0) stc(sh + (threadIdx.x >> 5), {x, y});
    __syncthreads();
    if (threadIdx.x >= 32) return;
    const cplxd v = threadIdx.x < blockDim.x >> 5 ? ldc(sh + threadIdx.x) : cplxd{0, 0};
    x = v.x;
    y = v.y;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        x += __shfl_xor_sync(0xffffffffu, x, o);
        y += __shfl_xor_sync(0xffffffffu, y, o);
    }
    if (threadIdx.x == 0) stc(reinterpret_cast<cplxd *>(out), {x, y});
}

// Floors of the binary exponents of the root mean squares that n pairs of partial sums
// of squares give; bits 0 and 1 of the result: that sum was a normal number.  One warp,
// every lane has the result.
__device__ __forceinline__ int pair_rms_exponents(const double *sums, int n, double invM, int2 &e)
{
    double t0 = 0, t1 = 0;
    for (int i = threadIdx.x & 31; i < n; i += 32) {
        const double2 v = __ldcg(reinterpret_cast<const double2 *>(sums) + i);
        t0 += v.x;
        t1 += v.y;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        t0 += __shfl_xor_sync(0xffffffffu, t0, o);
        t1 += __shfl_xor_sync(0xffffffffu, t1, o);
    }
    // times 1.7: a uniform field of ones is not at the edge of a binade, where the last
    // bit of a sum would decide
    const int b0 = __double2hiint(t0 * invM * 1.7) >> 20, b1 = __double2hiint(t1 * invM * 1.7) >> 20;
    e = {(b0 - 1023) >> 1, (b1 - 1023) >> 1};
    return (b0 > 0 && b0 < 2047) | (b1 > 0 && b1 < 2047) << 1;
}

// Exponents of step s + 1 of a slot from mid's n partial sums of step s, whose terms
// were scaled by 2^-(exponent of q(s)) (and by 2^k in the second part); those of step s
// where a sum is no use.  Any CTA.
__device__ __forceinline__ void pair_next_exponents(const PropsArgs<double> &a, int slot, int s, int n)
{
    if (threadIdx.x >= 32) return;
    int2 *e = reinterpret_cast<int2 *>(a.pexp) + (size_t)slot * (a.g.Ns + 1) + s, d;
    const int2 now = __ldcg(e);
    const bool ok = pair_rms_exponents(a.partials + (size_t)slot * a.npart_stride, n, a.invM, d) == 3;
    if (threadIdx.x != 0) return;
    e[1] = ok ? make_int2(now.x + d.x, now.x + d.y - pair_shift(now.x, now.y)) : now;
}

// Exponents of a slice that no step led to, from the sums that n blocks took at three
// scales (pair_block_sums): in every thread of the CTA.
__device__ __forceinline__ int2 pair_slice_exponents(const double *sums, int n, double invM)
{
    __shared__ int2 sh;
    if (threadIdx.x < 32) {
        int2 e = {0, 0}, d;
        int got = 0;
        for (int j = 0; j < 3 && got < 3; j++) {
            const int have = pair_rms_exponents(sums + 2 * j * n, n, invM, d) & ~got, c = j == 0 ? 0 : j == 1 ? 600 : -600;
            if (have & 1) e.x = d.x - c;
            if (have & 2) e.y = d.y - c;
            got |= have;
        }
        if (threadIdx.x == 0) sh = e;
    }
    __syncthreads();
    return sh;
}

// Sums of squares of q and q^dagger at q, per block, at the scales 2^0, 2^600, 2^-600:
// no size of a normal number is lost.  For a grid of blocks along x.
__device__ __forceinline__ void pair_block_sums(const double *q, int M, double *sums)
{
    __shared__ double sh[6][32];
    const double c[3] = {1.0, pair_pow2(600), pair_pow2(-600)};
    double t[6] = {0, 0, 0, 0, 0, 0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < M; i += gridDim.x * blockDim.x) {
        const double x = q[i], y = q[i + M];
#pragma unroll
        for (int j = 0; j < 3; j++) {
            t[2 * j] = fma(x * c[j], x * c[j], t[2 * j]);
            t[2 * j + 1] = fma(y * c[j], y * c[j], t[2 * j + 1]);
        }
    }
#pragma unroll
    for (int k = 0; k < 6; k++) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t[k] += __shfl_xor_sync(0xffffffffu, t[k], o);
        if ((threadIdx.x & 31) == 0) sh[k][threadIdx.x >> 5] = t[k];
    }
    __syncthreads();
    if (threadIdx.x < 6) {
        double v = 0;
        for (int i = 0; i < (int)(blockDim.x >> 5); i++) v += sh[threadIdx.x][i];
        sums[2 * ((threadIdx.x >> 1) * gridDim.x + blockIdx.x) + (threadIdx.x & 1)] = v;
    }
}

// mid, slab x of a slot: sp = 0 the half-step spectrum (inverse slab, times E2,
// forward slab), sp = 1 the full-step spectrum (inverse slab, P = E2 qs1, and the sums
// of its squares)
template <class PS>
__device__ __forceinline__ void pair_mid_body(const PS &B, const PropsArgs<double> &a, int s, int x, int sp, int slot)
{
    using T = double;
    const Geo &g = a.g;
    const int area = B.area(), row = B.row();
    B.load_tables(a.tw, g.m0);
    const size_t off = (size_t)x * area;
    cplx<T> *spec = a.spec + ((size_t)slot * 2 + sp) * g.M + off;
    const T *Eq = pair_etab(a, slot, 0, s) + off, *Ep = pair_etab(a, slot, 1, s) + off;
    if (threadIdx.x == 0) {
        prefetch_l2(Eq, area * sizeof(T));
        prefetch_l2(Ep, area * sizeof(T));
    }
    __syncthreads();
    pdl_wait();
    if (pdl_early(g.m0)) pdl_trigger();
    const int eq = sp ? __ldcg(a.pexp + ((size_t)slot * (g.Ns + 1) + s) * 2) : 0;  // size of q(s)
    B.inverse_passes(spec);
    if (sp == 0) {
        B.template real_space<true, true>([&](cplx<T> *v, int o) {
#pragma unroll
            for (int r = 0; r < PS::RA; r++) {
                const T e0 = __ldg(Eq + o + row * r), e1 = __ldg(Ep + o + row * r);
                v[r].x *= e0 * e0;
                v[r].y *= e1 * e1;
            }
        });
        B.forward_passes(spec, false, true);
    } else {
        cplx<T> *P = reinterpret_cast<cplx<T> *>(a.pbuf) + (size_t)slot * g.M + off;
        T sx = 0, sy = 0;
        B.template real_space<true, false>([&](cplx<T> *v, int o) {
#pragma unroll
            for (int r = 0; r < PS::RA; r++) {
                const T e0 = __ldg(Eq + o + row * r), e1 = __ldg(Ep + o + row * r);
                v[r].x *= e0 * e0;
                v[r].y *= e1 * e1;
            }
            const T c = pair_pow2(-eq);
#pragma unroll
            for (int r = 0; r < PS::RA; r++) {
                stc(P + o + row * r, v[r]);
                const T x0 = v[r].x * c, y0 = v[r].y * c;
                sx = fma(x0, x0, sx);
                sy = fma(y0, y0, sy);
            }
        });
        // the twiddle factors (m1 + m2 of them, more than warps) have done their work
        pair_cta_sums(sx, sy, a.partials + (size_t)slot * a.npart_stride + 2 * (x * PS::CTAS + B.rank), B.twy);
        B.finish();
    }
}

// Products that the additions of the transform after them must not fuse with: whether a
// step follows another one, starts from a stored slice or makes its spectra in two
// CTAs, it then gives the same bits.
__device__ __forceinline__ cplxd rounded(cplxd v, double fx, double fy) { return {__dmul_rn(v.x, fx), __dmul_rn(v.y, fy)}; }

// combine, slab x of a slot: finishes step s (mode 0: Richardson combination;
// mode 1: q(s+1) = 1; mode 2: q(s+1) from the propagator store; mode 2 + n: the same,
// its sizes from the sums of n blocks) and starts step s + 1.  half: -1 one CTA makes both spectra; 0 / 1 this CTA makes only the
// half-step / full-step one (both repeat the inverse transform, which shortens
// the chain when the batch leaves SMs idle; they are a cluster of two) and half
// 0 stores q.  up: 2^k of step s + 1, down: 2^-k of step s.
template <class PS>
__device__ __forceinline__ void pair_combine_body(const PS &B, const PropsArgs<double> &a, int s, int mode, int x, int half,
                                                  int slot)
{
    using T = double;
    const Geo &g = a.g;
    const int area = B.area(), row = B.row();
    B.load_tables(a.tw, g.m0);
    const size_t M = g.M, off = (size_t)x * area;
    cplx<T> *specA = a.spec + (size_t)slot * 2 * M + off, *specB = specA + M;
    const int sn = s + 1;
    T *q0 = a.hist + ((size_t)slot * (g.Ns + 1) + sn) * 2 * M + off, *q1 = q0 + M;
    const bool next = sn < g.Ns, store = half != 1;
    const T *Nq = pair_etab(a, slot, 0, next ? sn : 0) + off, *Np = pair_etab(a, slot, 1, next ? sn : 0) + off;
    const T *Eq = pair_etab(a, slot, 0, s) + off, *Ep = pair_etab(a, slot, 1, s) + off;
    if (mode == 0 && threadIdx.x == 0) {
        prefetch_l2(Eq, area * sizeof(T));
        prefetch_l2(Ep, area * sizeof(T));
    }
    __syncthreads();
    pdl_wait();
    if (pdl_early(g.m0)) pdl_trigger();
    int *ex = a.pexp + ((size_t)slot * (g.Ns + 1) + sn) * 2;
    int2 now = {0, 0}, nxt = {0, 0};  // exponents of steps s and s + 1; 0 for q(0) = 1
    T up = 1, down = 1;
    if (mode != 1) nxt = __ldcg(reinterpret_cast<const int2 *>(ex));
    if (mode == 0) {
        now = __ldcg(reinterpret_cast<const int2 *>(ex) - 1);
        const cplx<T> *P = reinterpret_cast<const cplx<T> *>(a.pbuf) + (size_t)slot * M + off;
        if (threadIdx.x == 0) prefetch_l2(P, area * sizeof(cplx<T>));
        B.inverse_passes(specA, half >= 0);
        up = pair_pow2(nxt.x - nxt.y);  // here: the loads have had the passes to arrive
        down = pair_pow2(now.y - now.x);
        // Richardson, GPU_kernels.h:199-203
        auto finish = [&](cplx<T> *v, int o) {
#pragma unroll
            for (int r = 0; r < PS::RA; r++) {
                const cplx<T> p = ldc_cg(P + o + row * r);
                v[r].x = third(v[r].x * __ldg(Eq + o + row * r) * (T)4 - p.x);
                v[r].y = third(v[r].y * __ldg(Ep + o + row * r) * (T)4 - p.y) * down;
            }
            if (store) {
#pragma unroll
                for (int r = 0; r < PS::RA; r++) {
                    q0[o + row * r] = v[r].x;
                    q1[o + row * r] = v[r].y;
                }
            }
        };
        if (!next) {
            B.template real_space<true, false>(finish);
            B.finish();
            return;
        }
        B.template real_space<true, true>([&](cplx<T> *v, int o) {
            finish(v, o);
#pragma unroll
            for (int r = 0; r < PS::RA; r++) {
                T e0 = __ldg(Nq + o + row * r), e1 = __ldg(Np + o + row * r);
                if (half == 1) {
                    e0 *= e0;
                    e1 *= e1;
                }
                v[r] = rounded(v[r], e0, e1 * up);
            }
        });
    } else {
        if (mode == 1 && x == 0 && B.rank == 0 && store && threadIdx.x == 0) *reinterpret_cast<int2 *>(ex) = nxt;
        if (mode > 2) nxt = pair_slice_exponents(a.partials, mode - 2, a.invM);
        if (mode > 2 && x == 0 && B.rank == 0 && store && threadIdx.x == 0) *reinterpret_cast<int2 *>(ex) = nxt;
        up = pair_pow2(nxt.x - nxt.y);
        auto start = [&](cplx<T> *v, int o) {
#pragma unroll
            for (int r = 0; r < PS::RA; r++) {
                v[r] = mode == 1 ? cplx<T>{(T)1, (T)1} : cplx<T>{q0[o + row * r], q1[o + row * r]};
                T e0 = __ldg(Nq + o + row * r), e1 = __ldg(Np + o + row * r);
                if (half == 1) {
                    e0 *= e0;
                    e1 *= e1;
                }
                v[r] = rounded(v[r], e0, e1 * up);
            }
            if (mode == 1 && store) {
#pragma unroll
                for (int r = 0; r < PS::RA; r++) {
                    q0[o + row * r] = (T)1;
                    q1[o + row * r] = (T)1;
                }
            }
        };
        B.sync();  // every CTA of the slab runs before its rows are written
        B.template real_space<false, true>(start);
    }
    B.forward_passes(half == 1 ? specB : specA, half >= 0 && mode == 0, half >= 0);
    if (half >= 0) return;
    // full step input E2' q', from the slice this thread has just stored
    B.sync();
    B.template real_space<false, true>([&](cplx<T> *v, int o) {
#pragma unroll
        for (int r = 0; r < PS::RA; r++) {
            const T e0 = __ldg(Nq + o + row * r), e1 = __ldg(Np + o + row * r);
            v[r] = rounded({q0[o + row * r], q1[o + row * r]}, e0 * e0, e1 * e1 * up);
        }
    });
    B.forward_passes(specB, false, true);
}

// x pass of one tile of TC columns of spectrum sp (0: times K2, 1: times K1):
// forward transform, diffusion factor (Mult_self, GPU_kernels.h:175-181) and
// inverse transform; the 8-point passes around the factor share registers.
// Column c is [kz][p], p the y position of ky = p/rb + ra (p mod rb).
template <int M0, int TC>
struct PairPencil {
    static constexpr int SMEM = (M0 * TC + M0) * (int)sizeof(cplx<double>) + (M0 + TC) * (int)sizeof(double);
};

template <int M0, int TC, int NT>
__device__ __forceinline__ void pair_pencil_body(const PropsArgs<double> &a, int tile, int sp, int slot, int ra, int rb,
                                                 unsigned char *smem)
{
    using T = double;
    constexpr int R1 = M0 / 8, R2 = 8;
    const Geo &g = a.g;
    const int m1 = g.m1, m2 = g.m2, ncol = m1 * m2, c0 = tile * TC;
    cplx<T> *buf = reinterpret_cast<cplx<T> *>(smem);
    cplx<T> *tw = buf + M0 * TC;
    T *gx = reinterpret_cast<T *>(tw + M0), *colf = gx + M0;
    cplx<T> *spec = a.spec + ((size_t)slot * 2 + sp) * g.M + c0;
    const T *kf = a.kfac + (size_t)__ldg(a.slot_rep + slot) * a.kf_stride;  // the replica's box
    for (int i = threadIdx.x; i < M0; i += NT) {
        stc(tw + i, ldc_ro(a.tw + i));
        gx[i] = __ldg(kf + i);
    }
    for (int t = threadIdx.x; t < TC; t += NT) {
        const int c = c0 + t, kz = c / m1, p = c - kz * m1, ky = p / rb + ra * (p % rb);
        colf[t] = c < ncol ? __ldg(kf + M0 + ky) * __ldg(kf + M0 + m1 + (2 * kz > m2 ? m2 - kz : kz)) : (T)0;
    }
    pdl_wait();
    if (pdl_early(g.m0)) pdl_trigger();
#pragma unroll 1
    for (int b = threadIdx.x; b < R2 * TC; b += NT) {
        const int t = b % TC, j = b / TC;
        if (c0 + t < ncol) {
            cplx<T> v[R1];
#pragma unroll
            for (int r = 0; r < R1; r++) v[r] = ldc_cg(spec + (size_t)(j + R2 * r) * ncol + t);
            Reg<T, R1, -1>::run(v);
#pragma unroll
            for (int r = 0; r < R1; r++) stc(buf + (j + R2 * r) * TC + t, v[r]);
        }
    }
    __syncthreads();
    const T invM = a.invM, Mreal = a.Mreal;
#pragma unroll 1
    for (int b = threadIdx.x; b < R1 * TC; b += NT) {
        const int t = b % TC, k1 = b / TC;
        if (c0 + t < ncol) {
            cplx<T> v[R2], *p = buf + R2 * k1 * TC + t;
            v[0] = ldc(p);
#pragma unroll
            for (int i = 1; i < R2; i++) v[i] = cmul(ldc(p + i * TC), ldc(tw + k1 * i));
            Reg<T, R2, -1>::run(v);
            // K2 = g/M, K1 = g^2/M  (Prepare_dev_expKsq2_expKsq, GPU_kernels.h:207-213)
            const T ct = colf[t];
#pragma unroll
            for (int i = 0; i < R2; i++) {
                const T k2 = gx[k1 + R1 * i] * ct * invM;
                const T f = sp == 0 ? k2 : k2 * k2 * Mreal;
                v[i].x *= f;
                v[i].y *= f;
            }
            Reg<T, R2, 1>::run(v);
#pragma unroll
            for (int i = 1; i < R2; i++) v[i] = cmulc(v[i], ldc(tw + k1 * i));
#pragma unroll
            for (int i = 0; i < R2; i++) stc(p + i * TC, v[i]);
        }
    }
    __syncthreads();
    pdl_trigger();
#pragma unroll 1
    for (int b = threadIdx.x; b < R2 * TC; b += NT) {
        const int t = b % TC, j = b / TC;
        if (c0 + t < ncol) {
            cplx<T> v[R1];
#pragma unroll
            for (int r = 0; r < R1; r++) v[r] = ldc(buf + (j + R2 * r) * TC + t);
            Reg<T, R1, 1>::run(v);
#pragma unroll
            for (int r = 0; r < R1; r++) stc(spec + (size_t)(j + R2 * r) * ncol + t, v[r]);
        }
    }
}

// The same x pass with m0 = r1 R2 and the first radix known at run time.
template <int R2, int TC>
__device__ __forceinline__ void pair_pencil_any_body(const PropsArgs<double> &a, int tile, int sp, int slot, int ra, int rb,
                                                     unsigned char *smem)
{
    using T = double;
    const Geo &g = a.g;
    const int m0 = g.m0, m1 = g.m1, m2 = g.m2, ncol = m1 * m2, c0 = tile * TC, r1 = m0 / R2;
    const int nc = ncol - c0 < TC ? ncol - c0 : TC;
    cplx<T> *buf = reinterpret_cast<cplx<T> *>(smem);
    cplx<T> *tw = buf + m0 * TC;
    T *gx = reinterpret_cast<T *>(tw + m0), *colf = gx + m0;
    cplx<T> *spec = a.spec + ((size_t)slot * 2 + sp) * g.M + c0;
    const T *kf = a.kfac + (size_t)__ldg(a.slot_rep + slot) * a.kf_stride;
    for (int i = threadIdx.x; i < m0; i += blockDim.x) {
        stc(tw + i, ldc_ro(a.tw + i));
        gx[i] = __ldg(kf + i);
    }
    for (int t = threadIdx.x; t < nc; t += blockDim.x) {
        const int c = c0 + t, kz = c / m1, p = c - kz * m1, ky = p / rb + ra * (p % rb);
        colf[t] = __ldg(kf + m0 + ky) * __ldg(kf + m0 + m1 + (2 * kz > m2 ? m2 - kz : kz));
    }
    pdl_wait();
    if (pdl_early(g.m0)) pdl_trigger();
    const unsigned mag = 0xffffffffu / (unsigned)nc + 1u;  // nc = 1: butterfly b is (0, b)
    auto outer = [&](int b, int &t, int &j) {
        j = nc > 1 ? (int)__umulhi((unsigned)b, mag) : b;
        t = b - j * nc;
    };
    if (nc > 1) {
        pair_any<-1, false, true>(r1, spec, buf, tw, nc * R2, nc, mag, 1, ncol, R2 * ncol, 1, TC, R2 * TC);
    } else {
        // one column left: butterfly index b = R2-point position
        pair_any<-1, false, true>(r1, spec, buf, tw, R2, 1 << 30, 0, ncol, 0, R2 * ncol, TC, 0, R2 * TC);
    }
    __syncthreads();
    const T invM = a.invM, Mreal = a.Mreal;
#pragma unroll 1
    for (int b = threadIdx.x; b < r1 * nc; b += blockDim.x) {
        int t, k1;
        outer(b, t, k1);
        cplx<T> v[R2], *p = buf + R2 * k1 * TC + t;
        v[0] = ldc(p);
#pragma unroll
        for (int i = 1; i < R2; i++) v[i] = cmul(ldc(p + i * TC), ldc(tw + k1 * i));
        Reg<T, R2, -1>::run(v);
        const T ct = colf[t];
#pragma unroll
        for (int i = 0; i < R2; i++) {
            const T k2 = gx[k1 + r1 * i] * ct * invM;
            const T f = sp == 0 ? k2 : k2 * k2 * Mreal;
            v[i].x *= f;
            v[i].y *= f;
        }
        Reg<T, R2, 1>::run(v);
#pragma unroll
        for (int i = 1; i < R2; i++) v[i] = cmulc(v[i], ldc(tw + k1 * i));
#pragma unroll
        for (int i = 0; i < R2; i++) stc(p + i * TC, v[i]);
    }
    __syncthreads();
    pdl_trigger();
    if (nc > 1) {
        pair_any<1, false, false, true>(r1, buf, spec, tw, nc * R2, nc, mag, 1, TC, R2 * TC, 1, ncol, R2 * ncol);
    } else {
        pair_any<1, false, false, true>(r1, buf, spec, tw, R2, 1 << 30, 0, TC, 0, R2 * TC, ncol, 0, R2 * ncol);
    }
}

}  // namespace scft
