// real_slab.cuh -- the FP32 slab kernels of the compile-time shapes.
//
// The same transforms as slab_forward_fixed / slab_inverse_fixed (fft.cuh): two
// real rows per complex z line, the kz = 0 and kz = M2/2 columns as one complex y
// column, every butterfly with the same inputs, twiddle factors and order of
// operations, so the results are the same bits.  What differs is how a thread
// covers a line: an M = 8 R point line takes a radix-8 pass and one pass over the
// R remaining points, whose stages (12 = 4 3, 16 = 8 2, ...) share registers; the
// unpacking of row pairs is done by the thread that transforms both rows' y
// columns, in place; spectra are read from and written to global memory by the
// outer passes themselves, and real space is met in registers.  A slab transform
// makes three trips through shared memory; it made five to seven, with a barrier
// before and after each stage.
//
// The real-space operands (the E table, P, q) come and go through padded copies
// in shared memory, moved by bulk copies a row pair at a time: a thread holds the
// points n + 8 t of two rows, so a warp would touch global memory in runs of 32
// bytes, four wavefronts an access (they were 40 % of the LSU's work at 64^3; 16
// replicas of 64^3 9.15 -> 8.75 us per replica step).  Slabs of 96 and 128 rows go
// without: the copies would halve the CTAs per SM (96^3 44 us without, 57 with).
//
// Products that feed an addition directly are rounded on their own (__fmul_rn):
// they went through shared memory before, and a fused multiply-add would round
// differently.
#pragma once
#include "common.cuh"
#include "fft.cuh"
#include "kernels.h"
#include "pdl.cuh"
#include "tma.cuh"

namespace scft {

using cplxf = cplx<float>;

__device__ __forceinline__ cplxf ldf(const cplxf *p)
{
    const float2 v = *reinterpret_cast<const float2 *>(p);
    return {v.x, v.y};
}
__device__ __forceinline__ cplxf ldf_cg(const cplxf *p)
{
    const float2 v = __ldcg(reinterpret_cast<const float2 *>(p));
    return {v.x, v.y};
}
__device__ __forceinline__ void stf(cplxf *p, cplxf v) { *reinterpret_cast<float2 *>(p) = make_float2(v.x, v.y); }

// a w and a conj(w), with the roundings that cmul and cmulc compile to in the
// shared-memory stages (which product is rounded, which is fused)
template <int SIGN>
__device__ __forceinline__ cplxf twiddle(cplxf a, cplxf w)
{
    if (SIGN < 0) return {__fmaf_rn(a.x, w.x, -__fmul_rn(a.y, w.y)), __fmaf_rn(a.y, w.x, __fmul_rn(a.x, w.y))};
    return {__fmaf_rn(a.x, w.x, __fmul_rn(a.y, w.y)), __fmaf_rn(a.y, w.x, -__fmul_rn(a.x, w.y))};
}

// second stage radix of the R points left after radix 8 (1: one stage)
__host__ __device__ constexpr int tail_b(int r) { return r == 6 || r == 12 ? 3 : r == 16 ? 2 : 1; }

// The stages after the radix-8 one of a length-N line (N = 8 RA RB): inputs j = 0
// .. RA RB - 1 of output class k1, result slot t holds index k1 + 8 t.
template <int RA, int RB, int SIGN>
__device__ __forceinline__ void tail_run(cplxf *v, int k1, const cplxf *tw)
{
    constexpr int R = RA * RB;
    cplxf o[R];
#pragma unroll
    for (int j = 0; j < RB; j++) {
        cplxf u[RA];
#pragma unroll
        for (int a = 0; a < RA; a++) {
            u[a] = v[j + RB * a];
            if (a > 0) u[a] = twiddle<SIGN>(u[a], ldf(tw + RB * a * k1));
        }
        Dft<float, RA>::run(u, SIGN, nullptr, 0);
#pragma unroll
        for (int a = 0; a < RA; a++) {
            if (RB > 1 && j > 0) u[a] = twiddle<SIGN>(u[a], ldf(tw + j * (k1 + 8 * a)));
            o[RB * a + j] = u[a];
        }
    }
#pragma unroll
    for (int a = 0; a < RA; a++) {
        if constexpr (RB > 1) Dft<float, RB>::run(o + RB * a, SIGN, nullptr, 0);
#pragma unroll
        for (int b = 0; b < RB; b++) v[a + RA * b] = o[RB * a + b];
    }
}

template <int M1, int M2>
struct RealSlab {
    static constexpr int RY = M1 / 8, RZ = M2 / 8, H = M2 / 2, MK2 = H + 1, NP = M1 / 2, S = M2 + 1, NT = 4 * M1;
    static constexpr int BY = tail_b(RY), BZ = tail_b(RZ);
    static constexpr bool FUSED = RZ == 8;  // the last inverse and the first forward z pass hold the same points
    // staged copy of a real slab: row pair p at stage_at(p), padded so that the four
    // row pairs of a warp fall into different banks
    static constexpr int STAGE = NP * (2 * M2 + 8) + 16 * (NP / 8);  // floats
    static constexpr int BASE = 128 + (NP * S + M1 + M1 + M2) * (int)sizeof(cplxf);
    static constexpr bool STAGED = M1 <= 64;
    static constexpr int SMEM_MID = BASE + (STAGED ? STAGE * 4 : 0), SMEM = BASE + (STAGED ? 2 * STAGE * 4 : 0);
    static constexpr int FIT = 227 * 1024 / (SMEM + 1024), REG = 1024 / NT;
    static constexpr int MINB = FIT < 1 ? 1 : FIT < REG ? FIT : REG < 1 ? 1 : REG;
    static_assert(RY % 2 == 0 && M1 % 8 == 0 && M2 % 8 == 0, "shape");

    uint64_t *bars;
    cplxf *buf, *col, *twy, *twz;
    float *Es, *Qs;  // staged E table; staged P, then q'

    static __device__ __forceinline__ int stage_at(int p) { return p * (2 * M2 + 8) + 16 * (p >> 3); }

    // Bulk copies of a real slab, a row pair each, by warp 0.
    __device__ __forceinline__ void stage_in(float *dst, const float *src, uint64_t *bar) const
    {
        if (threadIdx.x >= 32) return;
        if (threadIdx.x == 0) mbar_expect_tx(bar, M1 * M2 * sizeof(float));
        __syncwarp();
        for (int p = threadIdx.x; p < NP; p += 32) bulk_g2s(dst + stage_at(p), src + p * 2 * M2, 2 * M2 * sizeof(float), bar);
    }
    // after a fence by the writers and a barrier; stage_out_done before the CTA exits
    __device__ __forceinline__ void stage_out(float *dst, const float *src) const
    {
        if (threadIdx.x >= 32) return;
        for (int p = threadIdx.x; p < NP; p += 32) bulk_s2g(dst + p * 2 * M2, src + stage_at(p), 2 * M2 * sizeof(float));
        bulk_commit();
    }
    __device__ __forceinline__ void stage_out_done() const
    {
        if (threadIdx.x < 32) tma_store_wait_read();
    }

    __device__ __forceinline__ RealSlab(unsigned char *smem)
    {
        bars = reinterpret_cast<uint64_t *>(smem);
        buf = reinterpret_cast<cplxf *>(smem + 128);
        Es = reinterpret_cast<float *>(smem + BASE);
        Qs = Es + STAGE;
        col = buf + NP * S;
        twy = col + M1;
        twz = twy + M1;
    }

    __device__ __forceinline__ void load_tables(const cplxf *tw, int m0) const
    {
        for (int i = threadIdx.x; i < M1 + M2; i += NT) stf(twy + i, ldf(tw + m0 + i));
    }

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

    // Row pair of index t where 8 lanes cover z: the two row pairs of a half-warp
    // are 8 apart, 8 S = 8 (mod 16) elements, in the other half of the banks.
    static __device__ __forceinline__ int prow(int t)
    {
        if constexpr (NP % 16 == 0)
            return (t & ~15) + ((t & 15) >> 1) + ((t & 1) << 3);
        else
            return t;
    }
    // slot of the partner column of kz in a packed row
    static __device__ __forceinline__ int mirror(int kz) { return kz ? M2 - kz : H; }

    // spectrum slab src [ky][kz] -> packed rows, up to the last z pass
    __device__ __forceinline__ void inverse_passes(const cplxf *src) const
    {
        each<H * RY>([&](int b) {
            const int kz = b % H, kk = b / H;
            cplxf v[8];
#pragma unroll
            for (int r = 0; r < 8; r++) v[r] = ldf_cg(src + (kk + RY * r) * MK2 + kz);
            if (kz == 0) {
#pragma unroll
                for (int r = 0; r < 8; r++) {
                    const cplxf ch = ldf_cg(src + (kk + RY * r) * MK2 + H);
                    v[r] = {v[r].x - ch.y, v[r].y + ch.x};
                }
            }
            Dft<float, 8>::run(v, 1, nullptr, 0);
            cplxf *p = buf + 4 * kk * S;
#pragma unroll
            for (int n = 0; n < 8; n += 2) {
                stf(p + (n / 2) * S + kz, v[n]);
                stf(p + (n / 2) * S + mirror(kz), v[n + 1]);
            }
        });
        __syncthreads();
        each<H * 4>([&](int b) {
            const int kz = b % H, n = b / H;
            cplxf e[RY], o[RY], *p = buf + n * S + kz, *q = buf + n * S + mirror(kz);
#pragma unroll
            for (int k = 0; k < RY; k++) {
                e[k] = ldf(p + 4 * k * S);
                o[k] = ldf(q + 4 * k * S);
            }
            tail_run<RY / BY, BY, 1>(e, 2 * n, twy);
            tail_run<RY / BY, BY, 1>(o, 2 * n + 1, twy);
            // rows 2p and 2p + 1 as one complex row
#pragma unroll
            for (int t = 0; t < RY; t++) {
                const cplxf A = e[t], B = o[t];
                if (kz) {
                    stf(p + 4 * t * S, {A.x - B.y, A.y + B.x});
                    stf(q + 4 * t * S, {A.x + B.y, B.x - A.y});
                } else {
                    stf(p + 4 * t * S, {A.x, B.x});
                    stf(q + 4 * t * S, {A.y, B.y});
                }
            }
        });
        __syncthreads();
        constexpr int PER = (NP * RZ + NT - 1) / NT;
        cplxf v[PER][8];
#pragma unroll
        for (int i = 0; i < PER; i++) {
            const int b = threadIdx.x + i * NT;
            if ((NP * RZ) % NT == 0 || b < NP * RZ) {
                const int p = b % NP, kk = b / NP;
#pragma unroll
                for (int r = 0; r < 8; r++) v[i][r] = ldf(buf + p * S + kk + RZ * r);
                Dft<float, 8>::run(v[i], 1, nullptr, 0);
            }
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < PER; i++) {
            const int b = threadIdx.x + i * NT;
            if ((NP * RZ) % NT == 0 || b < NP * RZ) {
                const int p = b % NP, kk = b / NP;
#pragma unroll
                for (int r = 0; r < 8; r++) stf(buf + p * S + r + 8 * kk, v[i][r]);
            }
        }
        __syncthreads();
    }

    // Real space: a thread holds the points z = n + 8 t, t < RZ, of rows 2p (.x) and
    // 2p + 1 (.y).  f(v, offset of (2p, n) in the slab, in a staged copy) changes (INV)
    // or fills them; FWD hands them to forward_passes.
    template <bool INV, bool FWD, class F>
    __device__ __forceinline__ void real_space(F f) const
    {
        const int n = threadIdx.x & 7, p = prow(threadIdx.x >> 3);
        cplxf v[RZ], *q = buf + p * S + n;
        if (INV) {
#pragma unroll
            for (int t = 0; t < RZ; t++) v[t] = ldf(q + 8 * t);
            tail_run<RZ / BZ, BZ, 1>(v, n, twz);
        }
        f(v, 2 * p * M2 + n, stage_at(p) + n);
        if (FWD) {
            if constexpr (FUSED) Dft<float, 8>::run(v, -1, nullptr, 0);
#pragma unroll
            for (int t = 0; t < RZ; t++) stf(q + 8 * t, v[t]);
        }
    }

    // packed rows -> spectrum slab dst [ky][kz]
    __device__ __forceinline__ void forward_passes(cplxf *dst, bool last) const
    {
        __syncthreads();
        if constexpr (!FUSED) {
            each<NP * RZ>([&](int b) {
                const int j = b % RZ, p = b / RZ;
                cplxf v[8], *q = buf + p * S + j;
#pragma unroll
                for (int r = 0; r < 8; r++) v[r] = ldf(q + RZ * r);
                Dft<float, 8>::run(v, -1, nullptr, 0);
#pragma unroll
                for (int r = 0; r < 8; r++) stf(q + RZ * r, v[r]);
            });
            __syncthreads();
        }
        {
            const int p = threadIdx.x % NP, k1 = threadIdx.x / NP;  // NT = 8 NP
            cplxf v[RZ];
#pragma unroll
            for (int i = 0; i < RZ; i++) v[i] = ldf(buf + p * S + RZ * k1 + i);
            tail_run<RZ / BZ, BZ, -1>(v, k1, twz);
            __syncthreads();
#pragma unroll
            for (int t = 0; t < RZ; t++) stf(buf + p * S + k1 + 8 * t, v[t]);
        }
        __syncthreads();
        each<H * (RY / 2)>([&](int b) {
            const int kz = b % H, a = b / H;
            cplxf e[8], o[8], *p = buf + a * S + kz, *q = buf + a * S + mirror(kz);
#pragma unroll
            for (int r = 0; r < 8; r++) {
                const cplxf ck = ldf(p + (RY / 2) * r * S), cm = ldf(q + (RY / 2) * r * S);
                if (kz) {
                    e[r] = {(ck.x + cm.x) * 0.5f, (ck.y - cm.y) * 0.5f};
                    o[r] = {(ck.y + cm.y) * 0.5f, (cm.x - ck.x) * 0.5f};
                } else {
                    e[r] = {ck.x, cm.x};
                    o[r] = {ck.y, cm.y};
                }
            }
            Dft<float, 8>::run(e, -1, nullptr, 0);
            Dft<float, 8>::run(o, -1, nullptr, 0);
#pragma unroll
            for (int r = 0; r < 8; r++) {
                stf(p + (RY / 2) * r * S, e[r]);
                stf(q + (RY / 2) * r * S, o[r]);
            }
        });
        __syncthreads();
        if (last) pdl_trigger();
        each<H * 8>([&](int b) {
            const int kz = b % H, k1 = b / H;
            cplxf v[RY], *p = buf + (RY / 2) * k1 * S + kz, *q = buf + (RY / 2) * k1 * S + mirror(kz);
#pragma unroll
            for (int j = 0; j < RY; j += 2) {
                v[j] = ldf(p + (j / 2) * S);
                v[j + 1] = ldf(q + (j / 2) * S);
            }
            tail_run<RY / BY, BY, -1>(v, k1, twy);
            if (kz) {
#pragma unroll
                for (int t = 0; t < RY; t++) stf(dst + (k1 + 8 * t) * MK2 + kz, v[t]);
            } else {
#pragma unroll
                for (int t = 0; t < RY; t++) stf(col + k1 + 8 * t, v[t]);
            }
        });
        __syncthreads();
        // the spectra of the kz = 0 and kz = H columns
        each<M1>([&](int k) {
            const cplxf c = ldf(col + k), cm = ldf(col + (k ? M1 - k : 0));
            stf(dst + k * MK2, {(c.x + cm.x) * 0.5f, (c.y - cm.y) * 0.5f});
            stf(dst + k * MK2 + H, {(c.y + cm.y) * 0.5f, (cm.x - c.x) * 0.5f});
        });
    }
};

__device__ __forceinline__ const float *real_etab(const PropsArgs<float> &a, int slot, int fld, int s)
{
    const Geo &g = a.g;
    if (g.jon && s == (fld == 0 ? g.jq : g.jqd)) return a.jtab + (size_t)slot * g.M;
    const int sel = fld == 0 ? (s < g.n1 ? 0 : 1) : (s < g.n2 ? 1 : 0);
    return a.etab + ((size_t)slot * 2 + sel) * g.M;
}

// mid: sp = 0 the half-step spectrum (inverse slab, times E2, forward slab), sp = 1
// the full-step one (inverse slab, P = E2 qs1)
template <int M1, int M2>
__global__ void __launch_bounds__(RealSlab<M1, M2>::NT, RealSlab<M1, M2>::MINB) k_real_mid(PropsArgs<float> a, int s)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    using R = RealSlab<M1, M2>;
    const R B(smem_raw);
    const Geo &g = a.g;
    const int x = blockIdx.x, fld = blockIdx.y & 1, sp = blockIdx.y >> 1, slot = blockIdx.z;
    const size_t off = (size_t)x * M1 * M2;
    cplxf *spec = a.spec + (((size_t)slot * 2 + fld) * 2 + sp) * g.Mk + (size_t)x * M1 * R::MK2;
    const float *E = real_etab(a, slot, fld, s) + off;
    float *P = a.pbuf + ((size_t)slot * 2 + fld) * g.M + off;
    // table value and P at offset i of the slab, is of a staged copy
    auto e_at = [&](int i, int is) { return R::STAGED ? B.Es[is] : __ldg(E + i); };
    if constexpr (R::STAGED) {
        if (threadIdx.x == 0) {
            mbar_init(&B.bars[0], 1);
            mbar_fence_init();
        }
        B.stage_in(B.Es, E, &B.bars[0]);  // settled: never the first kernel of a chain (pdl.cuh)
    } else {
        if (threadIdx.x == 0) prefetch_l2(E, M1 * M2 * sizeof(float));
    }
    B.load_tables(a.tw, g.m0);
    __syncthreads();
    pdl_wait();
    if (pdl_early(g.m0)) pdl_trigger();
    B.inverse_passes(spec);
    if constexpr (R::STAGED) mbar_wait(&B.bars[0], 0, a.err);
    if (sp == 0) {
        B.template real_space<true, true>([&](cplxf *v, int o, int os) {
#pragma unroll
            for (int t = 0; t < R::RZ; t++) {
                const float e0 = e_at(o + 8 * t, os + 8 * t), e1 = e_at(o + M2 + 8 * t, os + M2 + 8 * t);
                v[t].x = __fmul_rn(v[t].x, __fmul_rn(e0, e0));
                v[t].y = __fmul_rn(v[t].y, __fmul_rn(e1, e1));
            }
        });
        B.forward_passes(spec, true);
    } else {
        B.template real_space<true, false>([&](cplxf *v, int o, int os) {
#pragma unroll
            for (int t = 0; t < R::RZ; t++) {
                const float e0 = e_at(o + 8 * t, os + 8 * t), e1 = e_at(o + M2 + 8 * t, os + M2 + 8 * t);
                const float p0 = __fmul_rn(v[t].x, __fmul_rn(e0, e0)), p1 = __fmul_rn(v[t].y, __fmul_rn(e1, e1));
                (R::STAGED ? B.Es + os : P + o)[8 * t] = p0;
                (R::STAGED ? B.Es + os : P + o)[M2 + 8 * t] = p1;
            }
        });
        if constexpr (R::STAGED) {
            fence_proxy_async_smem();
            __syncthreads();
            B.stage_out(P, B.Es);
            B.stage_out_done();
        }
    }
}

// combine: finishes step s (mode 0: Richardson combination; mode 1: q(s+1) = 1;
// mode 2: q(s+1) from the propagator store) and starts step s + 1
template <int M1, int M2>
__global__ void __launch_bounds__(RealSlab<M1, M2>::NT, RealSlab<M1, M2>::MINB)
    k_real_combine(PropsArgs<float> a, int s, int mode)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    using R = RealSlab<M1, M2>;
    const R B(smem_raw);
    const Geo &g = a.g;
    const int x = blockIdx.x, fld = blockIdx.y, slot = blockIdx.z, sn = s + 1;
    const size_t off = (size_t)x * M1 * M2;
    cplxf *specA = a.spec + ((size_t)slot * 2 + fld) * 2 * g.Mk + (size_t)x * M1 * R::MK2, *specB = specA + g.Mk;
    float *qn = a.hist + (((size_t)slot * (g.Ns + 1) + sn) * 2 + fld) * (size_t)g.M + off;
    const bool next = sn < g.Ns;
    const float *En = real_etab(a, slot, fld, next ? sn : 0) + off;
    const float *E = mode == 0 ? real_etab(a, slot, fld, s) + off : En;
    const float *P = a.pbuf + ((size_t)slot * 2 + fld) * g.M + off;
    const bool same = E == En;  // the next step's table, unless the chain changes blocks here
    // table of step s, of step s + 1, P, and q' at offset i of the slab, is of a staged copy
    auto e_at = [&](int i, int is) { return R::STAGED ? B.Es[is] : __ldg(E + i); };
    auto en_at = [&](int i, int is) { return R::STAGED && same ? B.Es[is] : __ldg(En + i); };
    auto p_at = [&](int i, int is) { return R::STAGED ? B.Qs[is] : __ldcg(P + i); };
    auto q_at = [&](int i, int is) -> float & { return R::STAGED ? B.Qs[is] : qn[i]; };
    if constexpr (R::STAGED) {
        if (threadIdx.x == 0) {
            mbar_init(&B.bars[0], 1);
            mbar_init(&B.bars[1], 1);
            mbar_fence_init();
        }
        // settled unless this is the first kernel of a chain (pdl.cuh)
        if (mode == 0) B.stage_in(B.Es, E, &B.bars[0]);
    } else {
        if (threadIdx.x == 0) prefetch_l2(E, M1 * M2 * sizeof(float));
    }
    B.load_tables(a.tw, g.m0);
    __syncthreads();
    pdl_wait();
    if (pdl_early(g.m0)) pdl_trigger();
    if constexpr (R::STAGED) {
        if (mode != 0) B.stage_in(B.Es, E, &B.bars[0]);
        if (mode != 1) B.stage_in(B.Qs, mode == 0 ? P : qn, &B.bars[1]);
    } else {
        if (mode == 0 && threadIdx.x == 0) prefetch_l2(P, M1 * M2 * sizeof(float));
    }
    auto scale = [&](cplxf *v, int o, int os) {  // half step input E4' q'
#pragma unroll
        for (int t = 0; t < R::RZ; t++)
            v[t] = {__fmul_rn(v[t].x, en_at(o + 8 * t, os + 8 * t)), __fmul_rn(v[t].y, en_at(o + M2 + 8 * t, os + M2 + 8 * t))};
    };
    // Richardson, GPU_kernels.h:199-203
    auto finish = [&](cplxf *v, int o, int os) {
#pragma unroll
        for (int t = 0; t < R::RZ; t++) {
            const int i = o + 8 * t, is = os + 8 * t;
            const float q0 = (v[t].x * e_at(i, is) * 4.0f - p_at(i, is)) / 3.0f;
            const float q1 = (v[t].y * e_at(i + M2, is + M2) * 4.0f - p_at(i + M2, is + M2)) / 3.0f;
            q_at(i, is) = q0;
            q_at(i + M2, is + M2) = q1;
            v[t] = {q0, q1};
        }
    };
    if (mode == 0) {
        B.inverse_passes(specA);
        if constexpr (R::STAGED) {
            mbar_wait(&B.bars[0], 0, a.err);
            mbar_wait(&B.bars[1], 0, a.err);
        }
        if (next)
            B.template real_space<true, true>([&](cplxf *v, int o, int os) {
                finish(v, o, os);
                scale(v, o, os);
            });
        else
            B.template real_space<true, false>(finish);
    } else {
        if constexpr (R::STAGED) {
            mbar_wait(&B.bars[0], 0, a.err);
            if (mode == 2) mbar_wait(&B.bars[1], 0, a.err);
        }
        B.template real_space<false, true>([&](cplxf *v, int o, int os) {
#pragma unroll
            for (int t = 0; t < R::RZ; t++) {
                const int i = o + 8 * t, is = os + 8 * t;
                if (mode == 1) q_at(i, is) = q_at(i + M2, is + M2) = 1.0f;
                v[t] = mode == 1 ? cplxf{1.0f, 1.0f} : cplxf{q_at(i, is), q_at(i + M2, is + M2)};
            }
            scale(v, o, os);
        });
    }
    if constexpr (R::STAGED) {
        fence_proxy_async_smem();
        __syncthreads();
        if (mode != 2) B.stage_out(qn, B.Qs);
    }
    if (next) {
        B.forward_passes(specA, false);
        // full step input E2' q'
        __syncthreads();
        B.template real_space<false, true>([&](cplxf *v, int o, int os) {
#pragma unroll
            for (int t = 0; t < R::RZ; t++) {
                const int i = o + 8 * t, is = os + 8 * t;
                const float e0 = en_at(i, is), e1 = en_at(i + M2, is + M2);
                v[t] = {__fmul_rn(q_at(i, is), __fmul_rn(e0, e0)), __fmul_rn(q_at(i + M2, is + M2), __fmul_rn(e1, e1))};
            }
        });
        B.forward_passes(specB, true);
    }
    if constexpr (R::STAGED) B.stage_out_done();
}

// ---------------------------------------------------------------- x pass
// The inverse of tail_run for the x pass: slots t = a + RA b (frequency k1 + 8 t)
// back to points m = 0 .. RA RB - 1, in the stage order of fft_pair_fused (the
// radices reversed), then the factor of the radix-8 stage that follows.
template <int RA, int RB>
__device__ __forceinline__ void tail_back(cplxf *v, int k1, const cplxf *tw)
{
    constexpr int R = RA * RB;
    cplxf o[R];
#pragma unroll
    for (int a = 0; a < RA; a++) {
        cplxf u[RB];
#pragma unroll
        for (int b = 0; b < RB; b++) u[b] = v[a + RA * b];
        if constexpr (RB > 1) Dft<float, RB>::run(u, 1, nullptr, 0);
#pragma unroll
        for (int b = 0; b < RB; b++) o[RA * b + a] = (RB > 1 && a > 0) ? twiddle<1>(u[b], ldf(tw + 8 * a * b)) : u[b];
    }
#pragma unroll
    for (int b = 0; b < RB; b++) {
        Dft<float, RA>::run(o + RA * b, 1, nullptr, 0);
#pragma unroll
        for (int r = 0; r < RA; r++) {
            const int m = b + RB * r;
            v[m] = m > 0 ? twiddle<1>(o[RA * b + r], ldf(tw + k1 * m)) : o[RA * b + r];
        }
    }
}

template <int M0, int TC>
struct RealPencil {
    static constexpr int SMEM = (M0 * TC + M0) * (int)sizeof(cplxf) + (M0 + TC) * (int)sizeof(float);
};
constexpr int kRealPencilThreads = 256;

// One tile of TC columns of one spectrum: forward x transform, diffusion factor
// (Mult_self, GPU_kernels.h:175-181), inverse transform, with one trip through
// shared memory on each side of the factor.  sp 0: times K2, 1: times K1.
template <int M0, int TC>
__global__ void __launch_bounds__(kRealPencilThreads, 4) k_real_pencil(PropsArgs<float> a)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    constexpr int R2 = M0 / 8, RB = tail_b(R2), RA = R2 / RB, NT = kRealPencilThreads;
    const Geo &g = a.g;
    // opposite order of the slab kernels before and after: what they touched last is still in L2
    const int tile = gridDim.x - 1 - blockIdx.x, slot = gridDim.z - 1 - blockIdx.z;
    const int fld = blockIdx.y & 1, sp = blockIdx.y >> 1;
    const int ncol = g.m1 * g.mk2, c0 = tile * TC;
    cplxf *buf = reinterpret_cast<cplxf *>(smem_raw), *tw = buf + M0 * TC;
    float *gx = reinterpret_cast<float *>(tw + M0), *colf = gx + M0;
    cplxf *spec = a.spec + (((size_t)slot * 2 + fld) * 2 + sp) * g.Mk + c0;
    const float *kf = a.kfac + (size_t)__ldg(a.slot_rep + slot) * a.kf_stride;  // the replica's box
    for (int i = threadIdx.x; i < M0; i += NT) {
        stf(tw + i, ldf(a.tw + i));
        gx[i] = __ldg(kf + i);
    }
    for (int t = threadIdx.x; t < TC; t += NT) {
        const int c = c0 + t, y = c / g.mk2, kz = c - y * g.mk2;
        colf[t] = c < ncol ? __ldg(kf + M0 + y) * __ldg(kf + M0 + g.m1 + kz) : 0.0f;
    }
    pdl_wait();
    if (pdl_early(g.m0)) pdl_trigger();
#pragma unroll 1
    for (int b = threadIdx.x; b < R2 * TC; b += NT) {
        const int t = b % TC, j = b / TC;
        if (c0 + t < ncol) {
            cplxf v[8];
#pragma unroll
            for (int r = 0; r < 8; r++) v[r] = ldf_cg(spec + (size_t)(j + R2 * r) * ncol + t);
            Dft<float, 8>::run(v, -1, nullptr, 0);
#pragma unroll
            for (int r = 0; r < 8; r++) stf(buf + (j + R2 * r) * TC + t, v[r]);
        }
    }
    __syncthreads();
    const float invM = a.invM, Mreal = a.Mreal;
#pragma unroll 1
    for (int b = threadIdx.x; b < 8 * TC; b += NT) {
        const int t = b % TC, k1 = b / TC;
        if (c0 + t < ncol) {
            cplxf v[R2], *p = buf + R2 * k1 * TC + t;
#pragma unroll
            for (int i = 0; i < R2; i++) v[i] = ldf(p + i * TC);
            tail_run<RA, RB, -1>(v, k1, tw);
            // K2 = g/M, K1 = g^2/M  (Prepare_dev_expKsq2_expKsq, GPU_kernels.h:207-213);
            // the product may fuse with the additions that follow, as it does in
            // fft_pair_fused
            const float ct = colf[t];
#pragma unroll
            for (int i = 0; i < R2; i++) {
                const float k2 = gx[k1 + 8 * i] * ct;
                const float f = sp == 0 ? k2 * invM : (k2 * invM) * (k2 * invM) * Mreal;
                v[i].x *= f;
                v[i].y *= f;
            }
            tail_back<RA, RB>(v, k1, tw);
#pragma unroll
            for (int i = 0; i < R2; i++) stf(p + i * TC, v[i]);
        }
    }
    __syncthreads();
    pdl_trigger();
#pragma unroll 1
    for (int b = threadIdx.x; b < R2 * TC; b += NT) {
        const int t = b % TC, m = b / TC;
        if (c0 + t < ncol) {
            cplxf v[8];
#pragma unroll
            for (int r = 0; r < 8; r++) v[r] = ldf(buf + (m + R2 * r) * TC + t);
            Dft<float, 8>::run(v, 1, nullptr, 0);
#pragma unroll
            for (int r = 0; r < 8; r++) stf(spec + (size_t)(m + R2 * r) * ncol + t, v[r]);
        }
    }
}

}  // namespace scft
