// pair.cu -- kernels and launchers of the FP64 contour step on q + i q^dagger
// (pair.cuh).
//
// FP32 keeps the real transforms of props_kernels.cu: in single precision the
// densities follow the rounding of the transforms, and these kernels moved them
// by up to 5e-5 (2-norm) and their error against FP64 by up to twice.
#include <algorithm>

#include "pair.cuh"
#include "pair_shapes.h"
#include "step_order.cuh"

namespace scft {
namespace {

using T = double;

constexpr int kSms = 148;
constexpr int kTile = kPairTile;  // the wide form takes twice as many columns
constexpr int kPencilThreads = 256;

// grids with a persistent step kernel
#define PAIR_GRIDS(X) X(32, 32, 32) X(48, 48, 48) X(64, 64, 64) X(64, 64, 96) X(96, 96, 96)

constexpr int pencil_minb(int m0) { return m0 > 80 ? 2 : 3; }

template <int M1, int M2, int CL>
__global__ void __launch_bounds__(PairSlab<M1, M2, CL>::NT, PairSlab<M1, M2, CL>::MINB) k_pair_mid(PropsArgs<T> a, int s)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    pair_mid_body(PairSlab<M1, M2, CL>(smem_raw), a, s, blockIdx.x / CL, blockIdx.y, blockIdx.z);
}

template <int M1, int M2, int CL>
__global__ void __launch_bounds__(PairSlab<M1, M2, CL>::NT, PairSlab<M1, M2, CL>::MINB)
    k_pair_combine(PropsArgs<T> a, int s, int mode)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    pair_combine_body(PairSlab<M1, M2, CL>(smem_raw), a, s, mode, blockIdx.x / CL,
                      gridDim.y == 1 ? -1 : (int)blockIdx.y, blockIdx.z);
}

template <int M0, int TC>
__global__ void __launch_bounds__(kPencilThreads, pencil_minb(M0)) k_pair_pencil(PropsArgs<T> a, int s, int nsum, int ra, int rb)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    // slots (and tiles) in the opposite order of the slab kernels before and
    // after: what those touched last is still in L2
    const int tile = gridDim.x - 1 - blockIdx.x, slot = gridDim.z - 1 - blockIdx.z;
    if (tile * TC >= a.g.m1 * a.g.m2) {  // a tile past the last: the exponents of step s + 1
        pdl_wait();
        pdl_trigger();
        pair_next_exponents(a, slot, s, nsum);
        return;
    }
    pair_pencil_body<M0, TC, kPencilThreads>(a, tile, blockIdx.y, slot, ra, rb, smem_raw);
}

__device__ __forceinline__ int ld_acquire_gpu(const int *p)
{
    int v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

constexpr uint32_t kStepSpin = 1u << 22;

// The four launches of a step as work items of one launch: both spectra's x
// tiles, the slabs of mid (two per x), the half-step spectrum's x tiles and the
// exponents of the next step, the slabs of combine, each phase ordered by slot.  CTAs claim items from a
// counter in the order of step_order.cuh, and an item waits only for the
// previous phase of its own slot.  Items are claimed in order by running CTAs,
// so whatever an item waits for is held by a CTA that is running or done; no
// residency is assumed.  Every wait is bounded and records error 3 when it
// gives up, which ends the kernel.
template <int M0, int M1, int M2, int TC>
__global__ void __launch_bounds__(PairSlab<M1, M2, 1>::NT, PairSlab<M1, M2, 1>::MINB)
    k_pair_step(PropsArgs<T> a, int s, int nslots)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ int item_sh[3], ok_sh;
    using PS = PairSlab<M1, M2, 1>;
    constexpr int NT = PS::NT, ntiles = (M1 * M2 + TC - 1) / TC;
    int ra, rb;
    PS::radices(ra, rb);
    const int per[4] = {2 * ntiles, 2 * M0, ntiles + 1, M0};
    int *claim = a.sync + s;      // this step's claim counter
    int *done = a.sync + a.g.Ns;  // [phase][slot] completion counters, cumulative over the steps
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) {
            int ph = -1, gr = 0, un = 0;
            if (!step_item(atomicAdd(claim, 1), nslots, per, ph, gr, un)) ph = -1;
            item_sh[0] = ph;
            item_sh[1] = gr;
            item_sh[2] = un;
            ok_sh = 1;
            if (ph > 0) {
                const int need = per[ph - 1] * (s + 1);
                const int *cnt = done + (ph - 1) * nslots + gr;
                uint32_t i = 0;
                while (ld_acquire_gpu(cnt) < need && i < kStepSpin) {
                    __nanosleep(32);
                    i++;
                }
                if (i >= kStepSpin) {
                    ok_sh = 0;
                    *a.err = 3;
                }
            }
        }
        __syncthreads();
        const int phase = item_sh[0], slot = item_sh[1], unit = item_sh[2];
        if (phase < 0 || !ok_sh) break;
        if (phase == 0)
            pair_pencil_body<M0, TC, NT>(a, unit % ntiles, unit / ntiles, slot, ra, rb, smem_raw);
        else if (phase == 1)
            pair_mid_body(PS(smem_raw), a, s, unit >> 1, unit & 1, slot);
        else if (phase == 2 && unit == ntiles)
            pair_next_exponents(a, slot, s, M0);
        else if (phase == 2)
            pair_pencil_body<M0, TC, NT>(a, unit, 0, slot, ra, rb, smem_raw);
        else
            pair_combine_body(PS(smem_raw), a, s, 0, unit, -1, slot);
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            atomicAdd(done + phase * nslots + slot, 1);
        }
    }
}

template <int M0, int M1, int M2, int TC>
constexpr int step_smem()
{
    return PairSlab<M1, M2, 1>::SMEM > PairPencil<M0, TC>::SMEM ? PairSlab<M1, M2, 1>::SMEM
                                                                   : PairPencil<M0, TC>::SMEM;
}

}  // namespace

bool pair_applicable(int m0, int m1, int m2)
{
    PairAny q;
    int r1, r2;
    return (pair_slab_fixed(m1, m2) || pair_any_plan(m1, m2, q)) && (pair_axis_fixed(m0) || pair_x_radices(m0, r1, r2));
}

bool pair_axis_wide(int m0) { return pair_axis_fixed(m0); }

// raises the kernels' shared-memory limits; *grid = CTAs of the persistent step launch (0: none)
int pair_setup(int m0, int m1, int m2, int *grid)
{
    cudaError_t e = cudaSuccess;
    auto up = [&](auto *fn, int bytes) {
        if (e == cudaSuccess) e = raise_dyn_smem(fn, bytes);
    };
#define X(A, B)                                                     \
    if (m1 == A && m2 == B) {                                       \
        constexpr int CL = kCl<A, B>;                               \
        up(k_pair_mid<A, B, CL>, PairSlab<A, B, CL>::SMEM);         \
        up(k_pair_combine<A, B, CL>, PairSlab<A, B, CL>::SMEM);     \
    }
    PAIR_SLABS(X)
#undef X
#define X(A)                                                               \
    if (m0 == A) {                                                         \
        up(k_pair_pencil<A, kTile>, PairPencil<A, kTile>::SMEM);         \
        up(k_pair_pencil<A, 2 * kTile>, PairPencil<A, 2 * kTile>::SMEM); \
    }
    PAIR_AXES(X)
#undef X
    if (e == cudaSuccess && pair_any_setup(m0, m1, m2) != 0) return -1;
    *grid = 0;
#define X(A, B, C)                                                                                             \
    if (m0 == A && m1 == B && m2 == C) {                                                                       \
        if constexpr (kCl<B, C> == 1) {                                                                       \
            up(k_pair_step<A, B, C, kTile>, step_smem<A, B, C, kTile>());                                       \
            up(k_pair_step<A, B, C, 2 * kTile>, step_smem<A, B, C, 2 * kTile>());                               \
            int per_sm = 0;                                                                                    \
            if (e == cudaSuccess &&                                                                            \
                cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_pair_step<A, B, C, 2 * kTile>,         \
                                                              PairSlab<B, C, 1>::NT,                           \
                                                              step_smem<A, B, C, 2 * kTile>()) == cudaSuccess)  \
                *grid = per_sm * kSms;                                                                         \
        }                                                                                                      \
    }
    PAIR_GRIDS(X)
#undef X
    return e == cudaSuccess ? 0 : -1;
}

void pair_mid(const PropsArgs<T> &a, int nslots, int s, cudaStream_t st)
{
    const Geo &g = a.g;
#define X(A, B)                                                                                                      \
    if (g.m1 == A && g.m2 == B) {                                                                                    \
        constexpr int CL = kCl<A, B>;                                                                                \
        using P = PairSlab<A, B, CL>;                                                                                \
        launch_step(k_pair_mid<A, B, CL>, dim3(CL * g.m0, 2, nslots), P::NT, P::SMEM, CL, 1, st, a, s);               \
        return;                                                                                                      \
    }
    PAIR_SLABS(X)
#undef X
    pair_any_mid(a, nslots, s, st);
}

void pair_combine(const PropsArgs<T> &a, int nslots, int s, int mode, cudaStream_t st)
{
    const Geo &g = a.g;
    // two CTAs per slab while both find an SM of their own: the chain of a CTA
    // is then two slab transforms instead of three
    const int split = 2 * g.m0 * nslots <= kSms && s + 1 < g.Ns ? 2 : 1;
#define X(A, B)                                                                                                      \
    if (g.m1 == A && g.m2 == B) {                                                                                    \
        constexpr int CL = kCl<A, B>;                                                                                \
        const int half = CL > 1 ? 1 : split;                                                                         \
        using P = PairSlab<A, B, CL>;                                                                                \
        launch_step(k_pair_combine<A, B, CL>, dim3(CL * g.m0, half, nslots), P::NT, P::SMEM, CL, half, st, a, s, mode); \
        return;                                                                                                      \
    }
    PAIR_SLABS(X)
#undef X
    pair_any_combine(a, nslots, s, mode, split, st);
}

void pair_pencil(const PropsArgs<T> &a, int nslots, int s, int both, int wide, cudaStream_t st)
{
    const Geo &g = a.g;
    wide = wide > 0;  // the narrow tile where nothing is said
    const int tc = wide ? 2 * kTile : kTile;
    int ra = 1, rb = 1;
    pair_y_radices(g.m1, g.m2, ra, rb);
    const int nsum = pair_slab_ctas(g.m1, g.m2) * g.m0;  // partial sums of mid
    if (!pair_axis_fixed(g.m0)) {
        pair_any_pencil(a, nslots, s, both, nsum, ra, rb, st);
        return;
    }
    const dim3 grid((g.m1 * g.m2 + tc - 1) / tc + !both, both ? 2 : 1, nslots);
#define X(A)                                                                                                 \
    if (g.m0 == A) {                                                                                         \
        if (wide)                                                                                            \
            launch_step(k_pair_pencil<A, 2 * kTile>, grid, kPencilThreads, PairPencil<A, 2 * kTile>::SMEM, 1, 1, st, a, s, nsum, ra, rb);  \
        else                                                                                                 \
            launch_step(k_pair_pencil<A, kTile>, grid, kPencilThreads, PairPencil<A, kTile>::SMEM, 1, 1, st, a, s, nsum, ra, rb);          \
        return;                                                                                              \
    }
    PAIR_AXES(X)
#undef X
}

void pair_step(const PropsArgs<T> &a, int nslots, int s, int wide, int grid, cudaStream_t st)
{
    const Geo &g = a.g;
#define X(A, B, C)                                                                                                   \
    if (g.m0 == A && g.m1 == B && g.m2 == C) {                                                                       \
        if constexpr (kCl<B, C> == 1) {                                                                             \
            constexpr int NT = PairSlab<B, C, 1>::NT;                                                                \
            if (wide > 0)                                                                                            \
                k_pair_step<A, B, C, 2 * kTile><<<grid, NT, step_smem<A, B, C, 2 * kTile>(), st>>>(a, s, nslots);     \
            else                                                                                                     \
                k_pair_step<A, B, C, kTile><<<grid, NT, step_smem<A, B, C, kTile>(), st>>>(a, s, nslots);             \
        }                                                                                                            \
        return;                                                                                                      \
    }
    PAIR_GRIDS(X)
#undef X
}

}  // namespace scft
