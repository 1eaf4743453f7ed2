// pair_any.cu -- the kernels of pair.cuh for slab shapes and x lengths without
// compile-time sizes; a module of their own, so that the others load without them.
#include "pair.cuh"
#include "pair_shapes.h"

namespace scft {
namespace {

using T = double;

constexpr int kTile = kPairTile;
constexpr int kPencilThreads = 256;

template <int RA>
__global__ void __launch_bounds__(512, 1) k_pair_mid_any(PropsArgs<T> a, int s, PairAny q)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    pair_mid_body(PairSlabAny<RA>(smem_raw, q), a, s, blockIdx.x, blockIdx.y, blockIdx.z);
}

template <int RA>
__global__ void __launch_bounds__(512, 1) k_pair_combine_any(PropsArgs<T> a, int s, int mode, PairAny q)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    pair_combine_body(PairSlabAny<RA>(smem_raw, q), a, s, mode, blockIdx.x, gridDim.y == 1 ? -1 : (int)blockIdx.y,
                      blockIdx.z);
}

template <int R2>
__global__ void __launch_bounds__(kPencilThreads, 2) k_pair_pencil_any(PropsArgs<T> a, int s, int nsum, int ra, int rb)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int tile = gridDim.x - 1 - blockIdx.x, slot = gridDim.z - 1 - blockIdx.z;
    if (tile * kTile >= a.g.m1 * a.g.m2) {  // a tile past the last: the exponents of step s + 1
        pdl_wait();
        pdl_trigger();
        pair_next_exponents(a, slot, s, nsum);
        return;
    }
    pair_pencil_any_body<R2, kTile>(a, tile, blockIdx.y, slot, ra, rb, smem_raw);
}

}  // namespace

int pair_any_setup(int m0, int m1, int m2)
{
    cudaError_t e = cudaSuccess;
    auto up = [&](auto *fn, int bytes) {
        if (e == cudaSuccess) e = raise_dyn_smem(fn, bytes);
    };
    PairAny q;
    int r1, r2;
    if (!pair_slab_fixed(m1, m2) && pair_any_plan(m1, m2, q)) switch (q.ra) {
#define X(A)                                           \
    case A:                                            \
        up(k_pair_mid_any<A>, pair_any_smem(q));            \
        up(k_pair_combine_any<A>, pair_any_smem(q));        \
        break;
            PAIR_RADICES(X)
#undef X
        }
    if (!pair_axis_fixed(m0) && pair_x_radices(m0, r1, r2)) switch (r2) {
#define X(A) \
    case A: up(k_pair_pencil_any<A>, pair_any_pencil_smem(m0)); break;
            PAIR_RADICES(X)
#undef X
        }
    return e == cudaSuccess ? 0 : -1;
}

void pair_any_mid(const PropsArgs<T> &a, int nslots, int s, cudaStream_t st)
{
    const Geo &g = a.g;
    PairAny q;
    if (pair_any_plan(g.m1, g.m2, q)) switch (q.ra) {
#define X(A)                                                                                                           \
    case A: launch_step(k_pair_mid_any<A>, dim3(g.m0, 2, nslots), pair_any_threads(q, 2 * g.m0 * nslots), pair_any_smem(q), 1, 1, st, a, s, q); break;
            PAIR_RADICES(X)
#undef X
        }
}

void pair_any_combine(const PropsArgs<T> &a, int nslots, int s, int mode, int split, cudaStream_t st)
{
    const Geo &g = a.g;
    PairAny q;
    if (pair_any_plan(g.m1, g.m2, q)) switch (q.ra) {
#define X(A)                                                                                                         \
    case A:                                                                                                          \
        launch_step(k_pair_combine_any<A>, dim3(g.m0, split, nslots), pair_any_threads(q, split * g.m0 * nslots), pair_any_smem(q), 1, split, st, a, \
                    s, mode, q);                                                                                     \
        break;
            PAIR_RADICES(X)
#undef X
        }
}

void pair_any_pencil(const PropsArgs<T> &a, int nslots, int s, int both, int nsum, int ra, int rb, cudaStream_t st)
{
    const Geo &g = a.g;
    int r1, r2;
    if (pair_x_radices(g.m0, r1, r2)) {
        const dim3 grid((g.m1 * g.m2 + kTile - 1) / kTile + !both, both ? 2 : 1, nslots);
        switch (r2) {
#define X(A) \
    case A: launch_step(k_pair_pencil_any<A>, grid, kPencilThreads, pair_any_pencil_smem(g.m0), 1, 1, st, a, s, nsum, ra, rb); break;
            PAIR_RADICES(X)
#undef X
        }
    }
}

}  // namespace scft
