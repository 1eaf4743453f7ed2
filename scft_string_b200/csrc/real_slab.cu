// real_slab.cu -- launches of the FP32 slab kernels (real_slab.cuh).
#include "real_slab.cuh"
#include "schedule.h"

namespace scft {

#define REAL_SLABS(X) X(32, 32) X(48, 48) X(64, 64) X(64, 96) X(96, 96) X(128, 128)

bool real_slab_has(int m1, int m2)
{
#define X(A, B) \
    if (m1 == A && m2 == B) return true;
    REAL_SLABS(X)
#undef X
    return false;
}

int real_slab_setup(int m1, int m2)
{
    cudaError_t e = cudaSuccess;
#define X(A, B)                                                                               \
    if (m1 == A && m2 == B) {                                                                 \
        e = raise_dyn_smem(k_real_mid<A, B>, RealSlab<A, B>::SMEM_MID);                          \
        if (e == cudaSuccess) e = raise_dyn_smem(k_real_combine<A, B>, RealSlab<A, B>::SMEM); \
    }
    REAL_SLABS(X)
#undef X
    return e == cudaSuccess ? 0 : -1;
}

void real_mid(const PropsArgs<float> &a, int nslots, int s, cudaStream_t st)
{
    const Geo &g = a.g;
#define X(A, B)                                                                                                   \
    if (g.m1 == A && g.m2 == B)                                                                                   \
        launch_step(k_real_mid<A, B>, dim3(g.m0, 4, nslots), RealSlab<A, B>::NT, RealSlab<A, B>::SMEM_MID, 1, 1, st, a, s);
    REAL_SLABS(X)
#undef X
}

void real_combine(const PropsArgs<float> &a, int nslots, int s, int mode, cudaStream_t st)
{
    const Geo &g = a.g;
#define X(A, B)                                                                                                  \
    if (g.m1 == A && g.m2 == B)                                                                                  \
        launch_step(k_real_combine<A, B>, dim3(g.m0, 2, nslots), RealSlab<A, B>::NT, RealSlab<A, B>::SMEM, 1, 1, \
                    st, a, s, mode);
    REAL_SLABS(X)
#undef X
}

#define REAL_AXES(X) X(32) X(48) X(64) X(96) X(128)
constexpr int kRealTile = 32;

int real_pencil_setup(int m0)
{
    cudaError_t e = cudaSuccess;
#define X(A)                                                                                            \
    if (m0 == A) {                                                                                      \
        e = raise_dyn_smem(k_real_pencil<A, kRealTile>, RealPencil<A, kRealTile>::SMEM);                \
        if (e == cudaSuccess)                                                                           \
            e = raise_dyn_smem(k_real_pencil<A, 2 * kRealTile>, RealPencil<A, 2 * kRealTile>::SMEM);    \
    }
    REAL_AXES(X)
#undef X
    return e == cudaSuccess ? 0 : -1;
}

int real_pencil_wide(int wide, int m0, int ncol, int both, int nslots)
{
    return wide_tiles(wide, m0, ncol, kRealTile, both ? 4 : 2, nslots);
}

void real_pencil(const PropsArgs<float> &a, int nslots, int both, int wide, cudaStream_t st)
{
    const Geo &g = a.g;
    const int ncol = g.m1 * g.mk2;
    wide = real_pencil_wide(wide, g.m0, ncol, both, nslots);
    const int tc = wide ? 2 * kRealTile : kRealTile;
    const dim3 grid((ncol + tc - 1) / tc, both ? 4 : 2, nslots);
#define X(A)                                                                                                        \
    if (g.m0 == A) {                                                                                                \
        if (wide)                                                                                                   \
            launch_step(k_real_pencil<A, 2 * kRealTile>, grid, kRealPencilThreads, RealPencil<A, 2 * kRealTile>::SMEM, \
                        1, 1, st, a);                                                                               \
        else                                                                                                        \
            launch_step(k_real_pencil<A, kRealTile>, grid, kRealPencilThreads, RealPencil<A, kRealTile>::SMEM, 1, 1, \
                        st, a);                                                                                     \
    }
    REAL_AXES(X)
#undef X
}

}  // namespace scft
