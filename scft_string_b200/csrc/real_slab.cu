// real_slab.cu -- launches of the FP32 slab kernels (real_slab.cuh).
#include "real_slab.cuh"

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

}  // namespace scft
