// common.cuh -- shared types of the sm_100a SCFT kernels.
//
// Layouts (same as the reference, scft.cu:462-464 and density.h:90):
//   real grid      r = z + m2*(y + m1*x)
//   half spectrum  k = kz + mk2*(ky + m1*kx),  mk2 = m2/2 + 1
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>

namespace scft {

template <typename T>
struct cplx {
    T x, y;
};

template <typename T>
__device__ __forceinline__ cplx<T> cmul(cplx<T> a, cplx<T> b)
{
    return {a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x};
}
// a * conj(b)
template <typename T>
__device__ __forceinline__ cplx<T> cmulc(cplx<T> a, cplx<T> b)
{
    return {a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y};
}
template <typename T>
__device__ __forceinline__ cplx<T> cadd(cplx<T> a, cplx<T> b)
{
    return {a.x + b.x, a.y + b.y};
}
template <typename T>
__device__ __forceinline__ cplx<T> csub(cplx<T> a, cplx<T> b)
{
    return {a.x - b.x, a.y - b.y};
}

constexpr int kMaxStages = 12;
constexpr int kPairLanes = 8;  // slab pack/unpack: mk2 <= 32*kPairLanes

// Quotients by a run-time divisor n: b / n = umulhi(b, mag), mag = floor(2^32/n)
// + 1 (0 for n = 1), exact while b n < 2^32.  A 32-bit division is about 20
// instructions; the run-time shaped transforms take several per butterfly.
__host__ __device__ __forceinline__ unsigned div_mag(int n) { return n > 1 ? 0xffffffffu / (unsigned)n + 1u : 0u; }
__host__ __device__ __forceinline__ int div_by(int b, unsigned mag)
{
#ifdef __CUDA_ARCH__
    return mag ? (int)__umulhi((unsigned)b, mag) : b;
#else
    return mag ? (int)(((unsigned long long)(unsigned)b * mag) >> 32) : b;
#endif
}

// Compensated sum (W. Kahan, Commun. ACM 8, 1965): the value is sum - c.
__host__ __device__ __forceinline__ void kahan_add(double &sum, double &c, double term)
{
    const double y = term - c;
    const double t = sum + y;
    c = (t - sum) - y;
    sum = t;
}

// (sum, c) + (sum2, c2), either of which may be the larger: the rounding of the two sums
// by D. E. Knuth's exact addition goes into the compensation
__host__ __device__ __forceinline__ void kahan_join(double &sum, double &c, double sum2, double c2)
{
    const double t = sum + sum2, b = t - sum;
    c = (c + c2) - ((sum - (t - b)) + (sum2 - b));
    sum = t;
}

// Mixed-radix factorisation of one FFT length (radices 2, 3, 4, 5, 7, 8).
struct Plan1D {
    int n;
    int nst;
    int radix[kMaxStages];
    unsigned mag_nr[kMaxStages], mag_ns[kMaxStages];  // div_mag of n / radix and of the accumulated size, per stage
    int tw_step[kMaxStages];                          // twiddle table stride of the stage
};

inline void plan_mags(Plan1D &p)
{
    int ns = 1;
    for (int s = 0; s < p.nst; s++) {
        p.mag_nr[s] = div_mag(p.n / p.radix[s]);
        p.mag_ns[s] = div_mag(ns);
        ns *= p.radix[s];
        p.tw_step[s] = p.n / ns;
    }
}

// Everything a propagator kernel needs to know about the grid.
struct Geo {
    int m0, m1, m2, mk2;
    int M, Mk;
    int npair;       // ceil(m1/2): packed real y-line pairs per x-slab
    int slab_c;      // complex elements of one slab buffer (m1*mk2 + slack)
    Plan1D px, py, pz;
    int Ns, n1, n2, Nh;
    int ncol_tiles;  // x-pencil tiles per field
    int tc;          // columns per x-pencil tile
    // continuous A fraction (off when jon == 0): q's step jq and q^dagger's
    // step jqd see the junction field theta wA + (1 - theta) wB (E table 2)
    int jon, jq, jqd;
    double theta;
};

// Raises a kernel's dynamic shared-memory limit to at least `bytes`, never
// lowers it.  The limit belongs to the kernel, not to a context: the
// runtime-shaped kernels serve every context of any grid, so a context that
// set it to its own (smaller) need would make the launches of an earlier,
// larger context fail.  Serialised, so concurrent context creation keeps
// the largest value.
template <typename F>
inline cudaError_t raise_dyn_smem(F *fn, int bytes)
{
    static std::mutex mu;
    std::lock_guard<std::mutex> lock(mu);
    cudaFuncAttributes at;
    cudaError_t e = cudaFuncGetAttributes(&at, reinterpret_cast<const void *>(fn));
    if (e != cudaSuccess) return e;
    if (at.maxDynamicSharedSizeBytes >= bytes) return cudaSuccess;
    return cudaFuncSetAttribute(reinterpret_cast<const void *>(fn), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                bytes);
}

}  // namespace scft
