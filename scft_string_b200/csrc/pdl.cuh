// pdl.cuh -- overlap of the launches of a contour step: programmatic dependent
// launch, L2 prefetch, and the launch call that both take.
#pragma once
#include <cuda_runtime.h>

namespace scft {

// Programmatic dependent launch: the kernels of a step let the next one start
// as their last CTAs run (its CTAs set up and read constant tables), and wait
// here for the whole previous kernel before they touch what it wrote.  Both are
// no-ops in a kernel launched without the attribute.
//
// What a kernel may read before its wait: only what was complete when the kernel
// before it passed its own, for that kernel's trigger comes after its wait.  A chain
// is k_prepare, the first combine (modes 1 and 2), then pencil, mid, pencil, combine
// (mode 0) per step.  So every kernel may read the twiddle and diffusion factors and
// the replica list, which copies ahead of k_prepare wrote; the E tables, which
// k_prepare writes, may be read early by all but the first combine: k_prepare has no
// trigger, and its blocks may be gone before its stores are visible.  Where a chain
// starts again from a checkpoint, the kernel before the first combine is a copy, and
// the same rule is kept.  L2 prefetches are hints and may come at any time.
__device__ __forceinline__ void pdl_trigger()
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void pdl_wait()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Where a kernel lets the next one start.  As soon as its own wait is over, in
// small launches: the next kernel's CTAs then find SMs of their own and are set up
// in time (one replica step: 48^3 21.9 -> 19.7 us, 16x12x20 16.0 -> 14.6).  Before
// its last pass in larger ones, where early CTAs crowd the SMs that are done first
// (64^3 31.4 us late, 37.1 early; 16 replicas the same).
__device__ __forceinline__ bool pdl_early(int m0) { return 2 * m0 * gridDim.z <= 96; }

// asks for `bytes` at p to be brought into L2; a hint, no wait.  The copy engine
// wants 16-byte multiples; slabs of an odd number of doubles go without.
__device__ __forceinline__ void prefetch_l2(const void *p, int bytes)
{
    if (((unsigned)(size_t)p | (unsigned)bytes) & 15u) return;
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// the two CTAs of a split combine: each has read its input slab (arrive) before
// either overwrites it (wait)
__device__ __forceinline__ void pair_arrive()
{
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void pair_wait()
{
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Launch in clusters of (cx, cy) CTAs.  pdl: it may start while the kernel before
// it on the stream finishes; only for kernels that call pdl_wait.
template <class... Params, class... Args>
inline void launch_ex(bool pdl, void (*fn)(Params...), dim3 grid, int threads, int smem, int cx, int cy, cudaStream_t st,
                      const Args &...args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = pdl ? 1 : 0;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = cx;
    at[1].val.clusterDim.y = cy;
    at[1].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = cx * cy > 1 ? 2 : 1;
    cudaLaunchKernelEx(&cfg, fn, Params(args)...);
}

template <class... Params, class... Args>
inline void launch_step(void (*fn)(Params...), dim3 grid, int threads, int smem, int cx, int cy, cudaStream_t st,
                        const Args &...args)
{
    launch_ex(true, fn, grid, threads, smem, cx, cy, st, args...);
}

}  // namespace scft
