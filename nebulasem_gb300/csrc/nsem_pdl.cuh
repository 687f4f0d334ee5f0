/*
 * Programmatic dependent launch: a kernel of a chain may start while the
 * kernel before it in the stream still runs, and waits for it inside.  What
 * comes before the wait overlaps the predecessor's tail: the launch itself,
 * index arithmetic and loads of data that no kernel of the chain writes (mesh,
 * metric, background, tables).
 *
 * Rules for a kernel launched with nsem_launch_chained:
 *   - every CTA calls nsem_chain_wait() before its first access to anything an
 *     earlier kernel wrote or still reads (its own stores included); the wait
 *     returns when the kernel before it has completed, which had itself waited
 *     for the one before;
 *   - nsem_chain_begin() lets the next kernel's CTAs start once every CTA of
 *     this one has called it or ended: once a CTA, where its last long phase
 *     begins;
 *   - data that earlier kernels wrote is read by plain loads: the read-only
 *     path (__ldg) assumes that nothing writes during the kernel's lifetime,
 *     which here begins before the predecessor ends.
 * A kernel that calls neither function may precede or follow such a kernel:
 * the wait then covers its whole run.
 */
#ifndef NSEM_PDL_CUH
#define NSEM_PDL_CUH

#include <cuda_runtime.h>

__device__ __forceinline__ void nsem_chain_begin() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void nsem_chain_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <typename... P, typename... A>
inline int nsem_launch_chained(void (*kernel)(P...), unsigned grid, dim3 block, size_t smem,
                               cudaStream_t st, A... args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(grid);
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = st;
    c.attrs = &at;
    c.numAttrs = 1;
    return (int)cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
}

#endif
