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

/* The split of an SM's storage into L1 and shared memory is the driver's
 * choice per kernel, and an SM changes it only when it is empty: between
 * kernels of different splits the next one's CTAs wait for the last of this
 * one.  A chain's launches therefore name one split, the shared memory in
 * percent of the most there can be (0: the driver's choice).  FP64 form and
 * its adjoint, 150 elements of order 4: 1030 to 665 us for 5 steps, 1888 to
 * 1513; 576 of order 3: 885 to 702; convection of 336 elements of order 3, 15
 * steps: 355 to 248.  44, 58, 82 and 100 are each 3 to 6 % slower than 72
 * at some size. */
constexpr int NSEM_SPLIT = 72;

/* Grids of more than one wave keep the driver's choice: their own kernels
 * fill the SMs, and the best split of each counts for more (2184 elements of
 * order 3: 1323 us and 1358 with one split, of order 4 2151 and 2195).  The
 * convection and the segregated scheme, whose kernels are shorter, name theirs
 * at every size: convection, 20 steps, 343 elements of order 3 307 us with the
 * driver's choices and 247, 1000 456 and 307, 4096 727 and 728, of order 4 1390
 * and 1393; slower at 1728 of order 3, 491 and 541. */
template <typename... P>
inline int nsem_chain_split(int split, void (*kernel)(P...), unsigned grid, dim3 block, size_t smem) {
    int n = 0, dev = 0, sms = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, (int)(block.x * block.y), smem) != cudaSuccess ||
        cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
        (void)cudaGetLastError();
        return 0;
    }
    return grid <= (unsigned)n * (unsigned)sms ? split : 0;
}

template <typename... P, typename... A>
inline int nsem_launch_chained(void (*kernel)(P...), unsigned grid, dim3 block, size_t smem,
                               cudaStream_t st, int split, A... args) {
    cudaLaunchAttribute at[2] = {};
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
    at[1].val.sharedMemCarveout = (unsigned)split;
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(grid);
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = st;
    c.attrs = at;
    c.numAttrs = split > 0 ? 2 : 1;
    return (int)cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
}

#endif
