/*
 * How results reach the caller's arrays: together through a pinned buffer, or
 * each by a copy of its own.  The rules stand apart from the CUDA calls, which
 * the caller passes in, so that they can be checked without a GPU.
 */
#ifndef NSEM_COPY_H
#define NSEM_COPY_H

#include <cstddef>

struct NsemHostCopy {
    double* dst;
    const double* src;
    size_t n;
    bool joins;   /* src continues the result before it, within one allocation */
};

/* several results that fit the pinned buffer together are staged, when the host
 * may write every destination itself (pageable(dst)); an array that the caller
 * has pinned takes its copy directly, and one that is no host memory is left to
 * the copy call, which reports it */
template <typename Pageable>
bool nsem_stage_results(const NsemHostCopy* c, int n, size_t room, Pageable pageable) {
    size_t total = 0;
    for (int i = 0; i < n; i++) total += c[i].n * sizeof(double);
    if (n < 2 || total > room) return false;
    for (int i = 0; i < n; i++)
        if (!pageable(c[i].dst)) return false;
    return true;
}

/* the copies, by copy(dst, src, values) until one fails: into the buffer one
 * after the other, or (buffer null) to the destinations */
template <typename Copy>
int nsem_copy_results(const NsemHostCopy* c, int n, double* buffer, Copy copy) {
    for (int i = 0, k; i < n; i = k) {
        /* staged results of one allocation side by side: one copy.  Equal
         * addresses would not say so: allocations of their own can be neighbours,
         * and a copy must not cross from one into the next */
        size_t m = c[i].n;
        for (k = i + 1; buffer && k < n && c[k].joins; k++) m += c[k].n;
        const int e = copy(buffer ? buffer : c[i].dst, c[i].src, m);
        if (e) return e;
        if (buffer) buffer += m;
    }
    return 0;
}

#endif
