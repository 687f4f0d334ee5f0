/*
 * The device build of nsem_intfp.h and nsem_ddpow.h against the hardware's
 * operations and the accurate power, for test_intfp_device.py: reciprocal and
 * root seeds, funnel shifts and carry chains that the host build does not have.
 */
#include <cuda_runtime.h>

#include "nsem_ddpow.h"

enum { DIV, SQRT, MUL, SIGNED, POW, UNDECIDED, COUNTERS };

static __device__ uint64_t mix(uint64_t z) {
    z += 0x9E3779B97F4A7C15ULL;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    return z ^ (z >> 31);
}
/* a value of exponent within 2^+-100, its significand random or with a long run
 * of zeros or ones, so that results lie on and beside rounding boundaries */
static __device__ double operand(uint64_t w, uint64_t k) {
    uint64_t m = w & 0xfffffffffffffULL;
    const uint64_t low = ((uint64_t)1 << (k % 53)) - 1;
    const int kind = (int)(k >> 8) & 3;
    if (kind == 1) m &= ~low;
    if (kind == 2) m |= low;
    return __longlong_as_double((long long)((w & ((uint64_t)1 << 63)) | (uint64_t)(923 + (k >> 20) % 200) << 52 | m));
}
static __device__ bool same(double a, double b) {
    return nsem_bits(a) == nsem_bits(b) || (a != a && b != b);
}

static __global__ void sweep(int64_t n, uint64_t seed, double y, unsigned long long* bad) {
    unsigned long long c[COUNTERS] = {};
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const uint64_t s = seed + 4 * (uint64_t)i;
        const double a = i % 1000 == 0 ? (i % 2000 ? 0.0 : -0.0) : operand(mix(s), mix(s + 2)), b = operand(mix(s + 1), mix(s + 3));
        const double p = a * b, r = fabs(b), q = r * r;
        /* the product and the square, and the values beside them */
        for (int d = -1; d <= 1; d++) {
            const double pd = p == 0.0 ? p : __longlong_as_double(__double_as_longlong(p) + d);
            const double qd = __longlong_as_double(__double_as_longlong(q) + d);
            c[DIV] += !same(nsem_div(pd, b), pd / b);
            c[SQRT] += !same(nsem_sqrt(qd), sqrt(qd));
        }
        c[DIV] += !same(nsem_div(a, b), a / b);
        c[SQRT] += !same(nsem_sqrt(r), sqrt(r));
        c[MUL] += p != 0.0 ? !same(nsem_mul_normal(nsem_make_factor(a), b), p)
                           : nsem_bits(nsem_mul_normal(nsem_make_factor(a), b)) != 0;
        c[SIGNED] += !same(nsem_mul_signed(nsem_make_factor(a), b), p);
        /* x in (0.25, 4) */
        const double x = __longlong_as_double((long long)((1021 + (mix(s + 2) >> 40) % 4) << 52 | (mix(s) & 0xfffffffffffffULL)));
        double w;
        if (!nsem_pow_int(x, y, &w)) c[UNDECIDED]++;
        else c[POW] += !same(w, nsem_pow_accurate(x, y));
    }
    for (int k = 0; k < COUNTERS; k++)
        if (c[k]) atomicAdd(bad + k, c[k]);
}

static __global__ void special(const double* v, int n, unsigned long long* bad) {
    for (int i = threadIdx.x; i < n * n; i += blockDim.x) {
        const double a = v[i / n], b = v[i % n];
        if (!same(nsem_div(a, b), a / b)) atomicAdd(bad + DIV, 1ull);
        if (!same(nsem_sqrt(a), sqrt(a))) atomicAdd(bad + SQRT, 1ull);
    }
}

/* counts of each kind of mismatch (COUNTERS values); values null: the sweep */
extern "C" int run(int64_t n, uint64_t seed, double y, const double* values, int n_values,
                   unsigned long long* out) {
    unsigned long long* d = nullptr;
    double* v = nullptr;
    cudaError_t e = cudaMalloc(&d, COUNTERS * sizeof(*d));
    if (e == cudaSuccess) e = cudaMemset(d, 0, COUNTERS * sizeof(*d));
    if (e == cudaSuccess && values) {
        e = cudaMalloc(&v, n_values * sizeof(double));
        if (e == cudaSuccess) e = cudaMemcpy(v, values, n_values * sizeof(double), cudaMemcpyHostToDevice);
        if (e == cudaSuccess) special<<<1, 256>>>(v, n_values, d);
    } else if (e == cudaSuccess) {
        sweep<<<608, 128>>>(n, seed, y, d);
    }
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpy(out, d, COUNTERS * sizeof(*d), cudaMemcpyDeviceToHost);
    cudaFree(d);
    cudaFree(v);
    return (int)e;
}
