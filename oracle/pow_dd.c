/*
 * Host build of the double-double pow (TEST INFRASTRUCTURE: lets the oracle
 * evaluate the equation of state with a correctly rounded pow, to measure
 * how much of the FP64 parity floor comes from the C library's pow rounding).
 */
#include "nsem_oracle.h"
#include "nsem_ddpow.h"

double nsem_oracle_pow_dd(double x, double y) { return nsem_pow(x, y); }

/* the accurate (double-double) phase alone */
double nsem_oracle_pow_dd_accurate(double x, double y) { return nsem_pow_accurate(x, y); }

/* the fast phase's unrounded result 2^k (hi + lo) and its error bound */
int nsem_oracle_pow_fast_core(double x, double y, double* hi, double* lo, double* err, int* k) {
    return nsem_pow_fast_core(x, y, hi, lo, err, k);
}

/* n pseudo-random x (log-uniform in [xlo, xhi]) for one exponent y: counts
 * the calls the fast phase could not round and the calls whose result
 * differs from the accurate phase (must be zero) */
void nsem_oracle_pow_fast_sweep(int64_t n, uint64_t seed, double xlo, double xhi, double y,
                                int64_t* fallbacks, int64_t* mismatches) {
    int64_t fb = 0, mm = 0;
    const double la = log(xlo), lb = log(xhi);
#pragma omp parallel for reduction(+ : fb, mm) schedule(static)
    for (int64_t i = 0; i < n; i++) {
        /* splitmix64 of (seed, i) */
        uint64_t z = seed + (uint64_t)i * 0x9E3779B97F4A7C15ULL;
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
        z = z ^ (z >> 31);
        const double f = (double)(z >> 11) * 0x1p-53;
        const double x = exp(la + (lb - la) * f);
        double r;
        const int ok = nsem_pow_fast(x, y, &r);
        if (!ok) fb++;
        else if (r != nsem_pow_accurate(x, y)) mm++;
    }
    *fallbacks = fb;
    *mismatches = mm;
}

static uint64_t splitmix(uint64_t z) {
    z += 0x9E3779B97F4A7C15ULL;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    return z ^ (z >> 31);
}

/* the same sweep for the fixed-point phase */
void nsem_oracle_pow_int_sweep(int64_t n, uint64_t seed, double xlo, double xhi, double y,
                               int64_t* fallbacks, int64_t* mismatches) {
    int64_t fb = 0, mm = 0;
    const double la = log(xlo), lb = log(xhi);
#pragma omp parallel for reduction(+ : fb, mm) schedule(static)
    for (int64_t i = 0; i < n; i++) {
        const double f = (double)(splitmix(seed + (uint64_t)i) >> 11) * 0x1p-53;
        const double x = exp(la + (lb - la) * f);
        double r;
        if (!nsem_pow_int(x, y, &r)) fb++;
        else if (r != nsem_pow_accurate(x, y)) mm++;
    }
    *fallbacks = fb;
    *mismatches = mm;
}

/* nsem_div, nsem_sqrt and nsem_mul_normal against the hardware on n operand
 * pairs: random significands, and ones with long runs of zeros and ones, whose
 * quotients, roots and products lie on and next to rounding boundaries;
 * bad: the mismatches of each */
void nsem_oracle_intfp_sweep(int64_t n, uint64_t seed, int64_t bad[3]) {
    int64_t bd = 0, bs = 0, bm = 0;
#pragma omp parallel for reduction(+ : bd, bs, bm) schedule(static)
    for (int64_t i = 0; i < n; i++) {
        double v[2];
        for (int q = 0; q < 2; q++) {
            const uint64_t w = splitmix(seed + 4 * (uint64_t)i + q), k = splitmix(seed + 4 * (uint64_t)i + 2 + q);
            uint64_t m = w & 0xfffffffffffffULL;
            const uint64_t low = ((uint64_t)1 << (k % 53)) - 1;
            if ((k >> 8) % 4 == 1) m &= ~low;
            if ((k >> 8) % 4 == 2) m |= low;
            if ((k >> 8) % 4 == 3 && (k >> 12) % 4 == 0) m = (k & 0x10000) ? m & 15 : ~m & 15 ? 0xfffffffffffffULL - (m & 15) : m;
            const uint64_t u = (w & ((uint64_t)1 << 63)) | (uint64_t)(923 + (k >> 20) % 200) << 52 | m;
            memcpy(&v[q], &u, 8);
        }
        const double a = i % 1000 == 0 ? 0.0 : v[0], b = v[1], c = fabs(b), s = c * c, p = a * b;
        const double t[3] = {s, nextafter(s, 0.0), nextafter(s, INFINITY)};
        const double d[3] = {p, nextafter(p, 0.0), nextafter(p, INFINITY)};
        bd += nsem_bits(nsem_div(a, b)) != nsem_bits(a / b);
        bs += nsem_bits(nsem_sqrt(c)) != nsem_bits(sqrt(c));
        bm += nsem_bits(nsem_mul_normal(nsem_make_factor(a), b)) != nsem_bits(p) && (p != 0.0);
        for (int q = 0; q < 3; q++) {
            bd += nsem_bits(nsem_div(d[q], b)) != nsem_bits(d[q] / b);
            bs += nsem_bits(nsem_sqrt(t[q])) != nsem_bits(sqrt(t[q]));
        }
    }
    bad[0] = bd;
    bad[1] = bs;
    bad[2] = bm;
}

/* one value of each, for operands the sweep does not reach */
double nsem_oracle_intfp_div(double a, double b) { return nsem_div(a, b); }
double nsem_oracle_intfp_sqrt(double a) { return nsem_sqrt(a); }
