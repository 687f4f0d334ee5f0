/*
 * Weak-form volume term gathered per target node in the order of the
 * reference's scatter loop (src/field/field.h:3440-3464): sources on the
 * X line below the node, Y below, Z below, the node itself, Z above, Y above,
 * X above.  Every node has the same number of sources, NPX + NPY + NPZ - 2, so
 * the loop runs over source positions p with one trip count for all threads
 * of the element; the (direction, source) of a position differs per thread and
 * is chosen by integer selects, and the floating-point work is issued once per
 * position for the whole warp.  Per-line loops with trip counts set by the
 * node's own (i, j, k) leave about half of the lanes idle in every FP64
 * instruction of the gather.
 *
 * sm: W doubles per node in shared memory: the NC flux values of each
 * direction, [3][NC] (value v of direction c at c NC + v), then the metric
 * Jinv cV at offset 3 NC (components XX,YY,ZZ,XY,YZ,XZ,YX,ZY,ZX); dps: the
 * three dpsi tables (nsem_load_tables).  A source on
 * a line contributes its own metric column times one derivative (J[col] D),
 * the node itself the product Jinv . (Dx_ii, Dy_jj, Dz_kk) -- the reference's
 * products, evaluated in its operand order.  r[v] -= the contribution.
 *
 * Bound by the FP64 pipe (about 1.6 instructions per clock and SM), so the
 * FP64 operation count is the time:
 *   - products run on the integer pipes (nsem_mul_normal: the same correctly
 *     rounded product), beside the FP64 pipe's additions, on an element whose
 *     values are zero or of a size at which every product is normal (`tame`;
 *     one value below 2^-400, as a wind far ahead of the sound front makes, sends
 *     its element to the full products in FP64);
 *   - on an element whose metric is also diagonal (every off-diagonal component
 *     of every node is zero) a line source has dj = (0, .., J_cc D, .., 0), and
 *     the products with the zeros are zeros that change no sum: r starts at +0
 *     and is never -0, so subtracting either zero leaves it, and x + (+-0) is x
 *     for x != 0.  Such an element takes J_cc D times the direction's own NC
 *     values, 1 + NC products and NC additions a source instead of 3 + 3 NC and
 *     3 NC; the node's own term is formed in full once, before the loop.
 * Zero times infinity is NaN and not zero, hence the bounds; any other element
 * takes the full products in FP64.  Same bits on every path.  Measured on 14 x
 * 12 x 13 elements of order 4, whole volume kernel: 453 us with the full
 * products, 168 us with the zeros left out and the integer divisions and power
 * (nsem_intfp.h, nsem_ddpow.h), 106 us with the integer products; a full metric
 * (12^3 elements tilted by 30 degrees, 5 SSP-RK3 steps) 6.7 -> 3.1 ms.
 */
#ifndef NSEM_GATHER_CUH
#define NSEM_GATHER_CUH

#include "nsem_internal.h"

/* the derivative tables into shared memory (their used entries), coalesced;
 * as a kernel parameter read per thread they serialise on the constant port,
 * about two microseconds of a one-warp CTA */
__device__ __forceinline__ void nsem_load_tables(const NsemDev& m, double* dps, int t) {
    const int npd[3] = {m.npx, m.npy, m.npz};
    for (int d = 0; d < 3; d++)
        for (int q = t; q < npd[d] * npd[d]; q += blockDim.x) {
            const int i = d * NSEM_MAX_NPD * NSEM_MAX_NPD + q;
            dps[i] = m.dpsi[i];
        }
}

/* |x| < 2^200 (false for infinities and NaN): products of up to five such
 * factors stay finite */
__device__ __forceinline__ bool nsem_bounded(double x) {
    return (__double2hiint(x) & 0x7fffffff) < ((1023 + 200) << 20);
}

/* the bits of a zero of either sign, without an FP64 compare */
__device__ __forceinline__ bool nsem_is_zero(double x) {
    return ((__double2hiint(x) & 0x7fffffff) | __double2loint(x)) == 0;
}

/* zero, or 2^-400 <= |x| < 2^200 */
__device__ __forceinline__ bool nsem_tame(double x) {
    const uint32_t h = (uint32_t)__double2hiint(x) & 0x7fffffffu;
    return h - ((1023u - 400u) << 20) < (600u << 20) || (h | (uint32_t)__double2loint(x)) == 0u;
}
/* zero, or 2^-K <= |x| < 2^K */
template <unsigned K>
__device__ __forceinline__ bool nsem_within(double x) {
    const uint32_t h = (uint32_t)__double2hiint(x) & 0x7fffffffu;
    return h - ((1023u - K) << 20) < (2u * K << 20) || (h | (uint32_t)__double2loint(x)) == 0u;
}
/* zero, or within 2^+-200: a product with a tame value is normal or zero */
__device__ __forceinline__ bool nsem_mild(double x) { return nsem_within<200>(x); }
/* a metric component whose product with a derivative (host-checked to be zero
 * or within 2^+-60) is mild */
__device__ __forceinline__ bool nsem_metric_tame(double J) { return nsem_within<140>(J); }

/* An axis flux multiplies up to five values and takes differences on the way,
 * which can cancel down to the last place of their terms, so mild values do not
 * suffice for its integer products.  With density, velocity, theta, pressure,
 * gradients, lambda, weights and normal within 2^+-180, the mass flux density
 * (rho U) within 2^+-360 and nu and 1 / Pr within 2^+-60 (tame_const), each
 * value is zero or, with its last place 52 bits below,
 *   U (rho U) + p' - mu g, theta (rho U) - (mu / Pr) g    2^-592 .. 2^542
 *   their weighted averages                               2^-772 .. 2^723
 *   averages less lambda (rho U), lambda (rho theta)      2^-824 .. 2^724
 *   that times the normal                                 2^-1004 .. 2^904
 * and no product leaves the normal range. */
__device__ __forceinline__ bool nsem_flux_mild(double x) { return nsem_within<180>(x); }
__device__ __forceinline__ bool nsem_mass_flux_mild(double x) { return nsem_within<360>(x); }

/* what nsem_volume_gather may do on an element: bit 0 every value tame, bit 1
 * the metric diagonal too */
enum { NSEM_EL_TAME = 1, NSEM_EL_DIAG = 2 };

/* this node's part of it: my = its record in the layout above.  */
template <int NC>
__device__ __forceinline__ int nsem_node_kind(const double* my) {
    bool tame = true, diag = true;
#pragma unroll
    for (int c = 0; c < 3 * NC; c++) tame = tame && nsem_tame(my[c]);
#pragma unroll
    for (int c = 0; c < 9; c++) {
        const double J = my[3 * NC + c];
        tame = tame && nsem_metric_tame(J);
        if (c >= 3) diag = diag && nsem_is_zero(J);
    }
    return (tame ? NSEM_EL_TAME : 0) | (tame && diag ? NSEM_EL_DIAG : 0);
}

/* the element's kind from its nodes' (barriers of the whole CTA) */
template <int NC>
__device__ __forceinline__ int nsem_element_kind(const NsemDev& m, bool active, const double* my) {
    const int k = active ? nsem_node_kind<NC>(my) : NSEM_EL_TAME | NSEM_EL_DIAG;
    const bool tame = __syncthreads_and(k & NSEM_EL_TAME), diag = __syncthreads_and(k & NSEM_EL_DIAG);
    return !(tame && m.tame_tables) ? 0 : diag ? NSEM_EL_TAME | NSEM_EL_DIAG : NSEM_EL_TAME;
}

struct NsemMulFp64 {
    double f;
    __device__ __forceinline__ explicit NsemMulFp64(double x) : f(x) {}
    __device__ __forceinline__ double operator()(double b) const { return f * b; }
};
struct NsemMulInt {
    nsem_factor f;
    __device__ __forceinline__ explicit NsemMulInt(double x) : f(nsem_make_factor(x)) {}
    __device__ __forceinline__ double operator()(double b) const { return nsem_mul_normal(f, b); }
};

/* a b, on the integer pipes (INT: operands mild, see nsem_mild) or in FP64 */
template <bool INT>
__device__ __forceinline__ double nsem_x(double a, double b) {
    if constexpr (INT) return nsem_mul_normal(nsem_make_factor(a), b);
    else return a * b;
}
/* x finite, by its bits */
__device__ __forceinline__ bool nsem_finite(double x) {
    return (__double2hiint(x) & 0x7ff00000) != 0x7ff00000;
}

/* x . dj as the reference sums it: vectors (rho, theta) from the last
 * component (its + 0.0 only turns -0 into +0, which no sum here shows), tensor
 * rows (ROW) from the first */
template <bool ROW, typename Mul>
__device__ __forceinline__ double nsem_dj_dot(double x0, double x1, double x2, const Mul* dj) {
    return ROW ? (dj[0](x0) + dj[1](x1)) + dj[2](x2) : dj[0](x0) + (dj[1](x1) + dj[2](x2));
}

/* the direction of source position p of the node (ia, ja, ka) = t, the
 * source's node and its derivative */
struct NsemSource {
    int npx, npy, npz, t, ia, ja, ka, xb, yb, zb, za, ya;
    __device__ __forceinline__ NsemSource(int nx, int ny, int nz, int t_)
        : npx(nx), npy(ny), npz(nz), t(t_), ia(t_ / (ny * nz)), ja((t_ / nz) % ny), ka(t_ % nz) {
        xb = ia; yb = ia + ja; zb = ia + ja + ka;   /* ends of X<, Y<, Z< */
        za = ia + ja + npz;                         /* end of Z> */
        ya = ia + npy + npz - 1;                    /* end of Y> */
    }
    __device__ __forceinline__ int count() const { return npx + npy + npz - 2; }
    __device__ __forceinline__ void at(int p, const double* dps, int& dir, int& lb, double& D) const {
        constexpr int M2 = NSEM_MAX_NPD * NSEM_MAX_NPD;
        const bool on_x = p < xb || p >= ya;
        const bool on_y = !on_x && (p < yb || p >= za);
        const int q = on_x ? (p < xb ? p : p - npy - npz + 2)
                    : on_y ? (p < yb ? p - ia : p - ia - npz + 1)
                           : p - ia - ja;               /* Z line; q == ka at the node itself */
        const int da = on_x ? ia : on_y ? ja : ka;
        const int dn = on_x ? npx : on_y ? npy : npz;
        const int st = on_x ? npy * npz : on_y ? npz : 1;
        dir = on_x ? 0 : on_y ? 1 : 2;
        lb = t + (q - da) * st;
        D = dps[dir * M2 + q * dn + da];
    }
};

/* the three components of Jinv . (d0, d1, d2) */
template <typename Mul>
__device__ __forceinline__ void nsem_dj_self(const double* J, const NsemSource& s, const double* dps,
                                             double* dj) {
    constexpr int M2 = NSEM_MAX_NPD * NSEM_MAX_NPD;
    const Mul d0(dps[s.ia * s.npx + s.ia]), d1(dps[M2 + s.ja * s.npy + s.ja]),
        d2(dps[2 * M2 + s.ka * s.npz + s.ka]);
    dj[0] = (d0(J[0]) + d1(J[3])) + d2(J[5]);
    dj[1] = (d0(J[6]) + d1(J[1])) + d2(J[4]);
    dj[2] = (d0(J[8]) + d1(J[7])) + d2(J[2]);
}

/* y[v] = value v's contribution F . dj of a node's record s */
template <int NC, unsigned ROWS, typename Mul>
__device__ __forceinline__ void nsem_dj_all(const double* s, const Mul* dj, double* y) {
#pragma unroll
    for (int v = 0; v < NC; v++)
        y[v] = (ROWS >> v & 1) ? nsem_dj_dot<true>(s[v], s[NC + v], s[2 * NC + v], dj)
                               : nsem_dj_dot<false>(s[v], s[NC + v], s[2 * NC + v], dj);
}

/* the full products, whatever the metric */
template <int NC, int W, unsigned ROWS, typename Mul>
__device__ __forceinline__ void nsem_gather_full(const NsemSource& src, const double* sm,
                                                 const double* dps, double* r) {
    constexpr int JOFF = 3 * NC;
    /* metric columns of the X, Y and Z derivatives: (XX,YX,ZX), (XY,YY,ZY),
     * (XZ,YZ,ZZ), four bits per component index */
    constexpr int COLS_X = 0 | (6 << 4) | (8 << 8);
    constexpr int COLS_Y = 3 | (1 << 4) | (7 << 8);
    constexpr int COLS_Z = 5 | (4 << 4) | (2 << 8);
    double dj_self[3];
    nsem_dj_self<Mul>(sm + (size_t)src.t * W + JOFF, src, dps, dj_self);
    const int L = src.count();
#pragma unroll 1
    for (int p = 0; p < L; p++) {
        int dir, lb;
        double D;
        src.at(p, dps, dir, lb, D);
        const int cols = dir == 0 ? COLS_X : dir == 1 ? COLS_Y : COLS_Z;
        const bool self = p == src.zb;
        const double* s = sm + (size_t)lb * W;
        const double* J = s + JOFF;
        const Mul d(D);
        const double l0 = d(J[cols & 15]), l1 = d(J[(cols >> 4) & 15]), l2 = d(J[cols >> 8]);
        const Mul dj[3] = {Mul(self ? dj_self[0] : l0), Mul(self ? dj_self[1] : l1),
                           Mul(self ? dj_self[2] : l2)};
        double y[NC];
        nsem_dj_all<NC, ROWS>(s, dj, y);
#pragma unroll
        for (int v = 0; v < NC; v++) r[v] -= y[v];
    }
}

/* r[v] -= volume term of the NC equations; ROWS: bit v set where equation v is
 * a tensor row; kind: nsem_element_kind.  JOFF = 3 NC, W >= 3 NC + 9. */
template <int NC, int W, unsigned ROWS>
__device__ __forceinline__ void nsem_volume_gather(int npx, int npy, int npz, const double* sm,
                                                   const double* dps, int t, int kind, double* r) {
    static_assert(W >= 3 * NC + 9, "record: 3 NC flux values and the metric");
    const NsemSource src(npx, npy, npz, t);
    if (!(kind & NSEM_EL_TAME)) {
        nsem_gather_full<NC, W, ROWS, NsemMulFp64>(src, sm, dps, r);
        return;
    }
    if (!(kind & NSEM_EL_DIAG)) {
        nsem_gather_full<NC, W, ROWS, NsemMulInt>(src, sm, dps, r);
        return;
    }
    constexpr int JOFF = 3 * NC;
    double own[NC];
    {
        double dj[3];
        nsem_dj_self<NsemMulInt>(sm + (size_t)t * W + JOFF, src, dps, dj);
        const NsemMulInt f[3] = {NsemMulInt(dj[0]), NsemMulInt(dj[1]), NsemMulInt(dj[2])};
        nsem_dj_all<NC, ROWS>(sm + (size_t)t * W, f, own);
    }
    const int L = src.count();
#pragma unroll 1
    for (int p = 0; p < L; p++) {
        int dir, lb;
        double D;
        src.at(p, dps, dir, lb, D);
        const double* s = sm + (size_t)lb * W;
        const NsemMulInt x(NsemMulInt(D)(s[JOFF + dir]));
        const bool self = p == src.zb;
        s += dir * NC;
#pragma unroll
        for (int v = 0; v < NC; v++) {
            const double y = x(s[v]);
            r[v] -= self ? own[v] : y;
        }
    }
}

/* the momentum and theta flux columns of a node in the record of NC values per
 * direction, Fc (x) U + p' I from value R0 on and Fc theta after it; INT: U and
 * T mild, Fc tame and below 2^400, p' bounded, so that the products run on the
 * integer pipes and the off-diagonal components' 0 p' is a zero that changes
 * nothing */
template <int NC, int R0, bool INT>
__device__ __forceinline__ void nsem_flux_columns(double* my, const double* Fc, const double* U, double T,
                                                  double pp) {
    for (int r = 0; r < 3; r++)
        for (int c = 0; c < 3; c++) {
            const double x = nsem_x<INT>(Fc[r], U[c]);
            my[NC * c + R0 + r] = r == c ? x + 1.0 * pp : INT ? x : x + 0.0 * pp;
        }
    for (int c = 0; c < 3; c++) my[NC * c + R0 + 3] = nsem_x<INT>(Fc[c], T);
}

/* r - (g s) cv */
__device__ __forceinline__ double nsem_sub_source(double r, double g, double s, double cv) {
    /* no gravity along the axis: 0 s cv is a zero that changes no sum */
    if (nsem_is_zero(g) && nsem_bounded(s) && nsem_bounded(cv)) return r;
    return r - (0.0 + g * s) * cv;
}

/* the axis a face slot's normal n lies along, with en its unit normal +-1 on
 * that axis, or -1 */
__device__ __forceinline__ int nsem_axis_of(const double* n, const double* en) {
    const bool z0 = nsem_is_zero(n[0]), z1 = nsem_is_zero(n[1]), z2 = nsem_is_zero(n[2]);
    const int axis = (!z0 && z1 && z2) ? 0 : (z0 && !z1 && z2) ? 1 : (z0 && z1 && !z2) ? 2 : -1;
    const double e = axis == 0 ? en[0] : axis == 1 ? en[1] : en[2];
    const double f = axis == 0 ? n[0] : axis == 1 ? n[1] : n[2];
    const bool unit = (__double2hiint(e) & 0x7fffffff) == 0x3ff00000 && __double2loint(e) == 0;
    return axis >= 0 && unit && nsem_bounded(f) ? axis : -1;
}
__device__ __forceinline__ double nsem_pick(int axis, double x0, double x1, double x2) {
    return axis == 0 ? x0 : axis == 1 ? x1 : x2;
}
/* e x for a unit normal component e = +-1 */
__device__ __forceinline__ double nsem_signed(double e, double x) {
    return __hiloint2double(__double2hiint(x) ^ (__double2hiint(e) & (int)0x80000000), __double2loint(x));
}

#endif
