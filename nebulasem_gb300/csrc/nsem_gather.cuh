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
 * three dpsi tables (dpsi[d][s * npd + i], NSEM_MAX_NPD^2 apart).  A source on
 * a line contributes its own metric column times one derivative (J[col] D),
 * the node itself the product Jinv . (Dx_ii, Dy_jj, Dz_kk) -- the reference's
 * products, evaluated in its operand order.  r[v] -= the contribution.
 *
 * Bound by the FP64 pipe (about 1.6 instructions per clock and SM), so the
 * operation count is the time.  On an element whose metric is diagonal
 * (`diag`: every off-diagonal component of every node is zero) a line source
 * has dj = (0, .., J_cc D, .., 0), and the products with the zeros are zeros
 * that change no sum: r starts at +0 and is never -0, so subtracting either
 * zero leaves it, and x + (+-0) is x for x != 0.  Such an element takes
 * J_cc D times the direction's own NC values, 1 + 2 NC operations a source
 * instead of 3 + 6 NC, with the same bits; the node's own term is formed in
 * full once, before the loop.  Zero times infinity is NaN and not zero, hence
 * `diag` also asks for values bounded so that no skipped product can overflow
 * (nsem_bounded); any other element takes the full products.  Measured
 * on 14 x 12 x 13 elements of order 4: an SSP-RK3 stage 552 -> 338 us (with
 * the faces' counterpart), a convection step of order 5 on 12 x 14 x 10
 * 196 -> 97 us.
 */
#ifndef NSEM_GATHER_CUH
#define NSEM_GATHER_CUH

#include "nsem_internal.h"

/* |x| < 2^200 (false for infinities and NaN): products of up to five such
 * factors stay finite */
__device__ __forceinline__ bool nsem_bounded(double x) {
    return (__double2hiint(x) & 0x7fffffff) < ((1023 + 200) << 20);
}

/* the bits of a zero of either sign, without an FP64 compare */
__device__ __forceinline__ bool nsem_is_zero(double x) {
    return ((__double2hiint(x) & 0x7fffffff) | __double2loint(x)) == 0;
}

/* this node's part of `diag`: my = its record in the layout above */
template <int NC>
__device__ __forceinline__ bool nsem_node_diag(const double* my) {
    bool ok = true;
#pragma unroll
    for (int c = 0; c < 3 * NC + 3; c++) ok = ok && nsem_bounded(my[c]);
#pragma unroll
    for (int c = 3; c < 9; c++) ok = ok && nsem_is_zero(my[3 * NC + c]);
    return ok;
}

/* x . dj as the reference sums it: vectors (rho, theta) from the last
 * component (its + 0.0 only turns -0 into +0, which no sum here shows), tensor
 * rows (ROW) from the first */
template <bool ROW>
__device__ __forceinline__ double nsem_dj_dot(double x0, double x1, double x2, const double* dj) {
    return ROW ? x0 * dj[0] + x1 * dj[1] + x2 * dj[2] : x0 * dj[0] + (x1 * dj[1] + x2 * dj[2]);
}

/* r[v] -= volume term of the NC equations; ROWS: bit v set where equation v is
 * a tensor row.  JOFF = 3 NC, W >= 3 NC + 9. */
template <int NC, int W, unsigned ROWS>
__device__ __forceinline__ void nsem_volume_gather(int npx, int npy, int npz, const double* sm,
                                                   const double* dps, int t, bool diag, double* r) {
    constexpr int M2 = NSEM_MAX_NPD * NSEM_MAX_NPD, JOFF = 3 * NC;
    static_assert(W >= JOFF + 9, "record: 3 NC flux values and the metric");
    /* metric columns of the X, Y and Z derivatives: (XX,YX,ZX), (XY,YY,ZY),
     * (XZ,YZ,ZZ), four bits per component index */
    constexpr int COLS_X = 0 | (6 << 4) | (8 << 8);
    constexpr int COLS_Y = 3 | (1 << 4) | (7 << 8);
    constexpr int COLS_Z = 5 | (4 << 4) | (2 << 8);
    const int ia = t / (npy * npz), ja = (t / npz) % npy, ka = t % npz;
    const int sx = npy * npz, sy = npz;
    auto full = [&](const double* s, const double* dj, double* out) {
#pragma unroll
        for (int v = 0; v < NC; v++)
            out[v] = (ROWS >> v & 1) ? nsem_dj_dot<true>(s[v], s[NC + v], s[2 * NC + v], dj)
                                     : nsem_dj_dot<false>(s[v], s[NC + v], s[2 * NC + v], dj);
    };
    double dj_self[3];
    {
        const double* J = sm + (size_t)t * W + JOFF;
        const double d0 = dps[ia * npx + ia], d1 = dps[M2 + ja * npy + ja],
                     d2 = dps[2 * M2 + ka * npz + ka];
        if (diag) {
            dj_self[0] = J[0] * d0;
            dj_self[1] = J[1] * d1;
            dj_self[2] = J[2] * d2;
        } else {
            dj_self[0] = J[0] * d0 + J[3] * d1 + J[5] * d2;
            dj_self[1] = J[6] * d0 + J[1] * d1 + J[4] * d2;
            dj_self[2] = J[8] * d0 + J[7] * d1 + J[2] * d2;
        }
    }
    const int L = npx + npy + npz - 2;
    const int xb = ia, yb = ia + ja, zb = ia + ja + ka;   /* ends of X<, Y<, Z< */
    const int za = ia + ja + npz;                         /* end of Z> */
    const int ya = ia + npy + npz - 1;                    /* end of Y> */
    /* direction of position p, the source's node and its derivative */
    auto source = [&](int p, int& dir, int& lb, double& D) {
        const bool on_x = p < xb || p >= ya;
        const bool on_y = !on_x && (p < yb || p >= za);
        const int q = on_x ? (p < xb ? p : p - npy - npz + 2)
                    : on_y ? (p < yb ? p - ia : p - ia - npz + 1)
                           : p - ia - ja;               /* Z line; q == ka at the node itself */
        const int da = on_x ? ia : on_y ? ja : ka;
        const int dn = on_x ? npx : on_y ? npy : npz;
        const int st = on_x ? sx : on_y ? sy : 1;
        dir = on_x ? 0 : on_y ? 1 : 2;
        lb = t + (q - da) * st;
        D = dps[dir * M2 + q * dn + da];
    };
    if (diag) {
        double own[NC];
        full(sm + (size_t)t * W, dj_self, own);
#pragma unroll 1
        for (int p = 0; p < L; p++) {
            int dir, lb;
            double D;
            source(p, dir, lb, D);
            const double* s = sm + (size_t)lb * W;
            const double x = s[JOFF + dir] * D;
            const bool self = p == zb;
            s += dir * NC;
#pragma unroll
            for (int v = 0; v < NC; v++) {
                const double y = s[v] * x;
                r[v] -= self ? own[v] : y;
            }
        }
        return;
    }
#pragma unroll 1
    for (int p = 0; p < L; p++) {
        int dir, lb;
        double D;
        source(p, dir, lb, D);
        const int cols = dir == 0 ? COLS_X : dir == 1 ? COLS_Y : COLS_Z;
        const bool self = p == zb;
        const double* s = sm + (size_t)lb * W;
        const double* J = s + JOFF;
        const double l0 = J[cols & 15] * D, l1 = J[(cols >> 4) & 15] * D, l2 = J[cols >> 8] * D;
        const double dj[3] = {self ? dj_self[0] : l0, self ? dj_self[1] : l1, self ? dj_self[2] : l2};
        double y[NC];
        full(s, dj, y);
#pragma unroll
        for (int v = 0; v < NC; v++) r[v] -= y[v];
    }
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
