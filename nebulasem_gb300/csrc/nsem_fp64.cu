/*
 * Plain (FP64) form of the dGSEM Euler right-hand side and SSP-RK3 stage.
 *
 * Compiled with --fmad=false: every product and sum is rounded on its own, in
 * the order the reference evaluates it, so the GPU reproduces the reference's
 * CPU result bit for bit wherever the C library's pow is correctly rounded
 * (the equation of state uses the double-double pow of nsem_ddpow.h).
 *
 * Three kernels per stage:
 *   prim    per node: U = rho U / rho, theta = rho theta / rho,
 *           p' = P0 ((rho theta) R / P0)^gamma - p_ref, |U|, c = sqrt(gamma R theta)
 *           (apps/euler/euler.cpp:181-186, 211-213); run once per step, later
 *           stages get it from the volume kernel's epilogue;
 *   face    per used face slot: Rusanov fluxes of the three equations dotted
 *           with the weighted normal (src/field/field.h:2881-2943, 3086-3117),
 *           ghost states from applyExplicitBCs (field.h:2670-2685);
 *   volume  per element (one thread per node): surface lift in div_flux
 *           order, weak volume term gathered in the order the reference's
 *           scatter loop (field.h:3440-3464) adds it, gravity source,
 *           L = -Su/cV, Shu-Osher combination, primitives of the new state.
 * Roofline: FP64-pipe bound (hundreds of FP64 instructions per node-stage
 * against 40-80 bytes of traffic); products with the zeros of a diagonal
 * metric or an axis normal are left out and the other products, divisions,
 * roots and the power run on the integer pipes (nsem_gather.cuh, nsem_intfp.h).
 */
#include <cuda_runtime.h>

#include "nsem_ddpow.h"
#include "nsem_gather.cuh"
#include "nsem_internal.h"
#include "nsem_mortar.cuh"
#include "nsem_pdl.cuh"

namespace {

enum { XX, YY, ZZ, XY, YZ, XZ, YX, ZY, ZX };

__device__ __forceinline__ double vdot3(const double* a, const double* b) {
    return a[0] * b[0] + (a[1] * b[1] + (a[2] * b[2] + 0.0));
}

__device__ __forceinline__ void tdot(const double* q, const double* p, double* r) {
    r[0] = q[XX] * p[0] + q[XY] * p[1] + q[XZ] * p[2];
    r[1] = q[YX] * p[0] + q[YY] * p[1] + q[YZ] * p[2];
    r[2] = q[ZX] * p[0] + q[ZY] * p[1] + q[ZZ] * p[2];
}

__device__ __forceinline__ void outer(const double* p, const double* q, double* r) {
    r[XX] = p[0] * q[0];
    r[YY] = p[1] * q[1];
    r[ZZ] = p[2] * q[2];
    r[XY] = p[0] * q[1];
    r[YZ] = p[1] * q[2];
    r[XZ] = p[0] * q[2];
    r[YX] = p[1] * q[0];
    r[ZY] = p[2] * q[1];
    r[ZX] = p[2] * q[0];
}

/* ghost velocity of the SYMMETRY condition (src/tensor/tensor.h:486-494), en
 * the slot's unit normal */
__device__ __forceinline__ void sym_vec(const double* p, const double* en, double* out) {
    const double A0 = 1.0 - en[0] * en[0];
    const double A1 = 1.0 - en[1] * en[1];
    const double A2 = 1.0 - en[2] * en[2];
    const double A3 = 0.0 - en[0] * en[1];
    const double A4 = 0.0 - en[1] * en[2];
    const double A5 = 0.0 - en[0] * en[2];
    double r[3];
    r[0] = A0 * p[0] + A3 * p[1] + A5 * p[2];
    r[1] = A3 * p[0] + A1 * p[1] + A4 * p[2];
    r[2] = A5 * p[0] + A4 * p[1] + A2 * p[2];
    const double magR = nsem_sqrt(vdot3(r, r));
    if (fabs(magR - 0.0) <= 1e-7) {
        out[0] = r[0]; out[1] = r[1]; out[2] = r[2];
        return;
    }
    const double s = nsem_div(nsem_sqrt(vdot3(p, p)), magR);
    out[0] = r[0] * s; out[1] = r[1] * s; out[2] = r[2] * s;
}

struct PrimArgs {
    const double* S[5];
    double* prim[NSEM_NPRIM];
};

/* p', |U| and c of (r, U, T); INT: all mild, and the fluid's constants
 * (tame_const) */
template <bool INT>
__device__ __forceinline__ void prim_rest(const NsemDev& m, double r, const double* U, double T,
                                          double* const* prim, int64_t i) {
    const double x = nsem_div_by(nsem_x<INT>(m.R, nsem_x<INT>(r, T)), m.dP0);
    const double y = nsem_pow(x, m.gamma);
    /* the power of a mild argument can leave that range */
    const double p = nsem_mild(y) ? nsem_x<INT>(m.P0, y) : m.P0 * y;
    /* the sum of squares' trailing + 0.0 changes no square */
    const double uu = nsem_x<INT>(U[0], U[0]) + (nsem_x<INT>(U[1], U[1]) + nsem_x<INT>(U[2], U[2]));
    prim[0][i] = U[0];
    prim[1][i] = U[1];
    prim[2][i] = U[2];
    prim[3][i] = T;
    prim[4][i] = p - m.p_ref[i];
    prim[5][i] = nsem_sqrt(uu);
    prim[6][i] = nsem_sqrt(nsem_x<INT>(m.gR, T));
}

/* primitives of the state S at node i */
__device__ __forceinline__ void prim_at(const NsemDev& m, const double* S, double* const* prim,
                                        int64_t i) {
    const double r = S[0];
    const nsem_divisor dr = nsem_make_divisor(r);
    double U[3];
    U[0] = nsem_div_by(S[1], dr);
    U[1] = nsem_div_by(S[2], dr);
    U[2] = nsem_div_by(S[3], dr);
    const double T = nsem_div_by(S[4], dr);
    if (m.tame_const && nsem_mild(r) && nsem_mild(U[0]) && nsem_mild(U[1]) && nsem_mild(U[2]) && nsem_mild(T))
        prim_rest<true>(m, r, U, T, prim, i);
    else
        prim_rest<false>(m, r, U, T, prim, i);
}

__global__ void __launch_bounds__(256) k_prim(const NsemDev m, PrimArgs a) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    nsem_chain_wait();
    nsem_chain_begin();
    if (i >= m.n_int) return;
    double S[5];
    for (int c = 0; c < 5; c++) S[c] = a.S[c][i];
    prim_at(m, S, a.prim, i);
}

struct FaceArgs {
    const double* S0;            /* rho of the stage state */
    const double* prim[NSEM_NPRIM];
    double* d[5];
    const double* G[12];         /* viscous runs: grad U, grad theta (else null) */
    /* non-conforming faces, per mortar slot */
    double* mq[19];              /* the coarse side's interpolated quantities */
    double* mf[15];              /* face flux vectors (rho 3, momentum 9, theta 3) */
    double* dC[5];               /* projected, lifted coarse-side fluxes */
    int early;                   /* the volume kernel's CTAs may start beside this kernel */
};

/* Non-conforming faces: the coarse side's node quantities of the stage
 * state interpolated onto each mortar slot, one thread per (slot, quantity):
 * |U|, c, U rho (3), rho, the momentum flux tensor (rho U) (x) U + p' I
 * - mu grad U (9), the theta flux (rho U) theta - (mu / Pr) grad theta (3),
 * rho theta; each exactly as the face kernel forms it at a node. */
__global__ void __launch_bounds__(128) k_mortar_coupled(const NsemDev m, FaceArgs a) {
    const int64_t id = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= 19 * m.n_ms) return;
    const int64_t ms = id / 19;
    const int c = (int)(id % 19);
    const int t = c - 6;   /* tensor component of the momentum flux */
    const int ra = (t >= 0 && t < 9) ? (t < 3 ? t : (t == 3 || t == 5) ? 0 : (t == 4 || t == 6) ? 1 : 2) : 0;
    const int rb = (t >= 0 && t < 9) ? (t < 3 ? t : (t == 6 || t == 8) ? 0 : (t == 3 || t == 7) ? 1 : 2) : 0;
    double out[1];
    mortar_interp<1>(m, ms, [&](int64_t node, double* v) {
        const double r = a.S0[node];
        if (c == 0) v[0] = a.prim[5][node];
        else if (c == 1) v[0] = a.prim[6][node];
        else if (c < 5) v[0] = a.prim[c - 2][node] * r;
        else if (c == 5) v[0] = r;
        else if (c < 15) {
            double x = (a.prim[ra][node] * r) * a.prim[rb][node];
            x = x + ((t < 3) ? 1.0 : 0.0) * a.prim[4][node];
            if (a.G[0]) x = x - (r * m.nu) * a.G[t][node];
            v[0] = x;
        } else if (c < 18) {
            double x = (a.prim[c - 15][node] * r) * a.prim[3][node];
            if (a.G[0]) x = x - ((r * m.nu) * m.iPr) * a.G[9 + c - 15][node];
            v[0] = x;
        } else {
            v[0] = r * a.prim[3][node];
        }
    }, out);
    a.mq[c][ms] = out[0];
}

/* the coarse side's lifted values: the projected flux vectors dotted with the
 * slot's own weighted normal; one thread per (mortar slot, output row) */
__global__ void __launch_bounds__(128) k_mortar_coupled_gather(const NsemDev m, FaceArgs a) {
    const int64_t id = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= 5 * m.n_ms) return;
    const int64_t ms = id / 5;
    const int r = (int)(id % 5);
    const int64_t k = ms_field(m, NSEM_MS_K, ms);
    const double n[3] = {m.fn[k], m.fn[m.n_slot + k], m.fn[2 * m.n_slot + k]};
    double P[3];
    if (r == 0 || r == 4) {
        double* src[3] = {a.mf[r == 0 ? 0 : 12], a.mf[r == 0 ? 1 : 13], a.mf[r == 0 ? 2 : 14]};
        mortar_project<3>(m, ms, src, P);
        a.dC[r][ms] = vdot3(P, n);
    } else {
        const int q = r - 1;
        const int cx = q == 0 ? XX : q == 1 ? YX : ZX;
        const int cy = q == 0 ? XY : q == 1 ? YY : ZY;
        const int cz = q == 0 ? XZ : q == 1 ? YZ : ZZ;
        double* src[3] = {a.mf[3 + cx], a.mf[3 + cy], a.mf[3 + cz]};
        mortar_project<3>(m, ms, src, P);
        a.dC[r][ms] = P[0] * n[0] + P[1] * n[1] + P[2] * n[2];
    }
}

/* the five lifted values of a slot whose normal lies along axis ax (FP64-pipe
 * bound: about 60 operations instead of 190, with INT 20 and the products on
 * the integer pipes; 14 x 12 x 13 elements of order 4: 92 -> 38 -> 25 us) */
template <bool INT>
__device__ __forceinline__ void face_axis(const NsemDev& m, const FaceArgs& a, int64_t k, int ax,
                                          const double* n, const double* en, double fi, double fo,
                                          double lam, double r1, const double* U1, double T1, double p1,
                                          double r2, const double* U2, double T2, double p2,
                                          int32_t c1, int32_t c2) {
    const double na = nsem_pick(ax, n[0], n[1], n[2]), ea = nsem_pick(ax, en[0], en[1], en[2]);
    const double Ua1 = nsem_pick(ax, U1[0], U1[1], U1[2]), Ua2 = nsem_pick(ax, U2[0], U2[1], U2[2]);
    double Fc1[3], Fc2[3];
    for (int c = 0; c < 3; c++) {
        Fc1[c] = nsem_x<INT>(r1, U1[c]);
        Fc2[c] = nsem_x<INT>(r2, U2[c]);
    }
    const double Fa1 = nsem_pick(ax, Fc1[0], Fc1[1], Fc1[2]);
    const double Fa2 = nsem_pick(ax, Fc2[0], Fc2[1], Fc2[2]);
    /* artificial viscosity: mu = rho nu */
    const double mu1 = a.G[0] ? nsem_x<INT>(m.nu, r1) : 0.0, mu2 = a.G[0] ? nsem_x<INT>(m.nu, r2) : 0.0;
    auto avg = [&](double x, double y) { return nsem_x<INT>(fi, x) + nsem_x<INT>(fo, y); };
    a.d[0][k] = nsem_x<INT>(na, avg(Fa1, Fa2) - nsem_signed(ea, nsem_x<INT>(lam, r2 - r1)));
    const double dq = nsem_signed(ea, nsem_x<INT>(lam, Fa2 - Fa1));
    for (int r = 0; r < 3; r++) {
        double A = nsem_x<INT>(Ua1, Fc1[r]), B = nsem_x<INT>(Ua2, Fc2[r]);
        /* the pressure sits on the diagonal: p added there, 0 elsewhere */
        if (r == ax) { A += p1; B += p2; }
        if (a.G[0]) {
            const double* g = r == ax ? a.G[r] : a.G[r == 0 ? (ax == 1 ? XY : XZ)
                                                     : r == 1 ? (ax == 2 ? YZ : YX) : (ax == 0 ? ZX : ZY)];
            A = A - nsem_x<INT>(mu1, g[c1]);
            B = B - nsem_x<INT>(mu2, c2 >= 0 ? g[c2] : 0.0);
        }
        double F = avg(A, B);
        if (r == ax) F -= dq;
        a.d[1 + r][k] = nsem_x<INT>(na, F);
    }
    double x = nsem_x<INT>(T1, Fa1), y = nsem_x<INT>(T2, Fa2);
    if (a.G[0]) {
        x = x - nsem_x<INT>(nsem_x<INT>(m.iPr, mu1), a.G[9 + ax][c1]);
        y = y - nsem_x<INT>(nsem_x<INT>(m.iPr, mu2), c2 >= 0 ? a.G[9 + ax][c2] : 0.0);
    }
    a.d[4][k] = nsem_x<INT>(na, avg(x, y) - nsem_signed(ea, nsem_x<INT>(lam, nsem_x<INT>(r2, T2) - nsem_x<INT>(r1, T1))));
}

/* FACE threads a CTA, so that a small mesh's slots spread over the SMs */
constexpr int FACE = 64;

__global__ void __launch_bounds__(FACE) k_face(const NsemDev m, FaceArgs a) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= m.n_slot) return;   /* a CTA has at least one slot */
    const int32_t c1 = m.c1[k], c2 = m.c2[k];
    const double n[3] = {m.fn[k], m.fn[m.n_slot + k], m.fn[2 * m.n_slot + k]};
    const double en[3] = {m.en[k], m.en[m.n_slot + k], m.en[2 * m.n_slot + k]};
    const double fi = m.fi[k], fo = 1 - fi;
    nsem_chain_wait();
    if (a.early) nsem_chain_begin();

    const double r1 = a.S0[c1];
    const double U1[3] = {a.prim[0][c1], a.prim[1][c1], a.prim[2][c1]};
    const double T1 = a.prim[3][c1], p1 = a.prim[4][c1];
    const double mu1 = a.prim[5][c1], cs1 = a.prim[6][c1];
    double r2, U2[3], T2, p2, mu2, cs2;
    if (c2 >= 0) {
        r2 = a.S0[c2];
        U2[0] = a.prim[0][c2]; U2[1] = a.prim[1][c2]; U2[2] = a.prim[2][c2];
        T2 = a.prim[3][c2]; p2 = a.prim[4][c2];
        mu2 = a.prim[5][c2]; cs2 = a.prim[6][c2];
    } else {
        /* ghost node: NEUMANN (value 0) for rho, theta, p; velocity per bc */
        r2 = r1 + 0.0;
        T2 = T1 + 0.0;
        p2 = p1;
        if (m.bc[k] == 2) {
            sym_vec(U1, en, U2);
        } else {
            U2[0] = U1[0] + 0.0; U2[1] = U1[1] + 0.0; U2[2] = U1[2] + 0.0;
        }
        mu2 = nsem_sqrt(vdot3(U2, U2));
        cs2 = cs1;   /* sqrt(gamma R theta) of the same theta */
    }
    /* a mortar's coarse side (1: c1, 2: c2) takes interpolated quantities */
    const int32_t ms = m.n_ms ? m.ms_of[k] : -1;
    const int side = ms >= 0 ? ms_field(m, NSEM_MS_SIDE, ms) : 0;
    double mu1v = mu1, cs1v = cs1, r1v = r1, r2v = r2;
    if (side == 1) { mu1v = a.mq[0][ms]; cs1v = a.mq[1][ms]; r1v = a.mq[5][ms]; }
    if (side == 2) { mu2 = a.mq[0][ms]; cs2 = a.mq[1][ms]; r2v = a.mq[5][ms]; }
    const double lam = ((mu1v * fi + mu2 * fo) + (cs1v * fi + cs2 * fo)) / 2;

    /* a normal along one axis: only the flux tensor's column of that axis meets
     * a nonzero normal component; the products left out are zeros that change
     * no sum (the lift starts at +0), provided the flux components that meet a
     * zero stay finite: they have up to five factors, the normal not among them */
    const int ax = side == 0 ? nsem_axis_of(n, en) : -1;
    if (ax >= 0) {
        bool bounded = true, mild = !a.G[0] || m.tame_const;
        auto look = [&](double x) {
            bounded = bounded && nsem_bounded(x);
            mild = mild && nsem_flux_mild(x);
        };
        look(r1); look(r2); look(T1); look(T2); look(p1); look(p2); look(lam);
        look(fi); look(fo);
        for (int c = 0; c < 3; c++) { look(U1[c]); look(U2[c]); look(n[c]); }
        if (a.G[0]) {
            bounded = bounded && nsem_bounded(m.nu) && nsem_bounded(m.iPr);
            for (int c = 0; c < 12; c++) {
                look(a.G[c][c1]);
                if (c2 >= 0) look(a.G[c][c2]);
            }
        }
        if (bounded) {
            if (mild) face_axis<true>(m, a, k, ax, n, en, fi, fo, lam, r1, U1, T1, p1, r2, U2, T2, p2, c1, c2);
            else face_axis<false>(m, a, k, ax, n, en, fi, fo, lam, r1, U1, T1, p1, r2, U2, T2, p2, c1, c2);
            return;
        }
    }

    /* continuity: flux U rho, state rho */
    {
        double F[3];
        const double jump = lam * (r2v - r1v);
        for (int c = 0; c < 3; c++) {
            double x = U1[c] * r1, y = U2[c] * r2;
            if (side == 1) x = a.mq[2 + c][ms];
            if (side == 2) y = a.mq[2 + c][ms];
            F[c] = (x * fi + y * fo) - en[c] * jump;
        }
        a.d[0][k] = vdot3(F, n);
        if (side)
            for (int c = 0; c < 3; c++) a.mf[c][ms] = F[c];
    }
    /* momentum: flux (rho U)(x)U + p' I, state rho U */
    {
        double Fc1[3] = {U1[0] * r1, U1[1] * r1, U1[2] * r1};
        double Fc2[3] = {U2[0] * r2, U2[1] * r2, U2[2] * r2};
        double A[9], B[9], O[9], F[9], dq[3], out[3];
        outer(Fc1, U1, A);
        outer(Fc2, U2, B);
        for (int c = 0; c < 9; c++) {
            const double i1 = (c < 3) ? 1.0 : 0.0;
            A[c] = A[c] + i1 * p1;
            B[c] = B[c] + i1 * p2;
        }
        if (a.G[0]) {
            /* artificial viscosity: - mu grad U, mu = rho nu; zero gradient
             * on the wall ghosts (euler.cpp:189-190, 232) */
            const double mu1 = r1 * m.nu, mu2 = r2 * m.nu;
            for (int c = 0; c < 9; c++) {
                A[c] = A[c] - mu1 * a.G[c][c1];
                B[c] = B[c] - mu2 * (c2 >= 0 ? a.G[c][c2] : 0.0);
            }
        }
        if (side == 1) {
            for (int c = 0; c < 9; c++) A[c] = a.mq[6 + c][ms];
            for (int c = 0; c < 3; c++) Fc1[c] = a.mq[2 + c][ms];
        } else if (side == 2) {
            for (int c = 0; c < 9; c++) B[c] = a.mq[6 + c][ms];
            for (int c = 0; c < 3; c++) Fc2[c] = a.mq[2 + c][ms];
        }
        for (int c = 0; c < 3; c++) dq[c] = (Fc2[c] - Fc1[c]) * lam;
        outer(en, dq, O);
        for (int c = 0; c < 9; c++) F[c] = (A[c] * fi + B[c] * fo) - O[c];
        tdot(F, n, out);
        a.d[1][k] = out[0];
        a.d[2][k] = out[1];
        a.d[3][k] = out[2];
        if (side)
            for (int c = 0; c < 9; c++) a.mf[3 + c][ms] = F[c];
    }
    /* potential temperature: flux (rho U) theta, state rho theta */
    {
        double F[3];
        double s1 = r1 * T1, s2 = r2 * T2;
        if (side == 1) s1 = a.mq[18][ms];
        if (side == 2) s2 = a.mq[18][ms];
        const double jump = lam * (s2 - s1);
        for (int c = 0; c < 3; c++) {
            double x = (U1[c] * r1) * T1, y = (U2[c] * r2) * T2;
            if (a.G[0]) {
                /* - (mu / Pr) grad theta (euler.cpp:250) */
                x = x - ((r1 * m.nu) * m.iPr) * a.G[9 + c][c1];
                y = y - ((r2 * m.nu) * m.iPr) * (c2 >= 0 ? a.G[9 + c][c2] : 0.0);
            }
            if (side == 1) x = a.mq[15 + c][ms];
            if (side == 2) y = a.mq[15 + c][ms];
            F[c] = (x * fi + y * fo) - en[c] * jump;
        }
        a.d[4][k] = vdot3(F, n);
        if (side)
            for (int c = 0; c < 3; c++) a.mf[12 + c][ms] = F[c];
    }
}

struct VolArgs {
    const double* S[5];     /* stage state (input)               */
    const double* U0[5];    /* u^n (stages 2, 3)                 */
    double* out[5];         /* new stage state, or L (stage 0)   */
    double* prim[NSEM_NPRIM];
    const double* d[5];
    int stage;
    double dt;
    const double* G[12];    /* viscous runs: grad U, grad theta (else null) */
    const double* dC[5];    /* non-conforming faces: the coarse side's lifted values */
};

/* shared record per node: per direction c the flux column (U rho)_c, the
 * momentum tensor's column c, the theta flux' component c; then jin[9] */
constexpr int SM_W = 24;
constexpr unsigned SM_ROWS = 0xe;   /* the momentum equations are tensor rows */

/* the Shu-Osher combination of a stage; INT: operands mild (a sum that is not
 * mild takes its product in FP64).  A zero product keeps its sign: a momentum
 * of -0 without a tendency, L = -0, stays -0. */
template <bool INT>
__device__ __forceinline__ void update(int stage, double dt, const double* S, const double* U0,
                                       const double* L, double* nu) {
    const double cu = stage == 2 ? 0.75 : 1.0 / 3.0, cs = stage == 2 ? 0.25 : 2.0 / 3.0;
    auto mul = [](double a, double b) { return INT ? nsem_mul_signed(nsem_make_factor(a), b) : a * b; };
    for (int c = 0; c < 5; c++) {
        const double s = S[c] + mul(dt, L[c]);
        nu[c] = stage == 1 ? s : mul(cu, U0[c]) + (!INT || nsem_mild(s) ? mul(cs, s) : cs * s);
    }
}

/* registers for the largest element (1000 nodes, N+1 = 10) */
__global__ void __launch_bounds__(1024) k_volume(const NsemDev m, VolArgs a) {
    extern __shared__ double sm[];
    const int NPX = m.npx, NPY = m.npy, NPZ = m.npz, NP = m.np;
    double* dps = sm + (size_t)NP * SM_W;           /* 3 * npd^2 tables */
    const int t = threadIdx.x;
    nsem_load_tables(m, dps, t);

    const int64_t e = blockIdx.x;
    const bool active = t < NP;
    const int64_t node = e * NP + t;
    double rho = 0, U[3] = {0, 0, 0}, T = 0, pp = 0;
    if (active)
        for (int c = 0; c < 9; c++) sm[(size_t)t * SM_W + 15 + c] = m.jin[(int64_t)c * m.n_int + node];
    nsem_chain_wait();
    if (active) {
        rho = a.S[0][node];
        U[0] = a.prim[0][node]; U[1] = a.prim[1][node]; U[2] = a.prim[2][node];
        T = a.prim[3][node];
        pp = a.prim[4][node];
        double* my = sm + (size_t)t * SM_W;
        const bool mild = nsem_mild(rho) && nsem_mild(U[0]) && nsem_mild(U[1]) && nsem_mild(U[2]) &&
                          nsem_mild(T) && nsem_bounded(pp);
        double Fc[3];
        for (int c = 0; c < 3; c++) Fc[c] = mild ? nsem_x<true>(rho, U[c]) : rho * U[c];
        if (mild) nsem_flux_columns<5, 1, true>(my, Fc, U, T, pp);
        else nsem_flux_columns<5, 1, false>(my, Fc, U, T, pp);
        for (int c = 0; c < 3; c++) my[5 * c] = Fc[c];        /* U*rho == rho*U */
        if (a.G[0]) {
            const double mu = rho * m.nu;
            for (int c = 0; c < 3; c++) {
                const int row[3] = {c == 0 ? XX : c == 1 ? XY : XZ, c == 0 ? YX : c == 1 ? YY : YZ,
                                    c == 0 ? ZX : c == 1 ? ZY : ZZ};
                for (int r = 0; r < 3; r++) my[5 * c + 1 + r] -= mu * a.G[row[r]][node];
                my[5 * c + 4] -= (mu * m.iPr) * a.G[9 + c][node];
            }
        }
    }
    const int kind = nsem_element_kind<5>(m, active, sm + (size_t)t * SM_W);
    if (!active) return;

    /* surface lift, in the order div_flux visits the element's faces */
    double r[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    for (int j = 0; j < m.n_lift; j++) {
        const int32_t code = m.lift[(int64_t)j * m.n_int + node];
        if (code < 0) break;
        const int64_t k = code >> 2;
        for (int v = 0; v < 5; v++) {
            const double x = (code & 2) ? a.dC[v][k] : a.d[v][k];
            /* r - x is r + (-x): one add, the sign flipped in the bits */
            r[v] += __hiloint2double(__double2hiint(x) ^ (code << 31), __double2loint(x));
        }
    }

    /* weak volume term.  Source b adds -F_b . (Jin_b . dpsi(b->a)); sources
     * arrive in lexicographic order of b: X-line below, Y-line below, Z-line
     * below, self, Z above, Y above, X above. */
    nsem_chain_begin();
    nsem_volume_gather<5, SM_W, SM_ROWS>(NPX, NPY, NPZ, sm, dps, t, kind, r);

    /* gravity source: Su -= ((rho - rho_ref) g) cV */
    const double cv = m.cv[node];
    {
        const double s = rho - m.rho_ref[node];
        for (int c = 0; c < 3; c++) r[1 + c] = nsem_sub_source(r[1 + c], m.g[c], s, cv);
    }
    const nsem_divisor dcv = nsem_make_divisor(cv);
    double L[5];
    for (int v = 0; v < 5; v++) L[v] = -nsem_div_by(r[v], dcv);

    if (a.stage == 0) {
        for (int c = 0; c < 5; c++) a.out[c][node] = L[c];
        return;
    }
    double nu[5];
    bool finite = true, mild = nsem_mild(a.dt);
    double S[5], U0[5];
    for (int c = 0; c < 5; c++) {
        S[c] = a.S[c][node];
        mild = mild && nsem_mild(L[c]) && nsem_mild(S[c]);
    }
    if (a.stage > 1)
        for (int c = 0; c < 5; c++) {
            U0[c] = a.U0[c][node];
            mild = mild && nsem_mild(U0[c]);
        }
    if (mild) update<true>(a.stage, a.dt, S, U0, L, nu);
    else update<false>(a.stage, a.dt, S, U0, L, nu);
    for (int c = 0; c < 5; c++) {
        a.out[c][node] = nu[c];
        finite = finite && nsem_finite(nu[c]);
    }
    if (!finite) atomicOr(m.status, NSEM_STATUS_NONFINITE);
    /* primitives of the new stage state for the next face kernel */
    prim_at(m, nu, a.prim, node);
}

inline int launch_err() { return (int)cudaGetLastError(); }

}  // namespace

extern "C" int nsem_fp64_prim(const NsemDev* m, NsemBuf* b, const double* const* S, void* stream) {
    PrimArgs a;
    for (int c = 0; c < 5; c++) a.S[c] = S[c];
    for (int c = 0; c < NSEM_NPRIM; c++) a.prim[c] = b->prim[c];
    const int64_t blocks = (m->n_int + 255) / 256;
    return nsem_launch_chained(k_prim, (unsigned)blocks, 256, 0, (cudaStream_t)stream, m->split, *m, a);
}

extern "C" int nsem_fp64_face(const NsemDev* m, NsemBuf* b, const double* rho, void* stream) {
    FaceArgs a;
    a.S0 = rho;
    for (int c = 0; c < NSEM_NPRIM; c++) a.prim[c] = b->prim[c];
    for (int c = 0; c < 5; c++) a.d[c] = b->d[c];
    for (int c = 0; c < 12; c++) a.G[c] = b->G[c];
    for (int c = 0; c < 19; c++) a.mq[c] = b->mq[c];
    for (int c = 0; c < 15; c++) a.mf[c] = b->mf[c];
    for (int c = 0; c < 5; c++) a.dC[c] = b->dC[c];
    a.early = m->early;
    const int64_t blocks = (m->n_slot + FACE - 1) / FACE;
    cudaStream_t st = (cudaStream_t)stream;
    const unsigned mb = (unsigned)((m->n_ms + 127) / 128);
    if (m->n_ms > 0) k_mortar_coupled<<<19 * mb, 128, 0, st>>>(*m, a);
    int e = launch_err();
    if (!e) e = nsem_launch_chained(k_face, (unsigned)blocks, FACE, 0, st, m->split, *m, a);
    if (e) return e;
    if (m->n_ms > 0) k_mortar_coupled_gather<<<5 * mb, 128, 0, st>>>(*m, a);
    return launch_err();
}

static size_t vol_smem(const NsemDev* m) {
    return ((size_t)m->np * SM_W + 3 * NSEM_MAX_NPD * NSEM_MAX_NPD) * sizeof(double);
}

extern "C" int nsem_fp64_prepare(NsemDev* m) {
    const size_t smem = vol_smem(m);
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(k_volume, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)smem);
        if (e != cudaSuccess) return (int)e;
    }
    /* Whether the volume kernel's CTAs may start beside the face kernel, where
     * they gather on the SMs that its grid leaves free.  10 steps, after the face
     * kernel and beside it:
     *   - more than 32 warps an SM even out: 4 warps an element (order 4), 35 an
     *     SM 2880 and 2838 us, 77 5215 and 5140;
     *   - from 8 to 32, warps that share the pipes unevenly cost more: order 4,
     *     10 an SM 1424 and 1548 us, 19 1859 and 2154; full metric 17 3037 and 3861
     *     (above 26 the two are within 2 %, but one-warp elements of 2D lose up
     *     to 13 % at 24);
     *   - fewer leave the pipes idle either way, and starting early is worth 1 to
     *     3 % (one-warp elements of order 1 5 to 14 %), where each SM has a few
     *     CTAs to even out: order 2, 5.9 an SM 1181 and 1159 us; 2D, order 4, 8
     *     1207 and 1169.  With up to two, one SM in many gets twice the others'
     *     work: order 5, 0.4 elements an SM 1098 and 1327 us, 0.7 1216 and 1401;
     *     order 4, 0.5 1044 and 1170; 2D, order 4, 2 984 and 1032.  (Order 7, half
     *     an element, loses 1.5 % by this line.) */
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return (int)e;
    const double elems = (double)m->n_elem / sms, warps = elems * ((m->np + 31) / 32);
    m->early = warps > 32 || (warps < 8 && elems > 2.5);
    m->split = nsem_chain_split(NSEM_SPLIT, k_volume, (unsigned)m->n_elem, ((m->np + 31) / 32) * 32, smem);
    return 0;
}

extern "C" int nsem_fp64_volume(const NsemDev* m, NsemBuf* b, int stage,
                                double dt, const double* const* S, const double* const* U0,
                                double* const* out, void* stream) {
    VolArgs a;
    a.stage = stage;
    a.dt = dt;
    for (int c = 0; c < 5; c++) {
        a.d[c] = b->d[c];
        a.S[c] = S[c];
        a.U0[c] = U0[c];
        a.out[c] = out[c];
    }
    for (int c = 0; c < NSEM_NPRIM; c++) a.prim[c] = b->prim[c];
    for (int c = 0; c < 12; c++) a.G[c] = b->G[c];
    for (int c = 0; c < 5; c++) a.dC[c] = b->dC[c];
    const int threads = ((m->np + 31) / 32) * 32;
    return nsem_launch_chained(k_volume, (unsigned)m->n_elem, (unsigned)threads, vol_smem(m),
                               (cudaStream_t)stream, m->split, *m, a);
}
