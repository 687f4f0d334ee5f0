/*
 * Precision form on axis-aligned affine elements: the fused SSP-RK3 stage
 * kernel k_mixed_stage (FP32 line sums, or TF32 tensor-core line sums at
 * order 7) and the viscous runs' gradient kernel
 * k_mixed_grad, with their launches.  The algorithm is described in
 * nsem_mixed.cu.
 */
#include <cuda_runtime.h>

#include "nsem_mixed_kern.cuh"
#include "nsem_pdl.cuh"

using namespace nsem_mx;

namespace {

template <int NX, int NY, int NZ, bool TC = false>
struct StageSmem {
    using G = Geo<NX, NY, NZ>;
    static constexpr int NP = G::NP, NFS = G::NFS;
    /* floats: volume fluxes, line-major per direction [3][n][5][NL] (tensor-core
     * line sums: F[3][5][TC_NP]); own values P[NP] (x4) of the faces' jumps and
     * speeds: rho', Theta', |u|, c; face fluxes FF4[NFS] (x4) + FF1[NFS]; metric */
    static constexpr int FLUX = TC ? 15 * TC_NP : line_floats<NX, NY, NZ>();
    static constexpr int OFF_P = (FLUX + 3) / 4 * 4;
    static constexpr int OFF_FF4 = OFF_P + 4 * NP;
    static constexpr int OFF_FF1 = OFF_FF4 + 4 * NFS;
    static constexpr int OFF_META = OFF_FF1 + NFS;
    /* tensor-core line sums: the B fragments of Q_d^T pre-split into TF32
     * high and low parts, [3][2][8][8] words after the metric */
    static constexpr int OFF_QTC = OFF_META + 4;
    static constexpr size_t BYTES = sizeof(float) * ((OFF_QTC + (TC ? TC_QTAB : 0) + 3) / 4 * 4);
};

/* Tensor-core line sums (order 7, 8 nodes per direction).  The volume term
 * of direction d is, per conserved variable v and line l through the
 * element, r_l = Q_d f_l: as a matrix product R^T = F^T Q_d^T with the rows
 * (v, l) of F^T as M (5 x 64 = 320 rows: 20 tiles of 16), the 8 nodes along
 * the line as K and the 8 output nodes as N, one mma.sync m16n8k8 per tile
 * and TF32 pass.  FP32 accuracy from three TF32 products (a_lo b_hi +
 * a_hi b_lo + a_hi b_hi, Markidis' split; FP32 accumulation).  The fluxes
 * are kept per direction as F_d[v][a][m][b] in the swizzled layout tc_pos. */
__device__ __forceinline__ int tc_pos(int a, int m, int b) {
    const int hi = (m >> 2) & 1;
    return a * TC_SA + ((m ^ hi) << 3) + (b ^ (hi << 2));
}

template <int D>
__device__ __forceinline__ int tc_idx(int i, int j, int k) {
    return D == 0 ? tc_pos(j, i, k) : D == 1 ? tc_pos(i, j, k) : tc_pos(i, k, j);
}

__device__ __forceinline__ void split_tf32(float x, uint32_t& hi, uint32_t& lo) {
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(hi) : "f"(x));
    const float r = x - __uint_as_float(hi);
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(lo) : "f"(r));
}

__device__ __forceinline__ void mma_tf32(float (&c)[4], const uint32_t (&a)[4], uint32_t b0,
                                         uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
        "{%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

/* registers sized for 8 resident CTAs per SM in stages 1-2 and 9 in stage 3,
 * which loads the FP64 state only at the update (measured best on GB300:
 * 152 us at 32^3, against 172 us with the state held in registers at 7 CTAs
 * and 163 us at 8); viscous runs, which hold 12 gradients, 7 and 6 in stage 3
 * (9240 elements of order 4, 20 steps: 5186 us; 5311 us at 6 and at 5 with the
 * state held; 5196 at 6 and 6, 5182 at 7 and 7 with spills) */
#ifndef NSEM_MIXED_MB12
#define NSEM_MIXED_MB12 8
#endif
#ifndef NSEM_MIXED_MB3
#define NSEM_MIXED_MB3 9
#endif
template <int NX, int NY, int NZ, int STAGE, bool VISC>
constexpr int stage_min_blocks() {
    /* order 7 (512 threads, 64 KB of shared memory): three CTAs, two for the
     * stages that hold more live values (no spills) */
    if (Geo<NX, NY, NZ>::BLOCK >= 512)
        return min_blocks((VISC || STAGE == 0) ? 2 : 3, Geo<NX, NY, NZ>::BLOCK,
                          StageSmem<NX, NY, NZ>::BYTES);
    if (Geo<NX, NY, NZ>::EPB > 1) return 1;   /* 2D: 40 registers, for 12 CTAs, spill */
    return min_blocks(VISC ? (STAGE == 3 ? 6 : 7) : (STAGE == 1 || STAGE == 2) ? NSEM_MIXED_MB12 : NSEM_MIXED_MB3,
                      Geo<NX, NY, NZ>::BLOCK, StageSmem<NX, NY, NZ>::BYTES);
}

/* Strong-form DG gradients of U and theta of a stage state (gradf<true>,
 * field.h:3327-3360) for the viscous fluxes: per node
 *   d_r q = J_r sum_m D_r[a_r][m] q_m  +  (J_r / w_end) (cds(q) - q)  on the
 *   lower (-) / upper (+) face normal to r through the node,
 * cds = (own + neighbour) / 2 inside, the ghost value on a wall (SYMMETRY
 * velocity, NEUMANN theta: cds(theta) - theta = 0 there).  The state is the
 * stage kernel's (FP32 shadow plus the previous increment for SIN >= 2).
 * Output [e][12][NP]: tidx(r, c) = d_r U_c, 9 + r = d_r theta.
 * Written with explicit rounding throughout (no contraction left to the
 * compiler), so any kernel using these helpers forms the same bits. */

/* U = m / rho as the stage kernel forms it, and theta - T0 from the
 * perturbation: the background has theta = T0 (Theta_ref = rho_ref T0), so
 * theta - T0 = (Theta' - T0 rho') / rho -- the same gradient as theta without
 * FP32 cancellation against T0 */
__device__ __forceinline__ float4 prim_ut(const float* s, float rref, float T0) {
    const float inv = rcp_nr(__fadd_rn(rref, s[0]));
    return make_float4(__fmul_rn(s[1], inv), __fmul_rn(s[2], inv), __fmul_rn(s[3], inv),
                       __fmul_rn(__fmaf_rn(-T0, s[0], s[4]), inv));
}

/* the face term cds - own of face node slot t: O the neighbour's values, or
 * (o == nullptr) the wall ghost of the face's axis */
__device__ __forceinline__ float4 cds_minus_own(const float4 S, const float4* O, int dir) {
    float4 c;
    if (O) {
        c = make_float4(__fadd_rn(__fmul_rn(0.5f, S.x), __fmul_rn(0.5f, O->x)),
                        __fadd_rn(__fmul_rn(0.5f, S.y), __fmul_rn(0.5f, O->y)),
                        __fadd_rn(__fmul_rn(0.5f, S.z), __fmul_rn(0.5f, O->z)),
                        __fadd_rn(__fmul_rn(0.5f, S.w), __fmul_rn(0.5f, O->w)));
    } else {
        /* wall ghost: SYMMETRY velocity, NEUMANN theta */
        float r0 = dir == 0 ? 0.0f : S.x;
        float r1 = dir == 1 ? 0.0f : S.y;
        float r2 = dir == 2 ? 0.0f : S.z;
        const float mr = safe_sqrt(__fmaf_rn(r0, r0, __fmaf_rn(r1, r1, __fmul_rn(r2, r2))));
        if (mr > 1e-7f) {
            const float sc =
                __fdiv_rn(safe_sqrt(__fmaf_rn(S.x, S.x, __fmaf_rn(S.y, S.y, __fmul_rn(S.z, S.z)))), mr);
            r0 = __fmul_rn(r0, sc); r1 = __fmul_rn(r1, sc); r2 = __fmul_rn(r2, sc);
        }
        c = make_float4(r0, r1, r2, S.w);
    }
    return make_float4(__fsub_rn(c.x, S.x), __fsub_rn(c.y, S.y), __fsub_rn(c.z, S.z),
                       __fsub_rn(c.w, S.w));
}

/* phase 2: flux through face node t, seen from the element.  The face's
 * axis is a run-time value (selects, no branches), so a warp whose face
 * nodes lie on faces of two axes runs one instruction stream; the operations
 * and their operands are those of the plain per-axis form, so the two
 * elements of a face still produce exact negatives.  oth, bgo: the other
 * side's state and background, on a wall (nb = -1) the own node's. */
template <int NX, int NY, int NZ, bool VISC, bool TC>
__device__ __forceinline__ void face_flux(const FaceSlot& fs, int32_t nb, const float* oth,
                                          const float* bgo, const float* gfo, const float* sF,
                                          const float4* sP, const StageArgs& a, float4& o4,
                                          float& o1) {
    const int dir = fs.dir;
    const bool d0 = dir == 0, d1 = dir == 1, d2 = dir == 2;
    const float sg = fs.side ? 1.0f : -1.0f;   /* outward normal = sg e_dir */
    const Pt q = pointwise(oth, bgo, a.eos, a.gamma, a.gR);
    const float mdo = d0 ? oth[1] : d1 ? oth[2] : oth[3];
    if (nb >= 0) {
        float A[5];
        if constexpr (TC) {
            const int i = fs.la / (NY * NZ), j = (fs.la / NZ) % NY, k = fs.la % NZ;
            const float* f = sF + dir * 5 * TC_NP +
                             (d0 ? tc_idx<0>(i, j, k) : d1 ? tc_idx<1>(i, j, k) : tc_idx<2>(i, j, k));
#pragma unroll
            for (int v = 0; v < 5; v++) A[v] = f[v * TC_NP];
        } else {
            /* the node's flux row along the face's axis: the face plane's
             * row (first or last) at the node's in-plane index */
            using L0 = LineLay<NX, NY, NZ, 0>;
            using L1 = LineLay<NX, NY, NZ, 1>;
            using L2 = LineLay<NX, NY, NZ, 2>;
            const int row = d0 ? L0::BASE + (fs.side ? NX - 1 : 0) * L0::ROW
                          : d1 ? L1::BASE + (fs.side ? NY - 1 : 0) * L1::ROW
                               : L2::BASE + (fs.side ? NZ - 1 : 0) * L2::ROW;
            const float* f = sF + row + fs.r;
            const int nl = d0 ? L0::NL : d1 ? L1::NL : L2::NL;
#pragma unroll
            for (int v = 0; v < 5; v++) A[v] = f[v * nl];
        }
        /* the neighbour's volume flux along the axis (vol_flux of its node) */
        const float ud = d0 ? q.u[0] : d1 ? q.u[1] : q.u[2];
        float B[5];
        B[0] = mdo;
        B[1] = __fmaf_rn(oth[1], ud, d0 ? q.pp : 0.0f);
        B[2] = __fmaf_rn(oth[2], ud, d1 ? q.pp : 0.0f);
        B[3] = __fmaf_rn(oth[3], ud, d2 ? q.pp : 0.0f);
        B[4] = __fmul_rn(mdo, q.th);
        if constexpr (VISC) {
            /* gfo: the neighbour's d_c U_dir (c = 0..2) and d_dir theta */
            const float mu = __fmul_rn(q.rho, a.nu), mt = __fmul_rn(q.rho, a.nu_pr);
            B[1] = __fmaf_rn(-mu, gfo[0], B[1]);
            B[2] = __fmaf_rn(-mu, gfo[1], B[2]);
            B[3] = __fmaf_rn(-mu, gfo[2], B[3]);
            B[4] = __fmaf_rn(-mt, gfo[3], B[4]);
        }
        const float4 P = sP[fs.la];
        const float lam = __fmul_rn(0.25f, __fadd_rn(__fadd_rn(P.z, q.umag), __fadd_rn(P.w, q.c)));
        const float jr = __fsub_rn(oth[0], P.x);
        const float jm = __fsub_rn(mdo, A[0]);      /* the mass flux is the normal momentum */
        const float jt = __fsub_rn(oth[4], P.y);
        const float av0 = __fmul_rn(0.5f, __fadd_rn(A[0], B[0]));
        const float av1 = __fmul_rn(0.5f, __fadd_rn(A[1], B[1]));
        const float av2 = __fmul_rn(0.5f, __fadd_rn(A[2], B[2]));
        const float av3 = __fmul_rn(0.5f, __fadd_rn(A[3], B[3]));
        const float av4 = __fmul_rn(0.5f, __fadd_rn(A[4], B[4]));
        const float s1 = sg * av1, s2 = sg * av2, s3 = sg * av3;
        o4.x = __fmaf_rn(-lam, jr, sg * av0);
        o4.y = d0 ? __fmaf_rn(-lam, jm, s1) : s1;
        o4.z = d1 ? __fmaf_rn(-lam, jm, s2) : s2;
        o4.w = d2 ? __fmaf_rn(-lam, jm, s3) : s3;
        o1 = __fmaf_rn(-lam, jt, sg * av4);
    } else {
        /* wall ghost: rho, theta, p NEUMANN; SYMMETRY velocity (tangential
         * projection rescaled to |U|, tensor.h:486-494), normal velocity 0.
         * The ghost value alone is the face average (fI = 0 on a wall,
         * field.cpp:257-266), so only the normal momentum flux remains:
         * s p' + lam m_n, lam = (|U_ghost| + c) / 2.  No viscous wall flux
         * (zero ghost gradient). */
        const float r0 = d0 ? 0.0f : q.u[0];
        const float r1 = d1 ? 0.0f : q.u[1];
        const float r2 = d2 ? 0.0f : q.u[2];
        const float mr = safe_sqrt(__fmaf_rn(r0, r0, __fmaf_rn(r1, r1, __fmul_rn(r2, r2))));
        const float um_g = mr > 1e-7f ? q.umag : mr;
        const float lam = __fmul_rn(0.5f, __fadd_rn(um_g, q.c));
        const float fn = __fmaf_rn(lam, mdo, sg * q.pp);
        o4 = make_float4(0.0f, d0 ? fn : 0.0f, d1 ? fn : 0.0f, d2 ? fn : 0.0f);
        o1 = 0.0f;
    }
}

/* one kernel per stage (0: tendency only): the stage's own loads and update */
template <int NX, int NY, int NZ, int STAGE, bool VISC, bool TC>
__global__ void __launch_bounds__(Geo<NX, NY, NZ>::BLOCK * Geo<NX, NY, NZ>::EPB, (stage_min_blocks<NX, NY, NZ, STAGE, VISC>()))
k_mixed_stage(StageArgs a) {
    static_assert(!TC || (NX == 8 && NY == 8 && NZ == 8), "tensor-core line sums: order 7");
    using G = Geo<NX, NY, NZ>;
    using SM = StageSmem<NX, NY, NZ, TC>;
    constexpr int NP = G::NP;
    constexpr int NFS = G::NFS;
    extern __shared__ float4 smem4[];
    float* smem = reinterpret_cast<float*>(G::template smem_of<SM::BYTES>(smem4));
    float4* sP = reinterpret_cast<float4*>(smem + SM::OFF_P);     /* [NP] */
    float4* sFF4 = reinterpret_cast<float4*>(smem + SM::OFF_FF4); /* [NFS] */
    float* sFF1 = smem + SM::OFF_FF1;                             /* [NFS] */
    float* sMeta = smem + SM::OFF_META;

    const int t = threadIdx.x;
    const int64_t e = G::element();
    if (G::EPB > 1 && e >= a.n_elem) return;
    constexpr bool has_din = STAGE >= 2;
    if constexpr (TC) {
        float* sQtc = smem + SM::OFF_QTC;
        for (int q = t; q < TC_QTAB; q += G::BLOCK) sQtc[q] = __ldg(a.Qg + QTAB + q);
    }

    /* what no kernel of the chain writes, before the wait for the previous
     * kernel: background, neighbours, metric */
    float own[5], din[5] = {0, 0, 0, 0, 0}, bgs[4] = {0, 0, 0, 0};
    float gown[12];
    /* 30 steps in 2D, at the update and here: 24 x 24 elements of order 4 303
     * and 295 us, 40 x 40 347 and 338, 88 x 90 748 and 741; viscous, whose 74
     * registers cost CTAs, 88 x 90 1381 and 1408 */
    constexpr bool EARLY_U = STAGE == 3 && G::EPB > 1 && !VISC;
    double u64[5];
    if (t < NP) load_bg<NX, NY, NZ>(a, __ldg(a.layer + e), -1, t, bgs);
    FaceSlot fs{};
    int32_t nb = -1;
    /* the other side's node; a wall's flux is formed from the own trace */
    int64_t eo = e;
    int lo = 0;
    float oth[5], bgo[4];
    float gfo[4] = {0, 0, 0, 0};
    if (t < NFS) {
        fs = face_slot<NX, NY, NZ, STAGE == 1 || STAGE == 2>(t);
        nb = __ldg(a.nbr + (int64_t)fs.face * a.n_elem + e);
        lo = fs.la;
        if (nb >= 0) { eo = nb; lo = fs.lo; }
        load_bg<NX, NY, NZ>(a, __ldg(a.layer + eo), nb >= 0 ? t : -1, lo, bgo);
    }
    if (t < 3) sMeta[t] = __ldg(a.J + (int64_t)t * a.n_elem + e);
    nsem_chain_wait();

    /* every other global load: own node, face neighbour, stage-3 FP64 */
    if (t < NP) {
        const float* s = a.S + e * 5 * NP + t;
#pragma unroll
        for (int v = 0; v < 5; v++) own[v] = s[v * NP];
        if constexpr (has_din) {
            const float* d = a.Din + e * 5 * NP + t;
#pragma unroll
            for (int v = 0; v < 5; v++) {
                din[v] = d[v * NP];
                own[v] = __fadd_rn(own[v], din[v]);
            }
        }
        if constexpr (STAGE == 3) {
            /* u'^n is needed only at the update: fetched into L2 here and
             * loaded there (with the increment reloaded from L1/L2), so that
             * neither holds registers through the element and nine CTAs (six
             * in viscous runs) fit per SM.  Inviscid runs in 2D load it here:
             * their registers suffice, and the wait at the update is gone */
            const double* u = a.U + e * 5 * NP + t;
#pragma unroll
            for (int v = 0; v < 5; v++) {
                if constexpr (EARLY_U) u64[v] = u[v * NP];
                else asm volatile("prefetch.global.L2 [%0];" ::"l"(u + v * NP));
            }
        }
        if constexpr (VISC) {
            const float* gr = a.G + e * 12 * NP + t;
#pragma unroll
            for (int c = 0; c < 12; c++) gown[c] = gr[c * NP];
        }
    }
    if (t < NFS) {
        if (nb <= -2) {
            /* a face on a 2:1 mortar: its outward values come from the
             * mortar kernels */
            const float* mf = a.MF + (int64_t)(-2 - nb) * MF_ROWS * a.nfmax + face_local<NX, NY, NZ>(t);
#pragma unroll
            for (int v = 0; v < 5; v++) oth[v] = mf[v * a.nfmax];
        } else {
            const float* s = a.S + eo * 5 * NP + lo;
#pragma unroll
            for (int v = 0; v < 5; v++) oth[v] = s[v * NP];
            if constexpr (has_din) {
                const float* d = a.Din + eo * 5 * NP + lo;
#pragma unroll
                for (int v = 0; v < 5; v++) oth[v] = __fadd_rn(oth[v], d[v * NP]);
            }
            if constexpr (VISC) {
                /* the neighbour's gradients along the face's axis only:
                 * d_c U_dir (c = 0..2) and d_dir theta */
                const float* gr = a.G + eo * 12 * NP + lo;
                const int d = fs.dir;
                gfo[0] = gr[tidx(0, d) * NP];
                gfo[1] = gr[tidx(1, d) * NP];
                gfo[2] = gr[tidx(2, d) * NP];
                gfo[3] = gr[(9 + d) * NP];
            }
        }
    }

    /* phase 1: own node primitives and volume fluxes */
    if (t < NP) {
        const Pt p = pointwise(own, bgs, a.eos, a.gamma, a.gR);
        sP[t] = make_float4(own[0], own[4], p.umag, p.c);
        float4 f4;
        float f1;
        if constexpr (TC) {
            const int i = t >> 6, j = (t >> 3) & 7, k = t & 7;
            auto put = [&](int d, int idx, const float4& v4, float v1) {
                float* f = smem + d * 5 * TC_NP + idx;
                f[0] = v4.x; f[TC_NP] = v4.y; f[2 * TC_NP] = v4.z; f[3 * TC_NP] = v4.w;
                f[4 * TC_NP] = v1;
            };
            vol_flux<0, VISC>(own, p, gown, a.nu, a.nu_pr, f4, f1);
            put(0, tc_idx<0>(i, j, k), f4, f1);
            vol_flux<1, VISC>(own, p, gown, a.nu, a.nu_pr, f4, f1);
            put(1, tc_idx<1>(i, j, k), f4, f1);
            vol_flux<2, VISC>(own, p, gown, a.nu, a.nu_pr, f4, f1);
            put(2, tc_idx<2>(i, j, k), f4, f1);
        } else {
            const int i = t / (NY * NZ), j = (t / NZ) % NY, k = t % NZ;
            auto put = [&](float* f, int nl, const float4& v4, float v1) {
                f[0] = v4.x; f[nl] = v4.y; f[2 * nl] = v4.z; f[3 * nl] = v4.w; f[4 * nl] = v1;
            };
            vol_flux<0, VISC>(own, p, gown, a.nu, a.nu_pr, f4, f1);
            put(smem + LineLay<NX, NY, NZ, 0>::at(i, j, k), LineLay<NX, NY, NZ, 0>::NL, f4, f1);
            if constexpr (G::HAS_Y) {
                vol_flux<1, VISC>(own, p, gown, a.nu, a.nu_pr, f4, f1);
                put(smem + LineLay<NX, NY, NZ, 1>::at(i, j, k), LineLay<NX, NY, NZ, 1>::NL, f4, f1);
            }
            vol_flux<2, VISC>(own, p, gown, a.nu, a.nu_pr, f4, f1);
            put(smem + LineLay<NX, NY, NZ, 2>::at(i, j, k), LineLay<NX, NY, NZ, 2>::NL, f4, f1);
        }
    }
    G::sync();
    /* phase 2: Rusanov flux on every face node */
    if (t < NFS) {
        float4 o4;
        float o1;
        if (nb <= -2) {
            o4 = make_float4(oth[0], oth[1], oth[2], oth[3]);
            o1 = oth[4];
        } else {
            face_flux<NX, NY, NZ, VISC, TC>(fs, nb, oth, bgo, gfo, smem, sP, a, o4, o1);
        }
        sFF4[t] = o4;
        sFF1[t] = o1;
    }
    G::sync();

    /* the next stage's CTAs may start: launched earlier (at the start, or after
     * the wait) they take the slots of a grid below one wave unevenly
     * (9 x 7 x 11 elements, 40 steps: 767 us at the start, 756 after the wait,
     * 666 here, 679 never; 10 x 10 in 2D, 50 steps: 465, 443, 444, 515) */
    nsem_chain_begin();
    /* phase 3: weak volume term (line sums with Q), lift, buoyancy, update */
    if constexpr (TC) {
        /* tensor-core line sums, results in place of the fluxes */
        const int lane = t & 31, w = t >> 5, gq = lane >> 2, tg = lane & 3;
        /* lane offsets of the A fragment (rows m = tg, tg + 4) and of the C
         * fragment (rows 2 tg, 2 tg + 1), line b = gq, within a tile */
        const int oa0 = tc_pos(0, tg, gq), oa2 = tc_pos(0, tg + 4, gq);
        const int oc0 = tc_pos(0, 2 * tg, gq), oc1 = tc_pos(0, 2 * tg + 1, gq);
        for (int q = w; q < 60; q += G::BLOCK / 32) {
            const int d = q / 20, r = q % 20, v = r >> 2, a0 = (r & 3) * 2;
            float* base = smem + d * 5 * TC_NP + v * TC_NP + a0 * TC_SA;
            uint32_t ah[4], al[4], bh0, bl0, bh1, bl1;
            split_tf32(base[oa0], ah[0], al[0]);
            split_tf32(base[TC_SA + oa0], ah[1], al[1]);
            split_tf32(base[oa2], ah[2], al[2]);
            split_tf32(base[TC_SA + oa2], ah[3], al[3]);
            /* B = Q_d^T, pre-split on the host exactly as split_tf32 would:
             * rows k = tg, tg + 4 of the high and the low part, column n = gq */
            const float* qb = smem + SM::OFF_QTC + d * 128 + tg * 8 + gq;
            bh0 = __float_as_uint(qb[0]);
            bh1 = __float_as_uint(qb[32]);
            bl0 = __float_as_uint(qb[64]);
            bl1 = __float_as_uint(qb[96]);
            float c[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            mma_tf32(c, al, bh0, bh1);
            mma_tf32(c, ah, bl0, bl1);
            mma_tf32(c, ah, bh0, bh1);
            base[oc0] = c[0];
            base[oc1] = c[1];
            base[TC_SA + oc0] = c[2];
            base[TC_SA + oc1] = c[3];
        }
        G::sync();
    } else {
        line_transform<NX, NY, NZ, 0>(smem, a, t);
        if constexpr (G::HAS_Y) line_transform<NX, NY, NZ, 1>(smem, a, t);
        line_transform<NX, NY, NZ, 2>(smem, a, t);
        G::sync();
    }
    if (t < NP) {
    const int i = t / (NY * NZ), j = (t / NZ) % NY, k = t % NZ;
    float L0, L1, L2, L3, L4;
    if constexpr (TC) {
        const float Jx = sMeta[0], Jy = sMeta[1], Jz = sMeta[2];
        const float* rx = smem + tc_idx<0>(i, j, k);
        const float* ry = smem + 5 * TC_NP + tc_idx<1>(i, j, k);
        const float* rz = smem + 10 * TC_NP + tc_idx<2>(i, j, k);
        float Lt[5];
#pragma unroll
        for (int v = 0; v < 5; v++)
            Lt[v] = fmaf(Jz, rz[v * TC_NP], fmaf(Jy, ry[v * TC_NP], Jx * rx[v * TC_NP]));
        L0 = Lt[0]; L1 = Lt[1]; L2 = Lt[2]; L3 = Lt[3]; L4 = Lt[4];
    } else {
        /* the three directions' line sums at this node, scaled by J_d */
        const float* rx = smem + LineLay<NX, NY, NZ, 0>::at(i, j, k);
        const float* rz = smem + LineLay<NX, NY, NZ, 2>::at(i, j, k);
        constexpr int NLX = LineLay<NX, NY, NZ, 0>::NL, NLZ = LineLay<NX, NY, NZ, 2>::NL;
        const float Jx = sMeta[0], Jz = sMeta[2];
        float Lt[5];
#pragma unroll
        for (int v = 0; v < 5; v++) Lt[v] = Jx * rx[v * NLX];
        if constexpr (G::HAS_Y) {
            const float* ry = smem + LineLay<NX, NY, NZ, 1>::at(i, j, k);
            constexpr int NLY = LineLay<NX, NY, NZ, 1>::NL;
            const float Jy = sMeta[1];
#pragma unroll
            for (int v = 0; v < 5; v++) Lt[v] = fmaf(Jy, ry[v * NLY], Lt[v]);
        }
#pragma unroll
        for (int v = 0; v < 5; v++) Lt[v] = fmaf(Jz, rz[v * NLZ], Lt[v]);
        L0 = Lt[0]; L1 = Lt[1]; L2 = Lt[2]; L3 = Lt[3]; L4 = Lt[4];
    }
    /* surface lift: -(J_d / w_end) F_out for the face of each axis through
     * the node (at most one per axis) */
    auto lift = [&](int slot, float coef) {
        const float4 f = sFF4[slot];
        L0 = fmaf(-coef, f.x, L0); L1 = fmaf(-coef, f.y, L1); L2 = fmaf(-coef, f.z, L2);
        L3 = fmaf(-coef, f.w, L3); L4 = fmaf(-coef, sFF1[slot], L4);
    };
    {
        const int sx = face_of_node<NX, NY, NZ, 0>(i, j, k);
        if (sx >= 0) lift(sx, sMeta[0] * a.lift[0]);
        if constexpr (G::HAS_Y) {
            const int sy = face_of_node<NX, NY, NZ, 1>(i, j, k);
            if (sy >= 0) lift(sy, sMeta[1] * a.lift[1]);
        }
        const int sz = face_of_node<NX, NY, NZ, 2>(i, j, k);
        if (sz >= 0) lift(sz, sMeta[2] * a.lift[2]);
    }
    /* buoyancy (rho - rho_ref) g */
    const float rp = own[0];
    L1 = fmaf(rp, a.g[0], L1);
    L2 = fmaf(rp, a.g[1], L2);
    L3 = fmaf(rp, a.g[2], L3);
    const float Lv[5] = {L0, L1, L2, L3, L4};

    if constexpr (STAGE == 0) {
        const int64_t n = e * NP + t;
#pragma unroll
        for (int v = 0; v < 5; v++) a.L[v][n] = f2d(Lv[v]);
    }
    const int64_t o = e * 5 * NP + t;
    const float dt = a.dt;
    if constexpr (STAGE == 1) {
#pragma unroll
        for (int v = 0; v < 5; v++) a.Dout[o + v * NP] = dt * Lv[v];
    } else if constexpr (STAGE == 2) {
#pragma unroll
        for (int v = 0; v < 5; v++) a.Dout[o + v * NP] = 0.25f * fmaf(dt, Lv[v], din[v]);
    } else if constexpr (STAGE == 3) {
        update_state<NP, EARLY_U>(a, o, Lv, din, u64);
    }
    }  /* t < NP */
}

template <int NX, int NY, int NZ, int SIN>
__global__ void __launch_bounds__(Geo<NX, NY, NZ>::BLOCK * Geo<NX, NY, NZ>::EPB)
k_mixed_grad(StageArgs a) {
    using G = Geo<NX, NY, NZ>;
    constexpr int NP = G::NP;
    constexpr int NFS = G::NFS;
    constexpr bool has_din = SIN >= 2;
    using GL = GradLay<NX, NY, NZ>;
    extern __shared__ float4 gsm[];
    __shared__ float sJ_of[G::EPB][3];
    float4* gsm4 = G::template smem_of<GL::BYTES>(gsm);
    float* sJ = sJ_of[G::EPB > 1 ? threadIdx.y : 0];
    float4* sD = gsm4 + GL::OFF_D;                                  /* [NFS] cds - own */
    const int t = threadIdx.x;
    const int64_t e = G::element();
    if (G::EPB > 1 && e >= a.n_elem) return;

    float own[5], bgs0 = 0.0f;
    if (t < NP) bgs0 = __ldg(a.bg + (int64_t)__ldg(a.layer + e) * 4 * NP + t);
    FaceSlot fs{};
    int32_t nb = -1;
    float oth[5], bgo0 = 0.0f;
    if (t < NFS) {
        fs = face_slot<NX, NY, NZ>(t);
        nb = __ldg(a.nbr + (int64_t)fs.face * a.n_elem + e);
        if (nb >= 0) bgo0 = __ldg(a.bg + (int64_t)__ldg(a.layer + nb) * 4 * NP + fs.lo);
    }
    if (t < 3) sJ[t] = __ldg(a.J + (int64_t)t * a.n_elem + e);
    nsem_chain_wait();
    if (t < NP) {
        const float* s = a.S + e * 5 * NP + t;
#pragma unroll
        for (int v = 0; v < 5; v++) own[v] = s[v * NP];
        if (has_din) {
            const float* d = a.Din + e * 5 * NP + t;
#pragma unroll
            for (int v = 0; v < 5; v++) own[v] = __fadd_rn(own[v], d[v * NP]);
        }
    }
    if (t < NFS && nb >= 0) {
        const float* s = a.S + (int64_t)nb * 5 * NP + fs.lo;
#pragma unroll
        for (int v = 0; v < 5; v++) oth[v] = s[v * NP];
        if (has_din) {
            const float* d = a.Din + (int64_t)nb * 5 * NP + fs.lo;
#pragma unroll
            for (int v = 0; v < 5; v++) oth[v] = __fadd_rn(oth[v], d[v * NP]);
        }
    }

    if (t < NP) gsm4[GL::at(t)] = prim_ut(own, bgs0, a.T0);
    G::sync();

    if (t < NFS && nb <= -2) {
        /* a face on a 2:1 mortar: the projected values from the mortar kernels */
        const float* gf = a.MF + ((int64_t)(-2 - nb) * MF_ROWS + 5) * a.nfmax + face_local<NX, NY, NZ>(t);
        sD[t] = make_float4(gf[0], gf[a.nfmax], gf[2 * a.nfmax], gf[3 * a.nfmax]);
    } else if (t < NFS) {
        const float4 O = nb >= 0 ? prim_ut(oth, bgo0, a.T0) : make_float4(0, 0, 0, 0);
        sD[t] = cds_minus_own(gsm4[GL::at(fs.la)], nb >= 0 ? &O : nullptr, fs.dir);
    }
    G::sync();

    nsem_chain_begin();
    grad_lines<NX, NY, NZ, true>(gsm4, a, t, sJ);
    G::sync();
    if (t >= NP) return;
    float* out = a.Gout + e * 12 * NP + t;
#pragma unroll
    for (int r = 0; r < 3; r++) {
        const float4 d = r == 1 && !G::HAS_Y ? make_float4(0, 0, 0, 0) : gsm4[GL::w(r) + GL::at(t)];
        out[tidx(r, 0) * NP] = d.x;
        out[tidx(r, 1) * NP] = d.y;
        out[tidx(r, 2) * NP] = d.z;
        out[(9 + r) * NP] = d.w;
    }
}

template <int NX, int NY, int NZ, bool VISC, bool TC>
int launch_stage_v(const StageArgs& a, int stage, cudaStream_t st) {
    const dim3 B = Geo<NX, NY, NZ>::block();
    constexpr size_t SMEM = Geo<NX, NY, NZ>::EPB * StageSmem<NX, NY, NZ, TC>::BYTES;
    const unsigned grid = Geo<NX, NY, NZ>::grid(a.n_elem);
    switch (stage) {
        case 0: return nsem_launch_chained(k_mixed_stage<NX, NY, NZ, 0, VISC, TC>, grid, B, SMEM, st, a.split, a);
        case 1: return nsem_launch_chained(k_mixed_stage<NX, NY, NZ, 1, VISC, TC>, grid, B, SMEM, st, a.split, a);
        case 2: return nsem_launch_chained(k_mixed_stage<NX, NY, NZ, 2, VISC, TC>, grid, B, SMEM, st, a.split, a);
        default: return nsem_launch_chained(k_mixed_stage<NX, NY, NZ, 3, VISC, TC>, grid, B, SMEM, st, a.split, a);
    }
}

/* the tensor-core line sums exist for order 7 only */
template <int NX, int NY, int NZ>
constexpr bool tc_dims() {
    return NX == 8 && NY == 8 && NZ == 8;
}

template <int NX, int NY, int NZ, bool VISC>
int launch_stage_tc(const StageArgs& a, int stage, cudaStream_t st, const LaunchCfg& c) {
    if constexpr (tc_dims<NX, NY, NZ>()) {
        if (c.tc) return launch_stage_v<NX, NY, NZ, VISC, true>(a, stage, st);
    }
    return launch_stage_v<NX, NY, NZ, VISC, false>(a, stage, st);
}

template <int NX, int NY, int NZ>
int launch_stage(const StageArgs& a, int stage, cudaStream_t st, const LaunchCfg& c) {
    return c.visc ? launch_stage_tc<NX, NY, NZ, true>(a, stage, st, c)
                  : launch_stage_tc<NX, NY, NZ, false>(a, stage, st, c);
}

/* viscous runs: the gradients of the stage state, before the stage */
template <int NX, int NY, int NZ>
int launch_grad(const StageArgs& a, int stage, cudaStream_t st) {
    using G = Geo<NX, NY, NZ>;
    const unsigned grid = Geo<NX, NY, NZ>::grid(a.n_elem);
    constexpr size_t gs = G::EPB * GradLay<NX, NY, NZ>::BYTES;
    const dim3 B = G::block();
    return stage <= 1 ? nsem_launch_chained(k_mixed_grad<NX, NY, NZ, 1>, grid, B, gs, st, a.split, a)
                      : nsem_launch_chained(k_mixed_grad<NX, NY, NZ, 2>, grid, B, gs, st, a.split, a);
}

template <int NX, int NY, int NZ, bool VISC, bool TC>
int set_smem(int stage) {
    constexpr int SMEM = (int)StageSmem<NX, NY, NZ, TC>::BYTES;
    if (SMEM <= 48 * 1024) return 0;
    const cudaFuncAttribute at = cudaFuncAttributeMaxDynamicSharedMemorySize;
    switch (stage) {
        case 0: return (int)cudaFuncSetAttribute(k_mixed_stage<NX, NY, NZ, 0, VISC, TC>, at, SMEM);
        case 1: return (int)cudaFuncSetAttribute(k_mixed_stage<NX, NY, NZ, 1, VISC, TC>, at, SMEM);
        case 2: return (int)cudaFuncSetAttribute(k_mixed_stage<NX, NY, NZ, 2, VISC, TC>, at, SMEM);
        default: return (int)cudaFuncSetAttribute(k_mixed_stage<NX, NY, NZ, 3, VISC, TC>, at, SMEM);
    }
}

template <int NX, int NY, int NZ>
int prepare_stage() {
    int e = 0;
    for (int st = 0; st < 4 && !e; st++) {
        e = set_smem<NX, NY, NZ, false, false>(st);
        if (!e) e = set_smem<NX, NY, NZ, true, false>(st);
        if constexpr (tc_dims<NX, NY, NZ>()) {
            if (!e) e = set_smem<NX, NY, NZ, false, true>(st);
            if (!e) e = set_smem<NX, NY, NZ, true, true>(st);
        }
    }
    constexpr size_t gs = GradLay<NX, NY, NZ>::BYTES;
    const cudaFuncAttribute at = cudaFuncAttributeMaxDynamicSharedMemorySize;
    if (!e && gs > 48 * 1024) {
        e = (int)cudaFuncSetAttribute(k_mixed_grad<NX, NY, NZ, 1>, at, (int)gs);
        if (!e) e = (int)cudaFuncSetAttribute(k_mixed_grad<NX, NY, NZ, 2>, at, (int)gs);
    }
    return e;
}

template <int NX, int NY, int NZ, bool VISC>
int chain_split(int64_t n_elem) {
    using G = Geo<NX, NY, NZ>;
    if (NX == 4 && !VISC) return 0;   /* order 3, the driver's choice: 267 us, 275 with one split */
    return nsem_chain_split(MIXED_SPLIT, k_mixed_stage<NX, NY, NZ, 1, VISC, false>, G::grid(n_elem), G::block(),
                            G::EPB * StageSmem<NX, NY, NZ>::BYTES);
}

}  // namespace

namespace nsem_mx {

int split_aligned(int nx, int ny, int nz, int64_t n_elem, bool visc) {
#define NSEM_SPLIT_OF(A, B, C)           \
    if (nx == A && ny == B && nz == C)   \
        return visc ? chain_split<A, B, C, true>(n_elem) : chain_split<A, B, C, false>(n_elem);
    NSEM_MIXED_DIMS(NSEM_SPLIT_OF)
#undef NSEM_SPLIT_OF
    return 0;
}

int prepare_aligned(int nx, int ny, int nz) {
#define NSEM_PREP(A, B, C) if (nx == A && ny == B && nz == C) return prepare_stage<A, B, C>();
    NSEM_MIXED_DIMS(NSEM_PREP)
#undef NSEM_PREP
    return (int)cudaErrorNotSupported;
}

int launch_stage_aligned(int nx, int ny, int nz, const StageArgs& a, int stage, cudaStream_t st,
                         const LaunchCfg& c) {
#define NSEM_DISP(A, B, C) \
    if (nx == A && ny == B && nz == C) return launch_stage<A, B, C>(a, stage, st, c);
    NSEM_MIXED_DIMS(NSEM_DISP)
#undef NSEM_DISP
    return (int)cudaErrorNotSupported;
}

int launch_grad_aligned(int nx, int ny, int nz, const StageArgs& a, int stage, cudaStream_t st) {
#define NSEM_DISPG(A, B, C) \
    if (nx == A && ny == B && nz == C) return launch_grad<A, B, C>(a, stage, st);
    NSEM_MIXED_DIMS(NSEM_DISPG)
#undef NSEM_DISPG
    return (int)cudaErrorNotSupported;
}

}  // namespace nsem_mx
