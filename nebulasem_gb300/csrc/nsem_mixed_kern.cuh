/*
 * Precision form: the stage kernels' arguments and the layouts and device
 * helpers shared by its translation units -- nsem_mixed.cu (setup, mortar and
 * layout kernels, launches), nsem_mixed_stage.cu (axis-aligned affine
 * elements) and nsem_mixed_gen.cu (inclined and curved elements).
 */
#ifndef NSEM_MIXED_KERN_CUH
#define NSEM_MIXED_KERN_CUH

#include <cuda_runtime.h>

#include <cstdint>

#include "nsem_mixed.h"
#include "nsem_mixed_dev.cuh"

namespace nsem_mx {

struct StageArgs {
    const double* U;           /* u'^n (FP64), [e][5][NP]                  */
    const float* S;            /* stage base state: FP32 shadow of u'^n    */
    const float* Din;          /* previous stage increment (or null)      */
    float* Dout;               /* stage increment out (stages 1, 2)       */
    double* Unew;              /* u'^{n+1} (stage 3)                      */
    float* Snew;               /* its FP32 shadow (stage 3)               */
    double* L[5];              /* tendency out (stage 0), node order      */
    const int32_t* nbr;        /* [6][n_elem]                             */
    const float* J;            /* [3][n_elem]                             */
    const int32_t* layer;      /* [n_elem]                                */
    const float* Qg;           /* line-sum weights                        */
    const float* G;            /* viscous runs: [e][12][NP] gradients      */
    float* Gout;               /* gradient kernel output                   */
    const float* bg;           /* [layers][4][NP]                          */
    const float4* bgp;         /* [layers][NP + NFS]: nodes, across face slots */
    const float* Jg;           /* general geometry: [e][10][NP] Jinv cV (9), 1/cV */
    const float* Fn;           /* general geometry: [e][3][NFS] outward weighted normals */
    const float* MF;           /* mortar faces: [n_mf][9][nfmax] outward face values (0-4),
                                  viscous runs' gradient face terms (5-8) */
    int nfmax;
    int64_t n_elem;
    float dt, gamma, gR, g[3];
    float nu, nu_pr, T0;
    float lift[3];             /* 1 / w_end per direction                  */
    float eos[6];              /* binomial coefficients C(gamma, k), k = 1..6 */
    uint32_t* status;
    int split;                 /* shared-memory split of the launches */
    /* line-sum weights Q_d[a][m] (gradient kernels: the derivative tables
     * D_d[a][m]) as kernel parameters: read with compile-time indices they
     * are constant-bank operands of the FMAs (several to a load when aligned:
     * 24^3 elements of order 4, 40 steps: 6980 us, 7014 eight bytes off) */
    alignas(16) float qc[3][8][8];
};

/* rows per element face of the mortar face buffer: the 5 outward values,
 * then the gradient face terms: 4 (cds - own, axis-aligned elements) or
 * 12 (fN_out[r] (cds - own)_c, general geometry) */
constexpr int MF_ROWS = 9, MF_ROWS_GEN = 17;

/* tensor-core flux layout (order 7): a variable's fluxes of one direction
 * F[a][m][b] -- m the node index along the direction, (a, b) the other two
 * (x: (j, k), y: (i, k), z: (i, j)) -- at a * TC_SA + p(m) * 8 + (b ^ s(m)),
 * p(m) = m ^ (m >> 2 & 1), s(m) = 4 (m >> 2 & 1).  TC_SA = 72 puts four
 * consecutive a in distinct groups of 8 banks; p keeps the rows m = 0-3,
 * 4-7, the even and the odd rows each in four distinct groups; s separates
 * the rows that share a group.  Every access is then conflict-free: the
 * node threads' stores and reads in all three directions (a warp holds one i,
 * four j and eight k), the face threads' reads, the A-fragment loads (rows
 * m = tg, tg + 4) and the in-place result stores (rows 2 tg, 2 tg + 1). */
constexpr int TC_SA = 72;
constexpr int TC_NP = 8 * TC_SA;
constexpr int TC_QTAB = 3 * 2 * 64;   /* B fragments per direction: high, low; [k][n] */

/* the in-place line transform of the stage kernels (layout: LineLay) */
template <int NX, int NY, int NZ, int D>
__device__ __forceinline__ void line_transform(float* F, const StageArgs& a, int t) {
    using LL = LineLay<NX, NY, NZ, D>;
    constexpr int BLOCK = Geo<NX, NY, NZ>::BLOCK;
    float* f = F + LL::BASE;
#pragma unroll 1
    for (int r = t; r < 5 * LL::NL; r += BLOCK) {
        float in[LL::n];
#pragma unroll
        for (int m = 0; m < LL::n; m++) in[m] = f[m * LL::ROW + r];
#pragma unroll
        for (int q = 0; q < LL::n; q++) {
            float acc = 0.0f;
#pragma unroll
            for (int m = 0; m < LL::n; m++) acc = fmaf(a.qc[D][q][m], in[m], acc);
            f[q * LL::ROW + r] = acc;
        }
    }
}

/* index of face slot t within its face: x (j, k), y (i, k), z (i, j) */
template <int NX, int NY, int NZ>
__device__ __forceinline__ int face_local(int t) {
    using G = Geo<NX, NY, NZ>;
    if (t < G::OFF_Y) return t % G::NFX;
    if (t < G::OFF_Z) return (t - G::OFF_Y) % G::NFY;
    return (t - G::OFF_Z) % G::NFZ;
}

/* The gradient kernels' shared memory, in float4 (U, theta - T0): the nodes'
 * values V, the face terms cds - own, and per direction the derivatives at
 * the nodes.  Rows of nodes along z have an odd pitch: a quarter warp's
 * 16-byte accesses down z lines are then conflict-free at even node counts. */
template <int NX, int NY, int NZ>
struct GradLay {
    using G = Geo<NX, NY, NZ>;
    static constexpr int PZ = NZ | 1;
    static constexpr int NV = NX * NY * PZ;
    static constexpr int OFF_D = NV;
    static constexpr int OFF_W = OFF_D + G::NFS;
    static constexpr size_t BYTES = sizeof(float4) * (OFF_W + (G::HAS_Y ? 3 : 2) * NV);
    /* first position of direction D's derivatives */
    __host__ __device__ static constexpr int w(int D) { return OFF_W + (D == 0 ? 0 : D == 1 ? NV : (G::HAS_Y ? 2 : 1) * NV); }
    __device__ static __forceinline__ int at(int i, int j, int k) { return (i * NY + j) * PZ + k; }
    /* node t of the element's own numbering */
    __device__ static __forceinline__ int at(int t) { return NZ == PZ ? t : t / NZ * PZ + t % NZ; }
};

/* derivatives along line l of direction D: W_a = sum_m D_D[a][m] V_m.  With
 * ALIGNED the metric and the face terms at the line's two ends join here:
 * J_D W_a - / + (J_D / w_end) (cds - own). */
template <int NX, int NY, int NZ, int D, bool ALIGNED>
__device__ __forceinline__ void grad_line(float4* sm, const StageArgs& a, int l, float Jd) {
    using G = Geo<NX, NY, NZ>;
    using L = GradLay<NX, NY, NZ>;
    constexpr int n = D == 0 ? NX : D == 1 ? NY : NZ;
    constexpr int STEP = D == 0 ? NY * L::PZ : D == 1 ? L::PZ : 1;
    constexpr int OFF = D == 0 ? G::OFF_X : D == 1 ? G::OFF_Y : G::OFF_Z;
    constexpr int NF = D == 0 ? G::NFX : D == 1 ? G::NFY : G::NFZ;
    /* lines in the order of the face's nodes: x (j, k), y (i, k), z (i, j) */
    const int n0 = D == 0 ? L::at(0, l / NZ, l % NZ) : D == 1 ? L::at(l / NZ, 0, l % NZ) : l * L::PZ;
    float4 in[n];
#pragma unroll
    for (int m = 0; m < n; m++) in[m] = sm[n0 + m * STEP];
#pragma unroll
    for (int q = 0; q < n; q++) {
        float4 acc = make_float4(0, 0, 0, 0);
#pragma unroll
        for (int m = 0; m < n; m++) {
            const float d = a.qc[D][q][m];
            acc.x = __fmaf_rn(d, in[m].x, acc.x); acc.y = __fmaf_rn(d, in[m].y, acc.y);
            acc.z = __fmaf_rn(d, in[m].z, acc.z); acc.w = __fmaf_rn(d, in[m].w, acc.w);
        }
        if constexpr (ALIGNED) {
            acc.x = __fmul_rn(acc.x, Jd); acc.y = __fmul_rn(acc.y, Jd);
            acc.z = __fmul_rn(acc.z, Jd); acc.w = __fmul_rn(acc.w, Jd);
            if (q == 0 || q == n - 1) {
                const float c = __fmul_rn(Jd, a.lift[D]);
                const float coef = q == 0 ? -c : c;
                const float4 f = sm[L::OFF_D + OFF + (q == 0 ? 0 : NF) + l];
                acc.x = __fmaf_rn(coef, f.x, acc.x); acc.y = __fmaf_rn(coef, f.y, acc.y);
                acc.z = __fmaf_rn(coef, f.z, acc.z); acc.w = __fmaf_rn(coef, f.w, acc.w);
            }
        }
        sm[L::w(D) + n0 + q * STEP] = acc;
    }
}

/* all lines of the element, one per thread, each direction's in warps of its
 * own.  The kernels are bound by shared-memory wavefronts: a line's values are
 * read once and shared by its sums, 10 float4 accesses per line of 5 nodes
 * where a thread per node makes 25 and 25 table reads (viscous step with its
 * stage kernels, 9240 elements of order 4, 20 steps: 4960 us against 5185;
 * 1716 of order 7: 3650 against 3884; 400 in 2D, order 3, 40 steps: 632
 * against 849; with the full metric 7280 against 7486, order 3 alone 1.5 %
 * slower, 3708 against 3652) */
template <int NX, int NY, int NZ, bool ALIGNED>
__device__ __forceinline__ void grad_lines(float4* sm, const StageArgs& a, int t, const float* sJ) {
    using G = Geo<NX, NY, NZ>;
    constexpr int WX = (G::NFX + 31) / 32 * 32, WY = G::HAS_Y ? (G::NFY + 31) / 32 * 32 : 0,
                  WZ = (G::NFZ + 31) / 32 * 32;
    for (int r = t; r < WX + WY + WZ; r += G::BLOCK) {
        if (r < WX) {
            if (r < G::NFX) grad_line<NX, NY, NZ, 0, ALIGNED>(sm, a, r, ALIGNED ? sJ[0] : 1.0f);
        } else if (r < WX + WY) {
            if constexpr (G::HAS_Y) {
                if (r - WX < G::NFY) grad_line<NX, NY, NZ, 1, ALIGNED>(sm, a, r - WX, ALIGNED ? sJ[1] : 1.0f);
            }
        } else if (r - WX - WY < G::NFZ) {
            grad_line<NX, NY, NZ, 2, ALIGNED>(sm, a, r - WX - WY, ALIGNED ? sJ[2] : 1.0f);
        }
    }
}

/* u'^{n+1} = u'^n + D and its FP32 shadow at position o of the element-blocked
 * arrays (stage 3): conversions for values in range, and once more with every
 * case where one is not.  The kernel is bound by issue, and the general
 * conversions were an eighth of its instructions (24^3 elements of order 4, 40
 * steps: 6979 to 6916 us; 693 elements 628 to 603; 4096 in 2D, 50 steps: 784
 * to 719; with the hardware's float-to-double conversion, which runs on the
 * FP64 pipe, 6950, 626 and 779) */
template <int NP, bool LOADED>
__device__ __forceinline__ void update_state(const StageArgs& a, int64_t o, const float* Lv, float* D,
                                             double* un) {
    /* LOADED: D and un hold the increment d2 and u'^n already */
    if constexpr (!LOADED) {
        /* every load before the first store, which could alias them */
#pragma unroll
        for (int v = 0; v < 5; v++) {
            D[v] = a.Din[o + v * NP];
            un[v] = a.U[o + v * NP];
        }
    }
    bool ok = true;
#pragma unroll
    for (int v = 0; v < 5; v++) {
        D[v] = (2.0f / 3.0f) * fmaf(a.dt, Lv[v], D[v]);
        ok = ok && (__float_as_uint(D[v]) & 0x7f800000u) != 0x7f800000u;
        un[v] += f2d_finite(D[v]);
        ok = ok && in_float_range(un[v]);
    }
    if (ok) {
#pragma unroll
        for (int v = 0; v < 5; v++) {
            a.Unew[o + v * NP] = un[v];
            a.Snew[o + v * NP] = d2f_in_range(un[v]);
        }
        return;
    }
    bool finite = true;
    double u[5];
    for (int v = 0; v < 5; v++) u[v] = a.U[o + v * NP];
    for (int v = 0; v < 5; v++) {
        const double x = u[v] + f2d(D[v]);
        a.Unew[o + v * NP] = x;
        a.Snew[o + v * NP] = d2f_rn(x);
        /* exponent field all ones = inf or nan (integer test, no FP64 op) */
        finite = finite && ((__double2hiint(x) & 0x7ff00000) != 0x7ff00000);
    }
    if (!finite) atomicOr(a.status, NSEM_STATUS_NONFINITE);
}

struct LaunchCfg {
    bool visc, tc, gen;
};

/* per translation unit: the kernels' shared-memory attributes, the stage
 * launches and the gradient launches of viscous runs, each dispatched on the
 * node counts per direction */
int prepare_aligned(int nx, int ny, int nz);
int prepare_general(int nx, int ny, int nz);
/* the shared-memory split of the stage (and gradient) launches (NSEM_SPLIT
 * explains it): what the stage kernels' resident CTAs fill.  20 steps of 693
 * elements: order 4 384 to 370 us, tilted 409 to 394, order 3 viscous 460 to
 * 425; 30 of 1600 in 2D, tilted 425 to 376; at 72 viscous runs of order 4 lose
 * 2 % */
constexpr int MIXED_SPLIT = 58;
int split_aligned(int nx, int ny, int nz, int64_t n_elem, bool visc);
int split_general(int nx, int ny, int nz, int64_t n_elem, bool visc);
int launch_stage_aligned(int nx, int ny, int nz, const StageArgs& a, int stage, cudaStream_t st,
                         const LaunchCfg& c);
int launch_stage_general(int nx, int ny, int nz, const StageArgs& a, int stage, cudaStream_t st,
                         bool visc);
int launch_grad_aligned(int nx, int ny, int nz, const StageArgs& a, int stage, cudaStream_t st);
int launch_grad_general(int nx, int ny, int nz, const StageArgs& a, int stage, cudaStream_t st);

}  // namespace nsem_mx

#endif
