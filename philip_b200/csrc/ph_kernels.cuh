// sm_100a kernels of the GLL-collocated strong-form DG/FR residual, the auxiliary
// (lifted-gradient) equation and the fused Runge-Kutta stage epilogue.
//
// Work decomposition. A CTA owns a tile of CPC cells. Every phase is a loop over
// work items with a fixed owner, so all accumulation happens in a fixed order and
// repeated runs are bitwise identical (no atomics on data):
//   1. gather the neighbour face traces (state, and the auxiliary gradient when viscous)
//   2. per node: FP64 positivity check, node quantities (rho, v, p, logs), viscous flux
//   3. per face node: numerical flux at the canonical orientation (left cell = int,
//      normal +e_d), lifted into this cell with the sign of its face
//   4. per direction: one warp segment of N1 lanes owns one 1-D line; each lane
//      evaluates the two-point flux with partner (pos+k) mod N1 and hands it to the
//      partner through a warp shuffle, so each unordered pair is evaluated once
//   5. per node: mass inverse (diagonal for cDG, B(x)B(x)B for FR) and the RK update
//
// Reference structure restated (GLL collocation makes chi = I and the entropy
// projection the identity, and the hybrid surface-volume terms cancel exactly):
//   volume split form ............ src/dg/strong_dg.cpp:1235-1543
//   face term ..................... src/dg/strong_dg.cpp:2367-3576
//   auxiliary equation ............ src/dg/strong_dg.cpp:498-1008
//   inverse mass (affine) ......... src/dg/dg_base.cpp:4207-4219
//   RK stage / sum ................ src/ode_solver/runge_kutta_ode_solver.cpp:15-100
#pragma once
#include <type_traits>

#include "ph_physics.cuh"

// resident CTAs per SM asked of the compiler (register budget) for the p = 3 and p = 5
// stage tiles, FP64 and FP32 (measured choices; see the Layout)
#ifndef PH_P5_MINB
#define PH_P5_MINB 3
#endif
#ifndef PH_P5_MINB_F32
#define PH_P5_MINB_F32 6
#endif
#ifndef PH_P3_MINB
#define PH_P3_MINB 6
#endif
#ifndef PH_P3_MINB_F32
#define PH_P3_MINB_F32 10
#endif
// 1: the pair fluxes between opposite nodes of a line (offset N1/2, even N1), which both lanes of
// the pair would evaluate, are computed once per pair in a pass of their own and read back by
// both nodes' lanes. Off: on B200 the extra shared memory costs more than the saved pair fluxes
// (24^3 p5 FP64 stage 0.505 ms against 0.494, 32^3 p3 0.425 against 0.396: one CTA per SM fewer)
#ifndef PH_PAIR_DEDUP
#define PH_PAIR_DEDUP 0
#endif
// 1: at p = 5 the volume phase accumulates each direction into an array of its own (the first
// in the state's space, two more after the layout), so the three directions run without a block
// barrier between them and without read-modify-write of the accumulator; phase 5 sums them in
// the order of the shared accumulator (bitwise the same). Only where the extra shared memory
// still fits the CTAs per SM the register budget allows. Off: on B200 at 24^3 p5 the stage
// kernel takes 0.509 ms against 0.492 in FP64 and 0.307 against 0.268 in FP32.
#ifndef PH_SEP_ACC
#define PH_SEP_ACC 0
#endif
// 1: the FP64 viscous stage kernel (even N1, affine cells) stages its tile's state and viscous
// divergence into shared memory with bulk copies (cp.async.bulk, completion on an mbarrier),
// issued before the neighbour gathers (B200: 24^3 p5 0.499 ms against 0.505, 32^3 p3 0.421
// against 0.425; the L2-resident 8^3 p3 inviscid case is 5 % slower with it, so only viscous)
#ifndef PH_BULK_TILE
#define PH_BULK_TILE 1
#endif

namespace ph {

constexpr int MAXN1 = 8;

// 1-D operator tables on the GLL nodes (double, row-major [a][l]).
struct OpTab {
    double D[MAXN1 * MAXN1];      // D[a][l] = l_l'(x_a)
    double Dsk[MAXN1 * MAXN1];    // (w_a D[a][l] - w_l D[l][a]) / w_a
    double B[MAXN1 * MAXN1];      // (M+K)^{-1} diag(w)  (FR mass inverse in G units)
    double Minv[MAXN1 * MAXN1];   // (M+K)^{-1}
    double w[MAXN1];              // GLL weights on [0,1]
    double Baux[MAXN1 * MAXN1];   // (M+K_aux)^{-1} diag(w), the auxiliary equation's FR mass inverse
    int aux_fr;                   // K_aux != 0: the auxiliary kernel applies Baux(x)Baux(x)Baux
};

struct StageArgs {
    const double* U;          // stage input state [nc][5][NP]
    const void* Fv;           // viscous terms from the auxiliary kernel, viscous_terms_per_cell<N1>() per
                              // cell, stored in the arithmetic type R (FP32 in the precision form)
    const int* nbr;           // [nc][6] neighbour cell per face
    const OpTab* ops;
    int nc;                   // one past the last cell of this launch
    int cell_begin;           // first cell of this launch (a multiple of the cells per tile)
    double h, inv_h;
    double pen;               // SIPG penalty p(p+1)/h * factor
    PhysConst pc;
    unsigned* status;
    int mode;                 // 0: R (before M^-1), 1: k = M^-1 R, 2: RK stage
    int fr;                   // apply the FR mass inverse B(x)B(x)B
    double* out;              // modes 0,1
    // RK stage epilogue (mode 2), all arrays in the state layout
    const double* Un;         // u_n
    const double* acc_in;     // running sum (nullptr on the first stage)
    double* acc_out;          // acc_in (or base) + c_acc * k
    double c_acc;
    int inc_mode;             // acc holds the increment sum (precision form) instead of u_n + sum
    double* comp;             // Kahan compensation of the final sum (precision form), or nullptr
    double* final_out;        // last stage: u_{n+1}
    double* next;             // next stage state: ((carry_in) + a_next k) dt + u_n
    const double* carry_in;
    double a_next;
    double* carry_out;        // a_carry * k for the stage after next
    double a_carry;
    double dt;
    // curvilinear cells: [nc][10][NP], rows k*3+d = metric cofactor C[k][d] at the
    // volume nodes, row 9 = 1 / det J (nullptr on affine meshes)
    const double* metric;
    // low-storage 3S* / 3S*+ stage (mode 3): S1 = the stage input U, S2 and S4 updated in
    // place, S3 = u_n, S1 of the next stage written to ls_s1_out
    double* ls_s2;
    const double* ls_s3;
    double* ls_s4;              // 3S*+ error register (nullptr for 3S*)
    double* ls_s1_out;          // nullptr on the FSAL evaluation
    double ls_g0, ls_g1, ls_g2, ls_beta, ls_delta, ls_bhat;
    int ls_first;               // stage 0: S2 starts at 0, S4 at u_n
    int ls_embedded;            // last 3S* stage: S2 = (S2 + d_s S1 + d_s1 S3) / sum(delta)
    double ls_delta_s, ls_delta_s1, ls_inv_sum_delta;
    double* err_partial;        // per-tile sums of the squared scaled error (or nullptr)
    double atol, rtol;
    // relaxation RK (mode 2): per-tile sums of v(u)^T M k, v the entropy variables of the
    // stage input (or nullptr; the generic flux-set kernel, FS = 0, computes them)
    double* ent_partial;
    // non-periodic meshes: a boundary face has nbr = -1 - k, btype[k] its boundary_id, and (Navier-
    // Stokes) Fb[k] the outward boundary viscous flux F*_v . n at its [4][NF] face nodes, in R,
    // written by the auxiliary kernel (nullptr on periodic meshes)
    const int* btype;
    const void* Fb;
    // optional tile list: CTA b works on the tile whose first cell is tiles[b] (ntiles CTAs); the
    // boundary-face kernels run on the tiles that touch a boundary, the periodic ones on the rest
    const int* tiles;
    int ntiles;
};

// Viscous terms per cell written by the auxiliary kernel and read by the stage kernel:
// [4][NP] the volume divergence sum_d D_d F_v,d of the momentum and energy rows, then
// [6 faces][4][NF] the face-normal viscous flux F_v,d(f) at each face's nodes (a cell reads
// its neighbour's block of the opposite face, whose nodes come in the same order).
template <int N1> __host__ __device__ constexpr int viscous_terms_per_cell() {
    return 4 * N1 * N1 * N1 + 24 * N1 * N1;
}

// CURV: curvilinear cells (split form, Euler or Navier-Stokes): the per-node metric cofactor
// (9 values) in sX, after the viscous rows.
template <typename R, int N1, int CPC, bool VISC, bool SPLIT, bool CURV = false>
struct Layout {
    static constexpr int NP = N1 * N1 * N1, NF = N1 * N1;
    static constexpr int NQV = 10;                     // rho v0 v1 v2 p E a b la lb vsq -> packed 11
    static constexpr int NQS = 11;
    static constexpr int TR = VISC ? 9 : 5;            // trace values per face node: u (5) [+ ext viscous flux (4)]
    static constexpr int NX = (VISC ? 4 : 0) + (SPLIT ? 0 : 15) + (CURV ? 9 : 0);
    static constexpr int OM = (VISC ? 4 : 0) + (SPLIT ? 0 : 15);   // curvilinear: first metric row of X
    static constexpr int oOps = 0;                      // D, Dsk, B, w as R
    static constexpr int nOps = 3 * N1 * N1 + N1;
    static constexpr int oU = (oOps + nOps + 1) & ~1;
    static constexpr int oD = oU + CPC * 5 * NP;
    static constexpr int oT = oD + CPC * NQS * NP;
    // the volume accumulator reuses the state's space: the state is read last by the face phase
    static constexpr int oA = oU;
    static constexpr int oX = oT + CPC * 6 * TR * NF;
    // opposite-node pair fluxes: [direction][cell][line][pair][5] (split form on affine cells,
    // even N1; in the frame of the line's direction)
    static constexpr int HP = (PH_PAIR_DEDUP && SPLIT && !CURV && (N1 % 2 == 0)) ? N1 / 2 : 0;
    static constexpr int oH = oX + CPC * NX * NP;
    static constexpr int oA1 = oH + 3 * CPC * NF * HP * 5;   // directions 1 and 2 (SEPA)
    static constexpr int SPW = 32 / N1;                // lines per warp
    static constexpr int WARPS_LINES = (CPC * NF + SPW - 1) / SPW;
    static constexpr int NT = WARPS_LINES * 32;
    // register budgets from timing the stage kernel on B200: p = 5 (one cell, 256 threads
    // per CTA) 3 CTAs per SM in FP64 (the unrolled partner loop needs 80 registers; at 4 CTAs
    // it spills and takes 0.533 ms against 0.496), 6 in FP32 (3-4 % faster than 4);
    // p = 3 (two cells, 128 threads) 6 in FP64 and 10 in FP32 (3 % faster than 8)
    static constexpr bool F32 = sizeof(R) == 4;
    static constexpr int MINB_ASKED = (N1 == 6) ? (F32 ? PH_P5_MINB_F32 : PH_P5_MINB)
                                    : (N1 == 4) ? (F32 ? PH_P3_MINB_F32 : PH_P3_MINB) : 1;
    // never more CTAs than 2048 threads per SM hold (the batched tile shapes are wider)
    static constexpr int MINB = MINB_ASKED * NT > 2048 ? 2048 / NT : MINB_ASKED;
    // separate direction accumulators where MINB CTAs (1 KB reserved each) still fit 228 KB
    static constexpr bool SEPA = PH_SEP_ACC && N1 == 6 &&
                                 (size_t)MINB * ((oA1 + 2 * CPC * 5 * NP) * sizeof(R) + 1024) <= 233472;
    static constexpr int total = oA1 + (SEPA ? 2 * CPC * 5 * NP : 0);
    static constexpr size_t bytes = (size_t)total * sizeof(R);
};

template <int N1> __device__ __forceinline__ int node_of(int x, int y, int z) { return (z * N1 + y) * N1 + x; }

// ---- bulk copies global -> shared with mbarrier completion (this CTA's own shared memory, no
// multicast). Sizes and both addresses are multiples of 16 bytes.
__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_copy_g2s(void* dst, const void* src, unsigned bytes, unsigned long long* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_addr(dst)), "l"(src), "r"(bytes), "r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, unsigned parity) {
    unsigned ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                 : "=r"(ok) : "r"(smem_addr(bar)), "r"(parity) : "memory");
    return ok != 0;
}
// Bounded wait on phase `parity`: true when the phase completed within `limit` polls.
__device__ __forceinline__ bool mbar_wait_bounded(unsigned long long* bar, unsigned parity, long long limit) {
    for (long long i = 0; i < limit; ++i)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}

// coordinates of face node `fn` of face f at boundary coordinate b
template <int N1> __device__ __forceinline__ int face_node_volume_index(int f, int fn, int b) {
    const int dn = f >> 1;
    int c[3];
    const int t1 = (dn == 0) ? 1 : 0, t2 = (dn == 2) ? 1 : 2;
    c[dn] = b; c[t1] = fn % N1; c[t2] = fn / N1;
    return node_of<N1>(c[0], c[1], c[2]);
}

template <typename R>
__device__ __forceinline__ void store_q(R* sD, int NP, int idx, const NodeQ<R>& q) {
    sD[0 * NP + idx] = q.rho; sD[1 * NP + idx] = q.v[0]; sD[2 * NP + idx] = q.v[1]; sD[3 * NP + idx] = q.v[2];
    sD[4 * NP + idx] = q.p; sD[5 * NP + idx] = q.E; sD[6 * NP + idx] = q.a; sD[7 * NP + idx] = q.b;
    sD[8 * NP + idx] = q.la; sD[9 * NP + idx] = q.lb; sD[10 * NP + idx] = q.vsq;
}
// Node quantities with the velocity expressed in the frame (e_d, e_{d+1}, e_{d+2}):
// every flux along direction d is then evaluated by the x-direction code.
template <typename R>
__device__ __forceinline__ void load_q_rot(const R* sD, int NP, int idx, int d, NodeQ<R>& q) {
    const int d1 = (d + 1) % 3, d2 = (d + 2) % 3;
    q.rho = sD[0 * NP + idx]; q.v[0] = sD[(1 + d) * NP + idx]; q.v[1] = sD[(1 + d1) * NP + idx];
    q.v[2] = sD[(1 + d2) * NP + idx];
    q.p = sD[4 * NP + idx]; q.E = sD[5 * NP + idx]; q.a = sD[6 * NP + idx]; q.b = sD[7 * NP + idx];
    q.la = sD[8 * NP + idx]; q.lb = sD[9 * NP + idx]; q.vsq = sD[10 * NP + idx];
}
template <typename R>
__device__ __forceinline__ void rotate_state(const R u[5], int d, R r[5]) {
    r[0] = u[0]; r[1] = u[1 + d]; r[2] = u[1 + (d + 1) % 3]; r[3] = u[1 + (d + 2) % 3]; r[4] = u[4];
}
// back from the rotated frame: F (rotated components) -> out (x, y, z components)
template <typename R>
__device__ __forceinline__ void unrotate_flux(const R F[5], int d, R out[5]) {
    out[0] = F[0]; out[4] = F[4];
    out[1 + d] = F[1]; out[1 + (d + 1) % 3] = F[2]; out[1 + (d + 2) % 3] = F[3];
}

template <typename R>
__device__ __forceinline__ void load_q(const R* sD, int NP, int idx, NodeQ<R>& q) {
    q.rho = sD[0 * NP + idx]; q.v[0] = sD[1 * NP + idx]; q.v[1] = sD[2 * NP + idx]; q.v[2] = sD[3 * NP + idx];
    q.p = sD[4 * NP + idx]; q.E = sD[5 * NP + idx]; q.a = sD[6 * NP + idx]; q.b = sD[7 * NP + idx];
    q.la = sD[8 * NP + idx]; q.lb = sD[9 * NP + idx]; q.vsq = sD[10 * NP + idx];
}

// FP64 positivity check of a stored state (the check stays in FP64 for the precision form).
__device__ __forceinline__ void check_state_fp64(double u[5], double gm1, unsigned* st) {
    double v2 = 0.0;
#pragma unroll
    for (int d = 0; d < 3; ++d) { const double v = u[1 + d] / u[0]; v2 = v2 + v * v; }
    const double p = gm1 * (u[4] - 0.5 * u[0] * v2);
    if (u[0] < 0.0 || p < 0.0) atomicOr(st, ST_NONPHYSICAL);
}

// One face node of phase 3: the numerical flux at the canonical orientation (the
// left cell is the interior side, normal +e_d) lifted into this cell with its sign.
// The convective flux is evaluated in the frame whose x axis is the face normal.
// fvface: this cell's face blocks of the viscous terms (viscous only).
// BND (non-periodic meshes): on a boundary face (bnd) the trace holds the convective boundary state
// and, Navier-Stokes, the boundary viscous flux F*_v . e_d itself (no average, no penalty term).
template <typename R, int N1, int CPC, bool VISC, bool SPLIT, bool CURV, bool BND = false>
__device__ __forceinline__ void face_item(const Cst<R>& cst, int tp, int cf, int df, int ucv, const R* sU,
                                          const R* sD, R* sT, const R* sX, int c, int f, int fn, R pen,
                                          R inv_wend, const R* __restrict__ fvface, bool bnd = false) {
    using L = Layout<R, N1, CPC, VISC, SPLIT, CURV>;
    constexpr int NP = L::NP, NF = L::NF, TR = L::TR, NQS = L::NQS;
    const int d = f >> 1;
    const bool plus = (f & 1);                    // this cell is the left (minus) side
    const R sgn = plus ? R(1) : R(-1);
    const int node = face_node_volume_index<N1>(f, fn, plus ? N1 - 1 : 0);
    R* tr = sT + (c * 6 + f) * TR * NF;
    R uo[5], ue[5];
#pragma unroll
    for (int s = 0; s < 5; ++s) { uo[s] = sU[(c * 5 + s) * NP + node]; ue[s] = tr[s * NF + fn]; }
    if constexpr (CURV) {
        // normal metric C[:, d] at this face node: the canonical normal (from the left cell
        // into the right one) is the same vector seen from either side; |C n| scales the flux
        const R* X = sX + c * L::NX * NP;
        constexpr int OM = L::OM;
        const R m[3] = {X[(OM + 0 * 3 + d) * NP + node], X[(OM + 1 * 3 + d) * NP + node],
                        X[(OM + 2 * 3 + d) * NP + node]};
        const R J = rsqrt_<R>(m[0] * m[0] + m[1] * m[1] + m[2] * m[2]);
        const R nrm[3] = {qdiv<R>(m[0], J), qdiv<R>(m[1], J), qdiv<R>(m[2], J)};
        NodeQ<R> qo, qe;
        load_q<R>(sD + c * NQS * NP, NP, node, qo);
        node_prepare<R, LOG_STORED, N1 % 2 == 0>(ue, tp, cst.gm1, qe, nullptr);
        R F[5];
        if (plus) conv_num_flux_n<R>(uo, ue, qo, qe, nrm, tp, cf, cst, F);
        else conv_num_flux_n<R>(ue, uo, qe, qo, nrm, tp, cf, cst, F);
        R term[5];
#pragma unroll
        for (int s = 0; s < 5; ++s) term[s] = -sgn * J * F[s];
        if constexpr (!SPLIT) {   // the cell's own contravariant flux F . C[:, d] at the face node
            constexpr int o = VISC ? 4 : 0;
#pragma unroll
            for (int s = 0; s < 5; ++s) term[s] += sgn * X[(o + d * 5 + s) * NP + node];
        }
        if constexpr (VISC) {
            // the metric-scaled normal viscous flux F~_d = sum_k C[k][d] F_k of both sides (the
            // auxiliary kernels' face blocks; BR2 / central: their average, strong_dg.cpp:3354-3452)
#pragma unroll
            for (int k = 0; k < 4; ++k) {   // (a boundary face: the trace holds the boundary flux itself)
                const R Fo = __ldg(&fvface[(f * 4 + k) * NF + fn]);
                const R Fn = (BND && bnd) ? tr[(5 + k) * NF + fn] : R(0.5) * (Fo + tr[(5 + k) * NF + fn]);
                term[1 + k] += sgn * (Fo - Fn);
            }
        }
#pragma unroll
        for (int s = 0; s < 5; ++s) tr[s * NF + fn] = term[s] * inv_wend;
        return;
    }
    R ro[5], re[5];
    rotate_state<R>(uo, d, ro);
    rotate_state<R>(ue, d, re);
    NodeQ<R> qo, qe;
    load_q_rot<R>(sD + c * NQS * NP, NP, node, d, qo);
    node_prepare<R, LOG_STORED, N1 % 2 == 0>(re, tp, cst.gm1, qe, nullptr);
    R Fr[5], Fs[5];
    if (plus) conv_num_flux<R, 0>(ro, re, qo, qe, tp, cf, cst, Fr);
    else conv_num_flux<R, 0>(re, ro, qe, qo, tp, cf, cst, Fr);
    unrotate_flux<R>(Fr, d, Fs);
    R term[5];
#pragma unroll
    for (int s = 0; s < 5; ++s) term[s] = -sgn * Fs[s];
    const R* X = sX + c * L::NX * NP;
    if constexpr (!SPLIT) {
        constexpr int o = VISC ? 4 : 0;
#pragma unroll
        for (int s = 0; s < 5; ++s) term[s] += sgn * X[(o + d * 5 + s) * NP + node];
    }
    if constexpr (VISC) {
        R Fo[4], Fn[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            Fo[k] = __ldg(&fvface[(f * 4 + k) * NF + fn]);
            Fn[k] = (BND && bnd) ? tr[(5 + k) * NF + fn] : R(0.5) * (Fo[k] + tr[(5 + k) * NF + fn]);
        }
        if (df == DF_SIPG && !(BND && bnd)) {
            const R* uL = plus ? uo : ue;
            const R* uR = plus ? ue : uo;
            R gj[5][3];
#pragma unroll
            for (int s = 0; s < 5; ++s)
#pragma unroll
                for (int k = 0; k < 3; ++k) gj[s][k] = (k == d) ? (uL[s] - uR[s]) : R(0);
            R AL[3][4], AR[3][4];
            viscous_flux<R>(uL, gj, ucv, cst, AL, 7, nullptr);
            viscous_flux<R>(uR, gj, ucv, cst, AR, 7, nullptr);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const R al = d == 0 ? AL[0][k] : d == 1 ? AL[1][k] : AL[2][k];
                const R ar = d == 0 ? AR[0][k] : d == 1 ? AR[1][k] : AR[2][k];
                Fn[k] = Fn[k] - pen * (R(0.5) * (al + ar));
            }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) term[1 + k] += sgn * (Fo[k] - Fn[k]);
    }
#pragma unroll
    for (int s = 0; s < 5; ++s) tr[s * NF + fn] = term[s] * inv_wend;
}

// unroll count of the volume phase's partner loop (k = 1 .. N1/2): unrolled where B200 timings
// favour it (FP32 at every order; FP64 at p = 3 and p = 5, the latter with 3 CTAs per SM), rolled
// at the other FP64 orders, which were not measured unrolled
template <typename R, int N1> __host__ __device__ constexpr int PAIR_UNROLL() {
    return (sizeof(R) == 4 || N1 == 4 || N1 == 6) ? N1 / 2 : 1;
}

// Phase 4 for direction d: warp segments of N1 lanes own 1-D lines along d. The
// two-point flux is evaluated in the frame whose x axis is e_d.
template <typename R, int N1, int CPC, bool VISC, bool SPLIT, bool CURV>
__device__ __forceinline__ void volume_dir(int d, const Cst<R>& cst, int tp, const R* sD, const R* sX, R* sA,
                                           const R* sOpsD, const R* sOpsDsk, const R* sH, int lc, int lt, int pos,
                                           int seg, bool lvalid) {
    using L = Layout<R, N1, CPC, VISC, SPLIT, CURV>;
    constexpr int NP = L::NP, NQS = L::NQS;
    const int st = (d == 0) ? 1 : (d == 1) ? N1 : N1 * N1;
    const int t1 = (d == 0) ? 1 : 0, t2 = (d == 2) ? 1 : 2;
    int cc[3];
    cc[0] = cc[1] = cc[2] = 0;
    cc[t1] = lt % N1; cc[t2] = lt / N1;
    const int node = node_of<N1>(d == 0 ? pos : cc[0], d == 1 ? pos : cc[1], d == 2 ? pos : cc[2]);
    const int base = node - pos * st;
    R acc[5] = {R(0), R(0), R(0), R(0), R(0)};
    if constexpr (CURV && SPLIT) {
        // curvilinear: the pair flux is dotted with the averaged metric column
        // 1/2 (C_i[:, d] + C_j[:, d]), symmetric in (i, j) like the flux itself
        const R* Dq = sD + lc * NQS * NP;
        const R* X = sX + (lc * L::NX + L::OM) * NP;   // the metric rows
        NodeQ<R> qi;
        load_q<R>(Dq, NP, node, qi);
        const R mi[3] = {X[(0 * 3 + d) * NP + node], X[(1 * 3 + d) * NP + node], X[(2 * 3 + d) * NP + node]};
        const int segbase = seg * N1;
#pragma unroll 1
        for (int k = 1; k <= N1 / 2; ++k) {
            const int jp = pos + k < N1 ? pos + k : pos + k - N1;      // (pos + k) mod N1
            const int jm = pos - k >= 0 ? pos - k : pos - k + N1;      // (pos - k) mod N1
            const int nj = base + jp * st;
            NodeQ<R> qj;
            load_q<R>(Dq, NP, nj, qj);
            const R nv[3] = {R(0.5) * (mi[0] + X[(0 * 3 + d) * NP + nj]), R(0.5) * (mi[1] + X[(1 * 3 + d) * NP + nj]),
                             R(0.5) * (mi[2] + X[(2 * 3 + d) * NP + nj])};
            R F[5];
            two_point_n<R>(qi, qj, nv, tp, cst, F);
            const R cj = sOpsDsk[pos * N1 + jp];
            const int src = segbase + jm;
            const R cr = sOpsDsk[pos * N1 + jm];
            const bool dup = ((N1 & 1) == 0) && (2 * k == N1);
#pragma unroll
            for (int s = 0; s < 5; ++s) {
                const R fr = __shfl_sync(0xffffffffu, F[s], src);
                acc[s] += cj * F[s];
                if (!dup) acc[s] += cr * fr;
            }
        }
    } else if constexpr (SPLIT) {
        const R* Dq = sD + lc * NQS * NP;
        NodeQ<R> qi;
        load_q_rot<R>(Dq, NP, node, d, qi);
        R accr[5] = {R(0), R(0), R(0), R(0), R(0)};
#ifdef PH_ALL_ORDERED_PAIRS
#pragma unroll 1
        for (int l = 0; l < N1; ++l) {
            if (l == pos) continue;
            NodeQ<R> qj;
            load_q_rot<R>(Dq, NP, base + l * st, d, qj);
            R F[5];
            two_point_dir<R, 0>(qi, qj, tp, cst, F);
            const R cj = sOpsDsk[pos * N1 + l];
#pragma unroll
            for (int s = 0; s < 5; ++s) accr[s] += cj * F[s];
        }
#else
        const int segbase = seg * N1;
        // the partner loop is unrolled (PAIR_UNROLL): the independent pair fluxes interleave.
        // At p = 5 on B200 the FP32 stage kernel takes 0.276 ms instead of 0.294 ms, the FP64
        // one 0.496 ms instead of 0.515 with 3 CTAs per SM (at 4 CTAs per SM the unrolled FP64
        // body spills at the 64-register bound and takes 0.533 ms)
#pragma unroll(PAIR_UNROLL<R, N1>())
        for (int k = 1; k <= N1 / 2; ++k) {
            const int jp = pos + k < N1 ? pos + k : pos + k - N1;      // (pos + k) mod N1
            const int jm = pos - k >= 0 ? pos - k : pos - k + N1;      // (pos - k) mod N1
            const bool dup = ((N1 & 1) == 0) && (2 * k == N1);
            const R cj = sOpsDsk[pos * N1 + jp];
            if (L::HP > 0 && dup) {   // the opposite node's pair flux, from the pair pass
                const int hp = pos < L::HP ? pos : pos - L::HP;
                const R* h = sH + ((((size_t)d * CPC + lc) * L::NF + lt) * L::HP + hp) * 5;
#pragma unroll
                for (int s = 0; s < 5; ++s) accr[s] += cj * h[s];
                continue;
            }
            NodeQ<R> qj;
            load_q_rot<R>(Dq, NP, base + jp * st, d, qj);
            R F[5];
            two_point_dir<R, 0>(qi, qj, tp, cst, F);
            const int src = segbase + jm;
            const R cr = sOpsDsk[pos * N1 + jm];
#pragma unroll
            for (int s = 0; s < 5; ++s) {
                const R fr = __shfl_sync(0xffffffffu, F[s], src);
                accr[s] += cj * F[s];
                if (!dup) accr[s] += cr * fr;
            }
        }
#endif
        unrotate_flux<R>(accr, d, acc);
    }
    if constexpr (!SPLIT) {   // (the viscous divergence comes precomputed from the auxiliary kernel)
        const R* X = sX + lc * L::NX * NP;
        constexpr int o = VISC ? 4 : 0;
#pragma unroll
        for (int l = 0; l < N1; ++l) {
            const int nl = base + l * st;
            const R coef = sOpsD[pos * N1 + l];
#pragma unroll
            for (int s = 0; s < 5; ++s) acc[s] += coef * X[(o + d * 5 + s) * NP + nl];
        }
    }
    if (lvalid) {
        R* A = sA + lc * 5 * NP;   // (SEPA: direction d's own accumulator)
#pragma unroll
        for (int s = 0; s < 5; ++s) {
            if (d == 0 || L::SEPA) A[s * NP + node] = acc[s];
            else A[s * NP + node] += acc[s];
        }
    }
}

// Entropy of the relaxation RK method (FP64): component s of the entropy variables
// (Euler::compute_entropy_variables, euler.cpp:811-829) and the numerical entropy function
// -rho log(p rho^-gamma) (compute_numerical_entropy_function, :437-447; compute_entropy,
// :512-530), from the conservative state.
__device__ __forceinline__ double entropy_variable(const double u[5], int s, double gam) {
    const double p = (gam - 1.0) * (u[4] - 0.5 * (u[1] * u[1] + u[2] * u[2] + u[3] * u[3]) / u[0]);
    const double ent = log(p * pow(u[0], -gam));
    const double rt = p / (gam - 1.0);
    if (s == 0) return (rt * (gam + 1.0 - ent) - u[4]) / rt;
    if (s == 4) return -u[0] / rt;
    return u[s] / rt;
}
__device__ __forceinline__ double numerical_entropy_fn(const double u[5], double gam) {
    const double p = (gam - 1.0) * (u[4] - 0.5 * (u[1] * u[1] + u[2] * u[2] + u[3] * u[3]) / u[0]);
    return -u[0] * log(p * pow(u[0], -gam));
}

// Integrated numerical entropy of u_n + gamma (u1 - u_n), per cell: sum over the nodes of
// W det J eta (GLL collocation: the volume quadrature is the solution nodes). One CTA per
// cell, fixed-order reduction.
template <int N1>
__global__ void rrk_entropy_kernel(const double* __restrict__ Un, const double* __restrict__ U1, double gamma,
                                   const OpTab* __restrict__ ops, int nc, double h3,
                                   const double* __restrict__ metric, double gam, double* __restrict__ partial) {
    constexpr int NP = N1 * N1 * N1;
    const int cell = blockIdx.x, node = threadIdx.x;
    double e = 0.0;
    if (node < NP) {
        double u[5];
#pragma unroll
        for (int s = 0; s < 5; ++s) {
            const size_t i = ((size_t)cell * 5 + s) * NP + node;
            u[s] = Un[i] + gamma * (U1[i] - Un[i]);
        }
        const int x = node % N1, y = (node / N1) % N1, z = node / (N1 * N1);
        const double W = ops->w[x] * ops->w[y] * ops->w[z];
        const double J = metric ? 1.0 / metric[((size_t)cell * 10 + 9) * NP + node] : h3;
        e = W * J * numerical_entropy_fn(u, gam);
    }
    __shared__ double red[32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) e += __shfl_down_sync(0xffffffffu, e, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = e;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < (int)((blockDim.x + 31) / 32); ++w) t += red[w];
        partial[cell] = t;
    }
}

// Relaxation RK: this tile's share of v(u_i)^T M k_i, the entropy variables of the stage
// input (FP64, from the state) times M k = W det J k = W (h^2, or 1 on curvilinear cells) G
// (RootFindingRRKODESolver::compute_entropy_change_estimate, root_finding_rrk_ode_solver.cpp:
// 355-390), written to a.ent_partial[tile]. Compiled into the generic flux-set kernels only
// (relaxed steps dispatch there), so the hot kernel's register allocation does not see it.
template <typename R, int N1, int CPC, int NT, bool CURV>
__device__ __forceinline__ void entropy_estimate_tile(const StageArgs& a, const R* sA, int cell0) {
    constexpr int NP = N1 * N1 * N1;
    const int tid = threadIdx.x;
    double ent = 0.0;
    for (int it = tid; it < CPC * 5 * NP; it += NT) {
        const int c = it / (5 * NP), rem = it % (5 * NP), s = rem / NP, node = rem % NP;
        const int cell = cell0 + c;
        if (cell >= a.nc) continue;
        double u[5];
#pragma unroll
        for (int q = 0; q < 5; ++q) u[q] = a.U[((size_t)cell * 5 + q) * NP + node];
        const double v = entropy_variable(u, s, a.pc.gam);
        const int x = node % N1, y = (node / N1) % N1, z = node / (N1 * N1);
        const double W = a.ops->w[x] * a.ops->w[y] * a.ops->w[z];
        const double G = (double)sA[it];
        ent += v * (CURV ? W * G : W * a.h * a.h * G);
    }
    __shared__ double ered[32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ent += __shfl_down_sync(0xffffffffu, ent, o);
    if ((tid & 31) == 0) ered[tid >> 5] = ent;
    __syncthreads();
    if (tid == 0) {
        double t = 0.0;
        for (int w = 0; w < (NT + 31) / 32; ++w) t += ered[w];
        a.ent_partial[cell0 / CPC] = t;
    }
}

// Warms L2 with the inputs a tile reads after its first phase: its own stage state, the
// RK registers the epilogue reads (u_n, running sum, carry, Kahan term) and its block of
// viscous terms. One L2 prefetch per 128-byte line, addresses clamped inside the tile's
// slices; a prefetch writes nothing. The FP64 stage kernel gains 3-4 % on B200; the
// precision form does not (its epilogue loads are already hidden), so only FP64 uses it.
template <typename R, int N1, int CPC, bool VISC>
__device__ __forceinline__ void prefetch_tile_l2(const StageArgs& a, int cell0) {
    constexpr int NP = N1 * N1 * N1;
    const int ncell = (a.nc - cell0) < CPC ? (a.nc - cell0) : CPC;
    const size_t n5 = (size_t)ncell * 5 * NP, o5 = (size_t)cell0 * 5 * NP;
    const bool rk = a.mode != 0;
    const double* arr[5] = {a.U, rk ? a.Un : nullptr, rk ? a.acc_in : nullptr, rk ? a.carry_in : nullptr,
                            rk ? a.comp : nullptr};
    const int nl = (int)((n5 + 15) / 16);   // 16 doubles per line
    for (int i = threadIdx.x; i < 5 * nl; i += blockDim.x) {
        const double* b = arr[i / nl];
        if (b) {
            const size_t e = (size_t)(i % nl) * 16;
            asm volatile("prefetch.global.L2 [%0];" ::"l"(b + o5 + (e < n5 ? e : n5 - 1)));
        }
    }
    if constexpr (VISC) {
        constexpr int VT = viscous_terms_per_cell<N1>();
        const R* fb = static_cast<const R*>(a.Fv) + (size_t)cell0 * VT;
        constexpr int per = 128 / (int)sizeof(R);
        const int nt = ncell * VT, nv = (nt + per - 1) / per;
        for (int i = threadIdx.x; i < nv; i += blockDim.x) {
            const int e = i * per;
            asm volatile("prefetch.global.L2 [%0];" ::"l"(fb + (e < nt ? e : nt - 1)));
        }
    }
}

// ------------------------------------------------------------------------------------
// Residual (+ mass inverse + RK epilogue) kernel
// ------------------------------------------------------------------------------------
// FS selects the flux set: 0 = any (two-point / convective / dissipative types read at
// run time), 1 = Chandrashekar split flux + entropy-conserving baseline with Roe
// dissipation (+ BR2 when viscous) fixed at compile time, which removes the unused
// variants from the instruction stream.
//
// residual_tile does the work of one CTA on the tile of CPC cells starting at cell0;
// residual_kernel runs one tile per CTA of one discretisation, residual_kernel_batched
// runs the tiles of many independent discretisations (a batch of solves) from a tile list.
// One DOF of a low-storage 3S* / 3S*+ stage (mode 3; LowStorageRungeKuttaODESolver stage,
// low_storage_runge_kutta_ode_solver.cpp:22-100): S2 += delta_i S1; S1 = g0 S1 + g1 S2 + g2 S3 +
// beta dt k; S4 += bhat_i dt k; the DOF's squared scaled error added to err2.
__device__ __forceinline__ void ls_stage_dof(const StageArgs& a, size_t dof, double k, double& err2) {
    const double s1 = a.U[dof];
    const double s3 = a.ls_s3[dof];
    const double kdt = a.dt * k;
    double e = 0.0, ref = 0.0;
    bool have_err = false;
    if (a.ls_s1_out) {
        const double s2 = (a.ls_first ? 0.0 : a.ls_s2[dof]) + a.ls_delta * s1;
        const double s1n = ((a.ls_g0 * s1 + a.ls_g1 * s2) + a.ls_g2 * s3) + a.ls_beta * kdt;
        a.ls_s1_out[dof] = s1n;
        if (a.ls_embedded) {   // embedded solution of the last 3S* stage
            const double s2e = ((s2 + a.ls_delta_s * s1n) + a.ls_delta_s1 * s3) * a.ls_inv_sum_delta;
            a.ls_s2[dof] = s2e;
            e = s1n - s2e; ref = fmax(fabs(s1n), fabs(s2e)); have_err = true;
        } else {
            a.ls_s2[dof] = s2;
        }
    }
    if (a.ls_s4) {
        const double s4 = (a.ls_first ? s3 : a.ls_s4[dof]) + a.ls_bhat * kdt;
        a.ls_s4[dof] = s4;
        if (!a.ls_s1_out) { e = s1 - s4; ref = fmax(fabs(s1), fabs(s4)); have_err = true; }
    }
    if (have_err && a.err_partial) {
        const double r = e / (a.atol + a.rtol * ref);
        err2 += r * r;
    }
}

// the block's sum of err2 (warp shuffles, then the warps in order) into *out: a tile's squared
// scaled error, summed in a fixed order
template <int NT>
__device__ __forceinline__ void ls_tile_error(double err2, double* out) {
    __shared__ double red[32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) err2 += __shfl_down_sync(0xffffffffu, err2, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = err2;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < (NT + 31) / 32; ++w) t += red[w];
        *out = t;
    }
}

template <typename R, int N1, int CPC, bool VISC, bool SPLIT, int FS, bool CURV, bool BULK = false, bool BND = false>
__device__ __forceinline__ void residual_tile(const StageArgs& a, const int cell0) {
    static_assert(!BULK || (std::is_same<R, double>::value && N1 % 2 == 0 && !CURV), "bulk staging: FP64, even N1");
    static_assert(!BND || !BULK, "boundary faces: plain loads");
    using L = Layout<R, N1, CPC, VISC, SPLIT, CURV>;
    constexpr int NP = L::NP, NF = L::NF, NT = L::NT, TR = L::TR, NQS = L::NQS;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    R* sm = reinterpret_cast<R*>(smem_raw);
    R* sOpsD = sm + L::oOps;
    R* sOpsDsk = sOpsD + N1 * N1;
    R* sOpsB = sOpsDsk + N1 * N1;
    R* sOpsW = sOpsB + N1 * N1;
    R* sU = sm + L::oU;
    R* sD = sm + L::oD;
    R* sT = sm + L::oT;
    R* sA = sm + L::oA;
    R* sX = sm + L::oX;

    // L2 prefetch of the tile's inputs: FP64, and FP32 at p = 3 (B200: 0.227 -> 0.217 ms at 32^3;
    // at p = 5 it costs FP32 8 %)
    if constexpr (std::is_same<R, double>::value || N1 == 4) prefetch_tile_l2<R, N1, CPC, VISC>(a, cell0);
    Cst<R> cst; cst.load(a.pc);
    const int tp = FS == 1 ? (int)TP_CH : a.pc.two_point;
    const int cf = FS == 1 ? (int)CF_EC_ROE : a.pc.conv_flux;
    const int df = FS == 1 ? (int)DF_BR2 : a.pc.diss_flux;
    const int ucv = a.pc.use_const_visc;
    const int tid = threadIdx.x;

    for (int i = tid; i < N1 * N1; i += NT) {
        sOpsD[i] = (R)a.ops->D[(i / N1) * MAXN1 + (i % N1)];
        sOpsDsk[i] = (R)a.ops->Dsk[(i / N1) * MAXN1 + (i % N1)];
        sOpsB[i] = (R)a.ops->B[(i / N1) * MAXN1 + (i % N1)];
    }
    for (int i = tid; i < N1; i += NT) sOpsW[i] = (R)a.ops->w[i];

    // bulk staging: the tile's state (cells contiguous) into sU and each cell's viscous
    // divergence into its sX rows, issued before the neighbour gathers so both overlap
    __shared__ __align__(8) unsigned long long tile_bar;
    const int ncell = (a.nc - cell0) < CPC ? (a.nc - cell0) : CPC;
    if constexpr (BULK) {
        if (tid == 0) {
            mbar_init(&tile_bar, 1);
            const unsigned ubytes = (unsigned)(ncell * 5 * NP * sizeof(double));
            const unsigned vbytes = VISC ? (unsigned)(4 * NP * sizeof(double)) : 0u;
            mbar_expect_tx(&tile_bar, ubytes + ncell * vbytes);
            bulk_copy_g2s(sU, a.U + (size_t)cell0 * 5 * NP, ubytes, &tile_bar);
            if constexpr (VISC) {
                for (int c = 0; c < ncell; ++c)
                    bulk_copy_g2s(sX + c * L::NX * NP,
                                  static_cast<const double*>(a.Fv) + (size_t)(cell0 + c) * viscous_terms_per_cell<N1>(),
                                  vbytes, &tile_bar);
            }
        }
    }

    // ---- phase 1: neighbour face traces (and the neighbour's viscous flux there)
    for (int it = tid; it < CPC * 6 * NF; it += NT) {
        const int fn = it % NF;
        const int f = (it / NF) % 6;
        const int c = it / (NF * 6);
        int cell = cell0 + c; if (cell >= a.nc) cell = a.nc - 1;
        const int cn = __ldg(&a.nbr[cell * 6 + f]);
        const int nn = face_node_volume_index<N1>(f, fn, (f & 1) ? 0 : N1 - 1);
        R* tr = sT + (c * 6 + f) * TR * NF;
        if constexpr (BND) {
            if (cn < 0) {   // boundary face: the boundary state of this cell's face value
                const int k = -1 - cn;
                const int bt = __ldg(&a.btype[k]);
                const int no = face_node_volume_index<N1>(f, fn, (f & 1) ? N1 - 1 : 0);
                const R sg = (f & 1) ? R(1) : R(-1);
                R ui[5], ub[5];
#pragma unroll
                for (int s = 0; s < 5; ++s) ui[s] = (R)__ldg(&a.U[((size_t)cell * 5 + s) * NP + no]);
                unsigned* st = std::is_same<R, double>::value ? a.status : nullptr;
                if constexpr (CURV) {   // the outward unit normal sg C[:, dn] / |C[:, dn]| at the face node
                    const int dn = f >> 1;
                    const double* M = a.metric + (size_t)cell * 10 * NP + no;
                    const double m0 = __ldg(&M[(0 * 3 + dn) * NP]), m1 = __ldg(&M[(1 * 3 + dn) * NP]),
                                 m2 = __ldg(&M[(2 * 3 + dn) * NP]);
                    const double Jf = sqrt(m0 * m0 + m1 * m1 + m2 * m2);
                    const R nv[3] = {(R)(sg * m0 / Jf), (R)(sg * m1 / Jf), (R)(sg * m2 / Jf)};
                    boundary_state_normal<R>(bt, nv, ui, a.pc, ub, st);
                } else {
                    boundary_state_face<R>(bt, f, ui, a.pc, ub, st);
                }
#pragma unroll
                for (int s = 0; s < 5; ++s) tr[s * NF + fn] = ub[s];
                if constexpr (VISC) {   // F*_v . e_d = sg (F*_v . n_out)
                    const R* fb = static_cast<const R*>(a.Fb) + (size_t)k * 4 * NF;
#pragma unroll
                    for (int q = 0; q < 4; ++q) tr[(5 + q) * NF + fn] = sg * __ldg(&fb[q * NF + fn]);
                }
                continue;
            }
        }
        R ue[5];
#pragma unroll
        for (int s = 0; s < 5; ++s) { ue[s] = (R)__ldg(&a.U[((size_t)cn * 5 + s) * NP + nn]); tr[s * NF + fn] = ue[s]; }
        if constexpr (VISC) {   // the neighbour's block of the opposite face: same node order, contiguous
            const R* fb = static_cast<const R*>(a.Fv) + (size_t)cn * viscous_terms_per_cell<N1>() + 4 * NP +
                          (f ^ 1) * 4 * NF;
#pragma unroll
            for (int k = 0; k < 4; ++k) tr[(5 + k) * NF + fn] = (R)__ldg(&fb[k * NF + fn]);
        }
    }

    if constexpr (BULK) {   // bounded wait for the staged tile; on a timeout no output is written
        __syncthreads();    // the barrier's initialisation is visible to every thread
        bool done = mbar_wait_bounded(&tile_bar, 0, 1ll << 22);
        if (!done && tid == 0) atomicOr(a.status, ST_COPY_TIMEOUT);
        if (__syncthreads_or(!done)) {
            if (!done) mbar_wait_bounded(&tile_bar, 0, 1ll << 22);   // the copies in flight, again bounded
            return;
        }
    }

    // ---- phase 2: node quantities (+ viscous / convective physical fluxes)
    for (int it = tid; it < CPC * NP; it += NT) {
        const int c = it / NP, node = it % NP;
        int cell = cell0 + c;
        const bool valid = cell < a.nc;
        if (!valid) cell = a.nc - 1;
        double ud[5];
        if constexpr (BULK) {   // from the staged tile (a missing cell of the last tile: its first cell)
            const int cs = valid ? c : 0;
#pragma unroll
            for (int s = 0; s < 5; ++s) ud[s] = (double)sU[(cs * 5 + s) * NP + node];
        } else {
#pragma unroll
            for (int s = 0; s < 5; ++s) ud[s] = __ldg(&a.U[((size_t)cell * 5 + s) * NP + node]);
        }
        // positivity in FP64: the FP64 path checks the pressure it computes anyway, the
        // precision form checks the FP64 state before rounding it
        if constexpr (!std::is_same<R, double>::value) {
            if (valid) check_state_fp64(ud, a.pc.gm1, a.status);
        } else {
            if (valid && ud[0] < 0.0) atomicOr(a.status, ST_NONPHYSICAL);
        }
        R u[5];
#pragma unroll
        for (int s = 0; s < 5; ++s) { u[s] = (R)ud[s]; if constexpr (!BULK) sU[(c * 5 + s) * NP + node] = u[s]; }
        if constexpr (BULK) {
            if (!valid) {
#pragma unroll
                for (int s = 0; s < 5; ++s) sU[(c * 5 + s) * NP + node] = u[s];
            }
        }
        NodeQ<R> q;
        node_prepare<R>(u, tp, cst.gm1, q, std::is_same<R, double>::value && valid ? a.status : nullptr);
        store_q<R>(sD + c * NQS * NP, NP, node, q);
        R* X = sX + c * L::NX * NP;
        if constexpr (VISC) {
            if (!BULK || !valid) {   // (staged by the bulk copy for the tile's cells)
                const R* dv = static_cast<const R*>(a.Fv) + (size_t)cell * viscous_terms_per_cell<N1>();
#pragma unroll
                for (int k = 0; k < 4; ++k) X[k * NP + node] = __ldg(&dv[k * NP + node]);
            }
        }
        if constexpr (CURV) {
#pragma unroll
            for (int i = 0; i < 9; ++i) X[(L::OM + i) * NP + node] = (R)__ldg(&a.metric[((size_t)cell * 10 + i) * NP + node]);
        }
        if constexpr (!SPLIT && CURV) {   // the contravariant fluxes F . C[:, d]
            constexpr int o = VISC ? 4 : 0;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const R m[3] = {X[(L::OM + 0 * 3 + d) * NP + node], X[(L::OM + 1 * 3 + d) * NP + node],
                                X[(L::OM + 2 * 3 + d) * NP + node]};
                R F[5];
                conv_flux_n<R>(q, m, cst.shift(), F);
#pragma unroll
                for (int s = 0; s < 5; ++s) X[(o + d * 5 + s) * NP + node] = F[s];
            }
        } else if constexpr (!SPLIT) {
            constexpr int o = VISC ? 4 : 0;
            R F[5];
            conv_flux_dir<R, 0>(q, cst.shift(), F);
#pragma unroll
            for (int s = 0; s < 5; ++s) X[(o + 0 * 5 + s) * NP + node] = F[s];
            conv_flux_dir<R, 1>(q, cst.shift(), F);
#pragma unroll
            for (int s = 0; s < 5; ++s) X[(o + 1 * 5 + s) * NP + node] = F[s];
            conv_flux_dir<R, 2>(q, cst.shift(), F);
#pragma unroll
            for (int s = 0; s < 5; ++s) X[(o + 2 * 5 + s) * NP + node] = F[s];
        }
    }
    __syncthreads();

    // ---- phase 3: face fluxes (canonical orientation), lifted with 1/w_end
    {
        const R inv_wend = R(1) / sOpsW[0];
        const R pen = (R)a.pen;
        for (int it = tid; it < CPC * 6 * NF; it += NT) {
            const int fn = it % NF;
            const int f = (it / NF) % 6;
            const int c = it / (NF * 6);
            const R* fvface = nullptr;
            int cell = cell0 + c; if (cell >= a.nc) cell = a.nc - 1;
            if constexpr (VISC) fvface = static_cast<const R*>(a.Fv) + (size_t)cell * viscous_terms_per_cell<N1>() + 4 * NP;
            const bool bnd = BND && __ldg(&a.nbr[cell * 6 + f]) < 0;
            face_item<R, N1, CPC, VISC, SPLIT, CURV, BND>(cst, tp, cf, df, ucv, sU, sD, sT, sX, c, f, fn, pen,
                                                         inv_wend, fvface, bnd);
        }
    }
    // ---- opposite-node pair fluxes (even N1): each evaluated once, read by both lanes in phase 4
    if constexpr (L::HP > 0) {
        constexpr int HP = L::HP, PER_D = CPC * NF * HP;
        R* sH = sm + L::oH;
        for (int t = tid; t < 3 * PER_D; t += NT) {
            const int d = t / PER_D, r = t - d * PER_D;
            const int c = r / (NF * HP), lt = (r / HP) % NF, i = r % HP;
            const int st = (d == 0) ? 1 : (d == 1) ? N1 : N1 * N1;
            const int t1 = (d == 0) ? 1 : 0, t2 = (d == 2) ? 1 : 2;
            int cc[3] = {0, 0, 0};
            cc[t1] = lt % N1; cc[t2] = lt / N1;
            const int base = node_of<N1>(cc[0], cc[1], cc[2]);
            const R* Dq = sD + c * NQS * NP;
            NodeQ<R> qi, qj;
            load_q_rot<R>(Dq, NP, base + i * st, d, qi);
            load_q_rot<R>(Dq, NP, base + (i + HP) * st, d, qj);
            R F[5];
            two_point_dir<R, 0>(qi, qj, tp, cst, F);
#pragma unroll
            for (int s = 0; s < 5; ++s) sH[(size_t)t * 5 + s] = F[s];
        }
    }

    // ---- phase 4: volume terms, one direction at a time
    {
        constexpr int SPW = L::SPW;
        const int warp = tid >> 5, lane = tid & 31;
        const int seg = lane / N1, pos = lane % N1;
        const int line = warp * SPW + seg;
        const bool lvalid = (seg < SPW) && (line < CPC * NF);
        const int lc = lvalid ? line / NF : 0;
        const int lt = lvalid ? line % NF : 0;
        // unrolled: the direction, its line stride and the frame rotation are compile-time
        // constants in each copy (5-12 % faster than one runtime-indexed copy on B200)
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            if (d == 0 || !L::SEPA) __syncthreads();
            R* Ad = (L::SEPA && d > 0) ? sm + L::oA1 + (d - 1) * CPC * 5 * NP : sA;
            volume_dir<R, N1, CPC, VISC, SPLIT, CURV>(d, cst, tp, sD, sX, Ad, sOpsD, sOpsDsk, sm + L::oH, lc, lt, pos,
                                                     seg, lvalid);
        }
        __syncthreads();
    }

    // ---- phase 5: G = -volume + lifted faces; mass inverse; outputs
    for (int it = tid; it < CPC * NP; it += NT) {
        const int c = it / NP, node = it % NP;
        const int x = node % N1, y = (node / N1) % N1, z = node / (N1 * N1);
        const int cx[3] = {x, y, z};
        R* A = sA + c * 5 * NP;
        R G[5];
        if constexpr (L::SEPA) {   // -(a0 + a1 + a2) = (-a0 - a1) - a2 exactly
            const R* A1 = sm + L::oA1 + c * 5 * NP;
            const R* A2 = A1 + CPC * 5 * NP;
#pragma unroll
            for (int s = 0; s < 5; ++s) G[s] = (-A[s * NP + node] - A1[s * NP + node]) - A2[s * NP + node];
        } else {
#pragma unroll
            for (int s = 0; s < 5; ++s) G[s] = -A[s * NP + node];
        }
        if constexpr (VISC) {
            const R* X = sX + c * L::NX * NP;
#pragma unroll
            for (int k = 0; k < 4; ++k) G[1 + k] -= X[k * NP + node];
        }
#pragma unroll
        for (int f = 0; f < 6; ++f) {
            const int dn = f >> 1;
            const int b = (f & 1) ? N1 - 1 : 0;
            if (cx[dn] != b) continue;
            const int t1 = (dn == 0) ? 1 : 0, t2 = (dn == 2) ? 1 : 2;
            const int fn = cx[t2] * N1 + cx[t1];
            const R* tr = sT + (c * 6 + f) * TR * NF;
#pragma unroll
            for (int s = 0; s < 5; ++s) G[s] += tr[s * NF + fn];
        }
#pragma unroll
        for (int s = 0; s < 5; ++s) A[s * NP + node] = G[s];
    }
    if (a.mode != 0 && a.fr) {
        // B (x) B (x) B applied direction by direction, ping-pong between sA and sD; curvilinear
        // cells: the weight-adjusted inverse B (x3) [ (1 / det J) B (x3) G ] (P = (M+K)^-1 W = B on
        // collocated GLL nodes, dg_base.cpp:4217-4249), 1 / det J applied between the two
        R* src = sA; R* dst = sD;
        for (int rep = 0; rep < (CURV ? 2 : 1); ++rep) {
            if (rep == 1) {
                __syncthreads();
                for (int it = tid; it < CPC * 5 * NP; it += NT) {
                    const int c = it / (5 * NP), node = it % NP;
                    int cell = cell0 + c; if (cell >= a.nc) cell = a.nc - 1;
                    src[it] = (R)((double)src[it] * __ldg(&a.metric[((size_t)cell * 10 + 9) * NP + node]));
                }
            }
            for (int d = 0; d < 3; ++d) {
                __syncthreads();
                const int st = (d == 0) ? 1 : (d == 1) ? N1 : N1 * N1;
                for (int it = tid; it < CPC * NP; it += NT) {
                    const int c = it / NP, node = it % NP;
                    const int pos = (node / st) % N1;
                    const int base = node - pos * st;
                    for (int s = 0; s < 5; ++s) {
                        R v = R(0);
                        for (int l = 0; l < N1; ++l) v += sOpsB[pos * N1 + l] * src[(c * 5 + s) * NP + base + l * st];
                        dst[(c * 5 + s) * NP + node] = v;
                    }
                }
                R* t = src; src = dst; dst = t;
            }
        }
        __syncthreads();
        if (src != sA) {
            for (int it = tid; it < CPC * 5 * NP; it += NT) sA[it] = src[it];
        }
    }
    __syncthreads();
    if (a.mode == 2) {
        // Butcher RK stage: the thread's inputs (u_n and the running sum) for all its DOFs
        // are loaded before its first store, so that the loads are in flight together
        // (the outputs may alias the inputs, but only DOF by DOF)
        constexpr int TOT = CPC * 5 * NP, PER = (TOT + NT - 1) / NT;
        double un[PER], bs[PER];
#pragma unroll
        for (int r = 0; r < PER; ++r) {
            const int it = tid + r * NT;
            un[r] = bs[r] = 0.0;
            if (it < TOT && cell0 + it / (5 * NP) < a.nc) {
                const size_t dof = (size_t)cell0 * 5 * NP + it;
                un[r] = a.Un[dof];
                bs[r] = a.acc_in ? a.acc_in[dof] : (a.inc_mode ? 0.0 : un[r]);
            }
        }
#pragma unroll
        for (int r = 0; r < PER; ++r) {
            const int it = tid + r * NT;
            if (it >= TOT) break;
            const int cell = cell0 + it / (5 * NP);
            if (cell >= a.nc) break;
            const int node = (it % (5 * NP)) % NP;
            const size_t dof = (size_t)cell0 * 5 * NP + it;
            const double G = (double)sA[it];
            const double k = CURV ? (a.fr ? G : G * __ldg(&a.metric[((size_t)cell * 10 + 9) * NP + node])) : G * a.inv_h;
            const double sum = bs[r] + a.c_acc * k;
            if (a.acc_out) a.acc_out[dof] = sum;
            if (a.final_out) {
                if (a.comp) {   // compensated u_{n+1} = u_n + increment
                    const double y = sum - a.comp[dof];
                    const double t = un[r] + y;
                    a.comp[dof] = (t - un[r]) - y;
                    a.final_out[dof] = t;
                } else {
                    a.final_out[dof] = a.inc_mode ? un[r] + sum : sum;
                }
            }
            if (a.next) {
                const double cin = a.carry_in ? a.carry_in[dof] : 0.0;
                a.next[dof] = (cin + a.a_next * k) * a.dt + un[r];
            }
            if (a.carry_out) a.carry_out[dof] = a.a_carry * k;
        }
        if constexpr (FS == 0) {
            if (a.ent_partial) entropy_estimate_tile<R, N1, CPC, NT, CURV>(a, sA, cell0);
        }
        return;
    }
    // residual (mode 0), k = M^-1 R (mode 1), low-storage stage (mode 3)
    double err2 = 0.0;   // low-storage error estimate: this thread's share of the tile
    for (int it = tid; it < CPC * 5 * NP; it += NT) {
        const int c = it / (5 * NP);
        const int rem = it % (5 * NP);
        const int node = rem % NP;
        const int cell = cell0 + c;
        if (cell >= a.nc) continue;
        const size_t dof = (size_t)cell * 5 * NP + rem;
        const double G = (double)sA[it];
        if (a.mode == 0) {
            const int x = node % N1, y = (node / N1) % N1, z = node / (N1 * N1);
            const double W = a.ops->w[x] * a.ops->w[y] * a.ops->w[z];
            a.out[dof] = CURV ? W * G : W * a.h * a.h * G;
            continue;
        }
        // affine: M^-1 R = G / h; curvilinear: R / (W det J) = G / det J (cDG), or the weight-adjusted
        // passes above, which applied 1 / det J already (FR)
        const double k = CURV ? (a.fr ? G : G * __ldg(&a.metric[((size_t)cell * 10 + 9) * NP + node])) : G * a.inv_h;
        if (a.mode == 1) { a.out[dof] = k; continue; }
        if (a.mode == 3) {
            ls_stage_dof(a, dof, k, err2);
            continue;
        }
    }
    if (a.mode == 3 && a.err_partial) ls_tile_error<NT>(err2, &a.err_partial[cell0 / CPC]);
}

template <typename R, int N1, int CPC, bool VISC, bool SPLIT, bool CURV>
__host__ __device__ constexpr bool stage_bulk() {
    return PH_BULK_TILE && std::is_same<R, double>::value && N1 % 2 == 0 && !CURV && VISC;
}

template <typename R, int N1, int CPC, bool VISC, bool SPLIT, int FS, bool CURV = false, bool BND = false>
__global__ void __launch_bounds__(Layout<R, N1, CPC, VISC, SPLIT, CURV>::NT, Layout<R, N1, CPC, VISC, SPLIT, CURV>::MINB)
residual_kernel(const StageArgs a) {
    residual_tile<R, N1, CPC, VISC, SPLIT, FS, CURV, !BND && stage_bulk<R, N1, CPC, VISC, SPLIT, CURV>(), BND>(
        a, a.tiles ? __ldg(&a.tiles[blockIdx.x]) : a.cell_begin + (int)blockIdx.x * CPC);
}

// One tile of a batch: instance index and its first cell.
struct BatchTile {
    int inst;
    int cell0;
};

// Persistent batched stage kernel: every CTA walks the tile list with a grid stride; the
// tile's discretisation (state pointers, physics, dt, RK coefficients of this stage) is
// staged from the instance table into shared memory. The per-tile work is the same code as
// residual_kernel, so a solve gives bitwise the same result alone and inside a batch.
// BND: the solves of the group have boundary faces (the boundary-face instance on all their tiles).
template <typename R, int N1, int CPC, bool VISC, bool SPLIT, int FS, bool CURV = false, bool BND = false>
__global__ void __launch_bounds__(Layout<R, N1, CPC, VISC, SPLIT, CURV>::NT, Layout<R, N1, CPC, VISC, SPLIT, CURV>::MINB)
residual_kernel_batched(const StageArgs* __restrict__ inst, const BatchTile* __restrict__ tiles, int ntiles) {
    static_assert(sizeof(StageArgs) % sizeof(int) == 0, "StageArgs is copied as ints");
    __shared__ __align__(16) StageArgs sa;
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const BatchTile tile = tiles[t];
        const int* src = reinterpret_cast<const int*>(inst + tile.inst);
        int* dst = reinterpret_cast<int*>(&sa);
        for (int i = threadIdx.x; i < (int)(sizeof(StageArgs) / sizeof(int)); i += blockDim.x) dst[i] = src[i];
        __syncthreads();
        residual_tile<R, N1, CPC, VISC, SPLIT, FS, CURV, false, BND>(sa, tile.cell0);
        __syncthreads();
    }
}

// ------------------------------------------------------------------------------------
// Auxiliary equation: lifted gradient q = M^{-1}[ vol grad + face (u* - u) n ] (kDG),
// then the viscous flux F_v(u, q) at every node (the split form evaluates it at the
// entropy-projected state, the nodal state for GLL), reduced to what the stage kernel
// needs: its volume divergence and its face-normal component on each face
// (viscous_terms_per_cell).
// ------------------------------------------------------------------------------------
// One thread per (direction, state, line) differentiates the line held in registers: every
// coefficient is a parameter-bank operand, the gradient and then the nodal flux share one buffer, and
// in FP64 every direction's derivative takes its flux's place and the three are summed as they are stored
// (FP32 adds direction by direction into the state's rows, so that its rounding stays what it is).
// Bound by shared memory (84 % of its wavefronts at p = 5): lines along x move as pairs, which leaves
// two-way conflicts along y only. Timed on B200 at 24^3 cells, p = 5: 0.140 ms in FP64 (0.148 with scalar
// x-lines and a divergence summed in shared memory), 0.094 in FP32 (0.099). At p <= 3 a thread per node
// with the coefficients in shared memory was the other form: 32^3 cells p = 3 0.142 against 0.127 here in
// FP64 and 0.090 against 0.076 in FP32, p = 2 0.078 / 0.063 and 0.053 / 0.048, p = 1 0.023 / 0.021.
// An FR auxiliary correction (K_aux != 0) multiplies the gradient by Baux(x)Baux(x)Baux before
// the flux.

// CTAs per SM of the periodic FP64 auxiliary kernel at p = 5 (224 threads): 66 registers, 0.140 ms at 24^3
// cells. Chosen on B200 before the lines along x moved in pairs: 3 (76 registers) 0.163 ms, 4 (70
// registers) 0.147 ms, 5 (56 registers, 32 bytes spilled) 0.155 ms. Asked for explicitly: launch
// bounds naming 1 CTA per SM gave 76 registers.
#ifndef PH_AUX_P5_MINB
#define PH_AUX_P5_MINB 4
#endif

template <int N1, int CPC, bool FRA = false>
struct AuxLayout {
    static constexpr int NP = N1 * N1 * N1, NF = N1 * N1;
    static constexpr int NT = ((CPC * NP + 31) / 32) * 32 > 512 ? 512 : ((CPC * NP + 31) / 32) * 32;
    // CTAs per SM asked of the register allocator (the periodic FP64 kernel at p = 5 with one
    // cell per CTA; the other forms take what they need)
    template <typename R, bool CURV, bool BND>
    static constexpr int minb() {
        return (sizeof(R) == 8 && N1 == 6 && CPC == 1 && !FRA && !CURV && !BND) ? PH_AUX_P5_MINB : 1;
    }
    // state, neighbour traces, then the gradient / nodal flux
    template <typename R>
    static constexpr size_t bytes() {
        return sizeof(R) * ((size_t)CPC * 5 * NP + (size_t)CPC * 6 * 5 * NF +
                            (size_t)CPC * 15 * NP);
    }
};

// The 1-D differentiation matrix and the lifting weight 1/w_end of the auxiliary kernel,
// passed by value (in the line form each coefficient is then a parameter-bank operand).
template <typename R> struct AuxCoef {
    R D[MAXN1 * MAXN1];    // D[pos][l] = l_l'(x_pos)
    R Ba[MAXN1 * MAXN1];   // (M+K_aux)^{-1} diag(w) (read only with an FR auxiliary correction)
    R inv_wend;
};

// node index of position pos along direction d on the line whose transverse coordinates
// are (line % N1, line / N1) (the lower transverse direction first, as face node order)
template <int N1> __device__ __forceinline__ int line_node(int d, int line, int pos) {
    const int a = line % N1, b = line / N1;
    return d == 0 ? node_of<N1>(pos, a, b) : d == 1 ? node_of<N1>(a, pos, b) : node_of<N1>(a, b, pos);
}

// Curvilinear cells (CURV, metric rows [cell][10][NP]: C[k][d] at row k * 3 + d, 1 / det J at
// row 9): the reference gradient r_j = D_j u + lift_j (inv_h = 1) becomes the physical one
// q_d = (1/J) sum_j C[d][j] r_j (the curvilinear volume and face terms of the auxiliary
// equation, strong_dg.cpp:666-1008, with the cDG weight-adjusted inverse mass 1 / (W J) at
// GLL nodes), and the nodal viscous flux its contravariant form F~_j = sum_m C[m][j] F_m, whose
// reference divergence and face values (F~_dn at face nodes, the metric-scaled normal flux) the
// stage kernel takes in place of the affine ones.
template <typename R, int N1>
__device__ __forceinline__ void aux_curv_flux(const R un[5], const R r[5][3], const double* __restrict__ metric,
                                              int cell, int node, int ucv, const Cst<R>& cst, R Ft[3][4]) {
    constexpr int NP = N1 * N1 * N1;
    const double* M = metric + (size_t)cell * 10 * NP + node;
    double C[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) C[i] = __ldg(&M[i * NP]);
    const double iJ = __ldg(&M[9 * NP]);
    R g[5][3];   // the metric products in FP64 (the metric stays FP64 in the precision form)
#pragma unroll
    for (int s = 0; s < 5; ++s)
#pragma unroll
        for (int d = 0; d < 3; ++d)
            g[s][d] = (R)(iJ * (C[d * 3 + 0] * (double)r[s][0] + C[d * 3 + 1] * (double)r[s][1] +
                                C[d * 3 + 2] * (double)r[s][2]));
    R F[3][4];
    viscous_flux<R>(un, g, ucv, cst, F, 7, nullptr);
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int k = 0; k < 4; ++k)
            Ft[j][k] = (R)(C[0 * 3 + j] * (double)F[0][k] + C[1 * 3 + j] * (double)F[1][k] +
                           C[2 * 3 + j] * (double)F[2][k]);
}

// Boundary faces (non-periodic meshes): the outward boundary viscous flux F*_v . n at one node's
// boundary faces (up to three at a corner), stored for the stage kernel in Fb[k][4][NF]
// (evaluate_auxiliary_flux with on_boundary, viscous_numerical_flux.cpp:66-328, called from
// assemble_boundary_term_strong, strong_dg.cpp:2279-2300): the exterior state is the viscous boundary
// state; BR2 and SIPG take its gradient (the interior's, the energy gradient zero on an adiabatic
// wall), the central flux the interior gradient; on an adiabatic 1001 wall both sides' fluxes drop
// the heat flux (dissipative_flux_dot_normal, navier_stokes.cpp:1224-1264).
// Out of line, called for the surface nodes of a boundary-face kernel only (un: the node's state,
// g15: its gradient [5][3] row-major). Curvilinear cells (metric != nullptr): g15 is the reference
// gradient, the physical one is (1/J) C g15 (as aux_curv_flux forms it), the outward unit normal is
// sg C[:, d] / |C[:, d]| and the stored flux |C[:, d]| F*_v . n (the face Jacobian's scaling of
// assemble_boundary_term_strong).
template <typename R, int N1>
__device__ __noinline__ void aux_boundary_fluxes(const int* __restrict__ nbr, const int* __restrict__ btype,
                                                 R* __restrict__ Fb, int cell, int node, const R* un, const R* g15,
                                                 const PhysConst& pc, R pen, const double* __restrict__ metric) {
    constexpr int NF = N1 * N1, NP = N1 * N1 * N1;
    Cst<R> cst; cst.load(pc);
    R g[5][3];
#pragma unroll
    for (int s = 0; s < 5; ++s)
#pragma unroll
        for (int e = 0; e < 3; ++e) g[s][e] = g15[s * 3 + e];
    double C[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    if (metric) {   // the physical gradient
        const double* M = metric + (size_t)cell * 10 * NP + node;
#pragma unroll
        for (int i = 0; i < 9; ++i) C[i] = __ldg(&M[i * NP]);
        const double iJ = __ldg(&M[9 * NP]);
#pragma unroll
        for (int s = 0; s < 5; ++s) {
            const double r0 = g15[s * 3 + 0], r1 = g15[s * 3 + 1], r2 = g15[s * 3 + 2];
#pragma unroll
            for (int e = 0; e < 3; ++e) g[s][e] = (R)(iJ * (C[e * 3 + 0] * r0 + C[e * 3 + 1] * r1 + C[e * 3 + 2] * r2));
        }
    }
    const int cx[3] = {node % N1, (node / N1) % N1, node / (N1 * N1)};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
#pragma unroll
        for (int side = 0; side < 2; ++side) {
            if (cx[d] != (side ? N1 - 1 : 0)) continue;
            const int cn = __ldg(&nbr[cell * 6 + 2 * d + side]);
            if (cn >= 0) continue;
            const int k = -1 - cn;
            const int bt = __ldg(&btype[k]);
            const int t1 = (d == 0) ? 1 : 0, t2 = (d == 2) ? 1 : 2;
            const int fn = cx[t2] * N1 + cx[t1];
            R ub[5];
            boundary_viscous_state<R>(bt, un, pc, ub, nullptr);
            const bool ad = bt == BC_WALL && !pc.bc_isothermal;
            R gb[5][3];
#pragma unroll
            for (int s = 0; s < 5; ++s)
#pragma unroll
                for (int e = 0; e < 3; ++e) gb[s][e] = (ad && s == 4) ? R(0) : g[s][e];
            const R sg = side ? R(1) : R(-1);
            R Fi[3][4], Fe[3][4];
            if (metric) {   // curvilinear: |C[:, d]| F*_v . n with n = sg C[:, d] / |C[:, d]|
                const double m0 = C[0 * 3 + d], m1 = C[1 * 3 + d], m2 = C[2 * 3 + d];
                const double Jf = sqrt(m0 * m0 + m1 * m1 + m2 * m2);
                const R nv[3] = {(R)(sg * m0 / Jf), (R)(sg * m1 / Jf), (R)(sg * m2 / Jf)};
                viscous_flux<R>(un, g, pc.use_const_visc, cst, Fi, 7, nullptr, ad);
                viscous_flux<R>(ub, pc.diss_flux == DF_CENTRAL ? g : gb, pc.use_const_visc, cst, Fe, 7, nullptr, ad);
                R out[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const R fi = Fi[0][q] * nv[0] + Fi[1][q] * nv[1] + Fi[2][q] * nv[2];
                    const R fe = Fe[0][q] * nv[0] + Fe[1][q] * nv[1] + Fe[2][q] * nv[2];
                    out[q] = (R)Jf * (R(0.5) * (fi + fe));
                }
                R* dst = Fb + (size_t)k * 4 * NF + fn;
#pragma unroll
                for (int q = 0; q < 4; ++q) dst[q * NF] = out[q];
                continue;
            }
            viscous_flux<R>(un, g, pc.use_const_visc, cst, Fi, 1 << d, nullptr, ad);
            if (pc.diss_flux == DF_CENTRAL) viscous_flux<R>(ub, g, pc.use_const_visc, cst, Fe, 1 << d, nullptr, ad);
            else viscous_flux<R>(ub, gb, pc.use_const_visc, cst, Fe, 1 << d, nullptr, ad);
            R out[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) out[q] = R(0.5) * (sg * Fi[d][q] + sg * Fe[d][q]);
            if (pc.diss_flux == DF_SIPG) {
                R J[5][3];
#pragma unroll
                for (int s = 0; s < 5; ++s)
#pragma unroll
                    for (int e = 0; e < 3; ++e) J[s][e] = (e == d) ? (un[s] - ub[s]) * sg : R(0);
                viscous_flux<R>(un, J, pc.use_const_visc, cst, Fi, 1 << d, nullptr, ad);
                viscous_flux<R>(ub, J, pc.use_const_visc, cst, Fe, 1 << d, nullptr, ad);
#pragma unroll
                for (int q = 0; q < 4; ++q) out[q] = out[q] - pen * (R(0.5) * (sg * Fi[d][q] + sg * Fe[d][q]));
            }
            R* dst = Fb + (size_t)k * 4 * NF + fn;
#pragma unroll
            for (int q = 0; q < 4; ++q) dst[q * NF] = out[q];
        }
    }
}

// the call above for a node on the cell's surface (a copy of its state and gradient is passed)
template <typename R, int N1>
__device__ __forceinline__ void aux_boundary_node(const int* __restrict__ nbr, const int* __restrict__ btype,
                                                  R* __restrict__ Fb, int cell, int node, const R un[5],
                                                  const R g[5][3], const PhysConst& pc, R pen,
                                                  const double* __restrict__ metric) {
    const int x = node % N1, y = (node / N1) % N1, z = node / (N1 * N1);
    if (x != 0 && x != N1 - 1 && y != 0 && y != N1 - 1 && z != 0 && z != N1 - 1) return;
    R uu[5], gg[15];
#pragma unroll
    for (int s = 0; s < 5; ++s) {
        uu[s] = un[s];
#pragma unroll
        for (int e = 0; e < 3; ++e) gg[s * 3 + e] = g[s][e];
    }
    aux_boundary_fluxes<R, N1>(nbr, btype, Fb, cell, node, uu, gg, pc, pen, metric);
}

// One line of N1 values at stride ST in shared memory, to and from registers. Lines along x at even N1 are
// contiguous and move two values at a time: a stride of N1 values between threads puts scalar accesses
// two to a bank, pairs of them none.
template <typename R, int N1, int ST> __device__ __forceinline__ void line_load(const R* p, R v[N1]) {
    using R2 = std::conditional_t<sizeof(R) == 8, double2, float2>;
    if constexpr (ST == 1 && N1 % 2 == 0) {
#pragma unroll
        for (int l = 0; l < N1; l += 2) {
            const R2 t = *reinterpret_cast<const R2*>(p + l);
            v[l] = t.x;
            v[l + 1] = t.y;
        }
    } else {
#pragma unroll
        for (int l = 0; l < N1; ++l) v[l] = p[l * ST];
    }
}
template <typename R, int N1, int ST> __device__ __forceinline__ void line_store(R* p, const R v[N1]) {
    using R2 = std::conditional_t<sizeof(R) == 8, double2, float2>;
    if constexpr (ST == 1 && N1 % 2 == 0) {
#pragma unroll
        for (int l = 0; l < N1; l += 2) {
            R2 t;
            t.x = v[l];
            t.y = v[l + 1];
            *reinterpret_cast<R2*>(p + l) = t;
        }
    } else {
#pragma unroll
        for (int l = 0; l < N1; ++l) p[l * ST] = v[l];
    }
}
template <int D> struct AuxDir { static constexpr int d = D; };

template <typename R, int N1, int CPC, bool FRA, bool CURV, bool BND = false>
__global__ void __launch_bounds__(AuxLayout<N1, CPC, FRA>::NT, AuxLayout<N1, CPC, FRA>::template minb<R, CURV, BND>())
aux_kernel(const double* __restrict__ U, const int* __restrict__ nbr, int cell_begin, int nc, R inv_h, PhysConst pc,
           AuxCoef<R> co, R* __restrict__ Fv, const double* __restrict__ metric, const int* __restrict__ btype,
           R* __restrict__ Fb, R pen, const int* __restrict__ tiles) {

    using L = AuxLayout<N1, CPC, FRA>;
    constexpr int NP = L::NP, NF = L::NF, NT = L::NT;
    constexpr int VT = viscous_terms_per_cell<N1>();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    R* sU = reinterpret_cast<R*>(smem_raw);   // [c][5][NP] state
    R* sT = sU + CPC * 5 * NP;                // [c][face][5][NF] neighbour traces
    Cst<R> cst; cst.load(pc);
    const int tid = threadIdx.x;
    const int cell0 = tiles ? __ldg(&tiles[blockIdx.x]) : cell_begin + (int)blockIdx.x * CPC;
    // loads unrolled so that all of a thread's loads are in flight before the first store
#pragma unroll
    for (int it = tid; it < CPC * 5 * NP; it += NT) {
        int cell = cell0 + it / (5 * NP); if (cell >= nc) cell = nc - 1;
        sU[it] = (R)__ldg(&U[(size_t)cell * 5 * NP + it % (5 * NP)]);
    }
    // neighbour traces: one thread per (cell, face, face node) finds the node once and loads
    // its five components
#pragma unroll
    for (int it = tid; it < CPC * 6 * NF; it += NT) {
        const int fn = it % NF, f = (it / NF) % 6, c = it / (6 * NF);
        int cell = cell0 + c; if (cell >= nc) cell = nc - 1;
        const int cn = __ldg(&nbr[cell * 6 + f]);
        R* dst = sT + (c * 6 + f) * 5 * NF + fn;
        if constexpr (BND) {
            if (cn < 0) {   // boundary face: the viscous boundary state of this cell's face value
                const int bt = __ldg(&btype[-1 - cn]);
                const int no = face_node_volume_index<N1>(f, fn, (f & 1) ? N1 - 1 : 0);
                R ui[5], ub[5];
#pragma unroll
                for (int s = 0; s < 5; ++s) ui[s] = (R)__ldg(&U[((size_t)cell * 5 + s) * NP + no]);
                boundary_viscous_state<R>(bt, ui, pc, ub, nullptr);
#pragma unroll
                for (int s = 0; s < 5; ++s) dst[s * NF] = ub[s];
                continue;
            }
        }
        const int nn = face_node_volume_index<N1>(f, fn, (f & 1) ? 0 : N1 - 1);
        const double* src = U + (size_t)cn * 5 * NP + nn;
#pragma unroll
        for (int s = 0; s < 5; ++s) dst[s * NF] = (R)__ldg(&src[s * NP]);
    }
    R* sG = sT + CPC * 6 * 5 * NF;   // [c][d][5][NP] gradient, later [c][d][4][NP] flux
    // FP32 up to p = 3: 1/h is applied as the gradient is read, where it joins the flux's first operation
    constexpr bool LATE = sizeof(R) == 4 && N1 <= 4 && !FRA;
    __syncthreads();
    // lifted gradient: D u along the line, the lifting u* - u = (u_ext - u)/2 at both ends;
    // the direction is a compile-time constant, so the line's stride is too
    auto gradient = [&](auto dir) {
        constexpr int d = decltype(dir)::d, st = d == 0 ? 1 : d == 1 ? N1 : N1 * N1;
        for (int task = tid; task < CPC * 5 * NF; task += NT) {
            const int c = task / (5 * NF), r = task % (5 * NF);
            const int line = r % NF, s = r / NF;
            const int base = line_node<N1>(d, line, 0);
            R v[N1], o[N1];
            line_load<R, N1, st>(sU + (c * 5 + s) * NP + base, v);
            const R ue0 = sT[((c * 6 + 2 * d) * 5 + s) * NF + line];
            const R ue1 = sT[((c * 6 + 2 * d + 1) * 5 + s) * NF + line];
#pragma unroll
            for (int pos = 0; pos < N1; ++pos) {
                R acc = R(0);
#pragma unroll
                for (int l = 0; l < N1; ++l) acc += co.D[pos * MAXN1 + l] * v[l];
                if (pos == 0) acc += co.inv_wend * (-(R(0.5) * (v[0] + ue0) - v[0]));
                if (pos == N1 - 1) acc += co.inv_wend * ((R(0.5) * (v[N1 - 1] + ue1) - v[N1 - 1]));
                o[pos] = LATE ? acc : acc * inv_h;
            }
            line_store<R, N1, st>(sG + (c * 15 + d * 5 + s) * NP + base, o);
        }
    };
    gradient(AuxDir<0>());
    gradient(AuxDir<1>());
    gradient(AuxDir<2>());
    __syncthreads();
    if constexpr (FRA) {
        // FR auxiliary correction (M+K_aux)^{-1} in three directions, applied to the DG
        // gradient diag(w)^{-1} r as Baux = (M+K_aux)^{-1} diag(w) along x, then y, then z
        // (the order of the sum-factorised inverse mass); one thread per (component, line)
#pragma unroll
        for (int e = 0; e < 3; ++e) {
            const int st = e == 0 ? 1 : e == 1 ? N1 : N1 * N1;
            for (int task = tid; task < CPC * 15 * NF; task += NT) {
                const int c = task / (15 * NF), r = task % (15 * NF);
                const int line = r % NF, k = r / NF;
                R* g = sG + (c * 15 + k) * NP + line_node<N1>(e, line, 0);
                R v[N1];
#pragma unroll
                for (int l = 0; l < N1; ++l) v[l] = g[l * st];
#pragma unroll
                for (int pos = 0; pos < N1; ++pos) {
                    R acc = R(0);
#pragma unroll
                    for (int l = 0; l < N1; ++l) acc += co.Ba[pos * MAXN1 + l] * v[l];
                    g[pos * st] = acc;
                }
            }
            __syncthreads();
        }
    }
    // viscous flux per node; it replaces the node's own gradient entries
    for (int it = tid; it < CPC * NP; it += NT) {
        const int c = it / NP, node = it % NP;
        R g[5][3];
#pragma unroll
        for (int d = 0; d < 3; ++d)
#pragma unroll
            for (int s = 0; s < 5; ++s)
                g[s][d] = LATE ? sG[(c * 15 + d * 5 + s) * NP + node] * inv_h : sG[(c * 15 + d * 5 + s) * NP + node];
        R un[5];
#pragma unroll
        for (int s = 0; s < 5; ++s) un[s] = sU[(c * 5 + s) * NP + node];
        R F[3][4];
        if constexpr (CURV) {
            int cell = cell0 + c; if (cell >= nc) cell = nc - 1;
            aux_curv_flux<R, N1>(un, g, metric, cell, node, pc.use_const_visc, cst, F);
        } else {
            viscous_flux<R>(un, g, pc.use_const_visc, cst, F, 7, nullptr);
        }
        if constexpr (BND) {
            if (cell0 + c < nc)
                aux_boundary_node<R, N1>(nbr, btype, Fb, cell0 + c, node, un, g, pc, pen, CURV ? metric : nullptr);
        }
#pragma unroll
        for (int d = 0; d < 3; ++d)
#pragma unroll
            for (int k = 0; k < 4; ++k) sG[(c * 15 + d * 4 + k) * NP + node] = F[d][k];
    }
    // divergence sum_d D_d F_d, one thread per (component, line), which also stores the line's face values
    auto derivative = [&](auto dir, int c, int k, int line, R o[N1]) {
        constexpr int d = decltype(dir)::d, st = d == 0 ? 1 : d == 1 ? N1 : N1 * N1;
        R v[N1];
        line_load<R, N1, st>(sG + (c * 15 + d * 4 + k) * NP + line_node<N1>(d, line, 0), v);
#pragma unroll
        for (int pos = 0; pos < N1; ++pos)
#pragma unroll
            for (int l = 0; l < N1; ++l) o[pos] += co.D[pos * MAXN1 + l] * v[l];
        if (cell0 + c < nc) {
            R* dst = Fv + (size_t)(cell0 + c) * VT + 4 * NP + (2 * d * 4 + k) * NF + line;
            dst[0] = v[0];
            dst[4 * NF] = v[N1 - 1];
        }
    };
    if constexpr (sizeof(R) == 8) {
        // FP64: every direction's derivative in place of its flux, summed as it is stored
        auto inplace = [&](auto dir) {
            constexpr int d = decltype(dir)::d, st = d == 0 ? 1 : d == 1 ? N1 : N1 * N1;
            for (int task = tid; task < CPC * 4 * NF; task += NT) {
                const int c = task / (4 * NF), r = task % (4 * NF);
                const int line = r % NF, k = r / NF;
                R o[N1];
#pragma unroll
                for (int pos = 0; pos < N1; ++pos) o[pos] = R(0);
                derivative(dir, c, k, line, o);
                line_store<R, N1, st>(sG + (c * 15 + d * 4 + k) * NP + line_node<N1>(d, line, 0), o);
            }
        };
        __syncthreads();
        inplace(AuxDir<0>());
        inplace(AuxDir<1>());
        inplace(AuxDir<2>());
        __syncthreads();
        for (int it = tid; it < CPC * 4 * NP; it += NT) {
            const int c = it / (4 * NP), i = it % (4 * NP);
            const R* f = sG + c * 15 * NP + i;
            if (cell0 + c < nc) Fv[(size_t)(cell0 + c) * VT + i] = (f[0] + f[4 * NP]) + f[8 * NP];
        }
    } else {
        // FP32: into the state's rows (the state is no longer read), one direction after the other
        auto summed = [&](auto dir) {
            constexpr int d = decltype(dir)::d, st = d == 0 ? 1 : d == 1 ? N1 : N1 * N1;
            __syncthreads();
            for (int task = tid; task < CPC * 4 * NF; task += NT) {
                const int c = task / (4 * NF), r = task % (4 * NF);
                const int line = r % NF, k = r / NF;
                R* dv = sU + (c * 4 + k) * NP + line_node<N1>(d, line, 0);
                R o[N1];
                if constexpr (d == 0) {
#pragma unroll
                    for (int pos = 0; pos < N1; ++pos) o[pos] = R(0);
                } else {
                    line_load<R, N1, st>(dv, o);
                }
                derivative(dir, c, k, line, o);
                line_store<R, N1, st>(dv, o);
            }
        };
        summed(AuxDir<0>());
        summed(AuxDir<1>());
        summed(AuxDir<2>());
        __syncthreads();
        for (int it = tid; it < CPC * 4 * NP; it += NT) {
            const int c = it / (4 * NP);
            const int cell = cell0 + c;
            if (cell >= nc) continue;
            Fv[(size_t)cell * VT + it % (4 * NP)] = sU[c * 4 * NP + it % (4 * NP)];
        }
    }
}

// ------------------------------------------------------------------------------------
// Self-test of the flux quotient against IEEE division on pseudo-random operands
// (one thread per sample, operands from a 64-bit LCG; out[0/1] = max relative error
// in FP64 / FP32 over this block, reduced by the host).
// ------------------------------------------------------------------------------------
static __global__ void quotient_selftest_kernel(unsigned long long seed, int n, double* out) {
    __shared__ double m64[256];
    __shared__ double m32[256];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    double e64 = 0.0, e32 = 0.0;
    if (i < n) {
        unsigned long long s = seed + 0x9E3779B97F4A7C15ull * (unsigned long long)(i + 1);
        s = s * 6364136223846793005ull + 1442695040888963407ull;
        const double u = (double)(s >> 11) * (1.0 / 9007199254740992.0);
        s = s * 6364136223846793005ull + 1442695040888963407ull;
        const double v = (double)(s >> 11) * (1.0 / 9007199254740992.0);
        const double a = (u - 0.5) * exp2(40.0 * v - 20.0);
        const double b = (v + 0.01) * exp2(40.0 * u - 20.0) * ((s >> 3) & 1 ? 1.0 : -1.0);
        const double q = a / b, qq = qdiv<double>(a, b);
        e64 = q != 0.0 ? fabs(qq - q) / fabs(q) : 0.0;
        const float af = (float)a, bf = (float)b;
        const float qf = af / bf, qqf = qdiv<float>(af, bf);
        e32 = qf != 0.0f ? fabs((double)qqf - (double)qf) / fabs((double)qf) : 0.0;
    }
    m64[threadIdx.x] = e64;
    m32[threadIdx.x] = e32;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) {
            m64[threadIdx.x] = fmax(m64[threadIdx.x], m64[threadIdx.x + o]);
            m32[threadIdx.x] = fmax(m32[threadIdx.x], m32[threadIdx.x + o]);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) { out[2 * blockIdx.x] = m64[0]; out[2 * blockIdx.x + 1] = m32[0]; }
}

// ------------------------------------------------------------------------------------
// Inverse mass on its own (DGBase::apply_inverse_global_mass_matrix, affine cells)
// ------------------------------------------------------------------------------------
template <int N1>
// metric != nullptr: curvilinear cDG cells, M^-1 = 1 / (W det J) per node (the weight-adjusted
// inverse of dg_base.cpp:4217-4249 on collocated GLL nodes)
// (curvilinear FR cells: the weight-adjusted B (x3) [ (1 / det J) (M+K)^-1 (x3) in ], fr != 0)
__global__ void inverse_mass_kernel(const double* __restrict__ in, double* __restrict__ out, const OpTab* ops,
                                    int nc, double inv_detj, const double* __restrict__ metric, int fr) {
    constexpr int NP = N1 * N1 * N1;
    __shared__ double s0[5 * NP], s1[5 * NP], sM[N1 * N1];
    const int cell = blockIdx.x;
    for (int i = threadIdx.x; i < N1 * N1; i += blockDim.x) sM[i] = ops->Minv[(i / N1) * MAXN1 + (i % N1)];
    for (int i = threadIdx.x; i < 5 * NP; i += blockDim.x) s0[i] = in[(size_t)cell * 5 * NP + i];
    double* src = s0; double* dst = s1;
    for (int d = 0; d < 3; ++d) {
        __syncthreads();
        const int st = (d == 0) ? 1 : (d == 1) ? N1 : N1 * N1;
        for (int i = threadIdx.x; i < 5 * NP; i += blockDim.x) {
            const int node = i % NP, s = i / NP;
            const int pos = (node / st) % N1, base = node - pos * st;
            double v = 0.0;
            for (int l = 0; l < N1; ++l) v += sM[pos * N1 + l] * src[s * NP + base + l * st];
            dst[i] = v;
        }
        double* t = src; src = dst; dst = t;
    }
    __syncthreads();
    if (metric && fr) {
        for (int i = threadIdx.x; i < 5 * NP; i += blockDim.x) src[i] *= metric[((size_t)cell * 10 + 9) * NP + i % NP];
        for (int i = threadIdx.x; i < N1 * N1; i += blockDim.x) sM[i] = ops->B[(i / N1) * MAXN1 + (i % N1)];
        for (int d = 0; d < 3; ++d) {
            __syncthreads();
            const int st = (d == 0) ? 1 : (d == 1) ? N1 : N1 * N1;
            for (int i = threadIdx.x; i < 5 * NP; i += blockDim.x) {
                const int node = i % NP, s = i / NP;
                const int pos = (node / st) % N1, base = node - pos * st;
                double v = 0.0;
                for (int l = 0; l < N1; ++l) v += sM[pos * N1 + l] * src[s * NP + base + l * st];
                dst[i] = v;
            }
            double* t = src; src = dst; dst = t;
        }
        __syncthreads();
        for (int i = threadIdx.x; i < 5 * NP; i += blockDim.x) out[(size_t)cell * 5 * NP + i] = src[i];
        return;
    }
    for (int i = threadIdx.x; i < 5 * NP; i += blockDim.x)
        out[(size_t)cell * 5 * NP + i] = src[i] * (metric ? metric[((size_t)cell * 10 + 9) * NP + i % NP] : inv_detj);
}

} // namespace ph
