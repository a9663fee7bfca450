// sm_100a kernels of the uncollocated strong-form DG/FR residual: solution on the (p+1)^3
// GLL support points of FE_DGQ(p), volume and face integrals on nq = p + 1 +
// overintegration flux nodes per direction (Gauss-Legendre, the reference's default
// flux_nodes_type, or Gauss-Lobatto with overintegration), affine periodic cells, FP64.
//
// Here the 1-D operators are dense: the interpolation chi (nq x nd) from the solution
// nodes to the flux nodes, its face rows, the entropy projection (chi M^-1 chi^T W), the
// flux-node differentiation and the FR mass inverse (M + K)^-1 with M = chi^T W chi. Every
// one is applied direction by direction (sum factorisation, operators.cpp:294-649): one thread
// per 1-D line holds the line in registers, and the operator, a kernel parameter, is read with
// compile-time indices (the extents are template arguments), so its entries are operands of
// the FMAs rather than memory loads.
//
// Three kernels per residual evaluation (one CTA per cell each):
//   gl_trace_kernel  the state's face values (chi_s (x) chi (x) chi U) and, for the split form, the
//                    states of the projected entropy variables at the face nodes and at the volume
//                    flux nodes (projected once, read by the other two kernels)
//   gl_aux_kernel    (Navier-Stokes; gl_aux_line_kernel on affine periodic cells) the lifted gradient q = (M_aux)^-1 [chi^T W D(chi u)
//                    + face (u* - u) n], kept at the flux nodes, then the viscous volume term
//                    W div(F_v) at the flux nodes, and per face node F_v(u, q) . n and the face-normal
//                    volume viscous flux
//   gl_stage_kernel  volume term (two-point split form with the skew operator on flux-node
//                    lines, or the conservative divergence), hybrid surface-volume two-point
//                    terms, numerical fluxes, lifts at the flux nodes, (M+K)^-1 folded into the last passes and
//                    the RK stage update
// The face data of a neighbour come from the buffers the earlier kernels wrote, so every
// face's numerical flux sees the same two states from either side.
//
// Reference structure restated (the oracle's Solver::assemble_residual follows the same lines):
//   auxiliary equation ................ src/dg/strong_dg.cpp:498-1008
//   volume term, split and conservative src/dg/strong_dg.cpp:1016-1579
//   entropy projection ................ src/dg/strong_dg.cpp:1235-1330, :3044-3142
//   hybrid surface-volume two-point ... src/dg/strong_dg.cpp:3144-3350
//   numerical fluxes and lifts ........ src/dg/strong_dg.cpp:3354-3576
//   inverse mass (affine) ............. src/dg/dg_base.cpp:4207-4219
#pragma once
#include "ph_kernels.cuh"
#include "ph_lines.cuh"

namespace ph {

constexpr int GL_MAXQ = 7;   // flux nodes per direction
constexpr int GL_MAXD = 7;   // solution nodes per direction

// 1-D operators, packed row-major with the actual sizes (nq, nd).
struct GlTab {
    double chi[GL_MAXQ * GL_MAXD];    // [q][i] solution basis l_i at flux node q
    double chis[2][GL_MAXD];          // solution basis at xi = 0 and xi = 1
    double phis[2][GL_MAXQ];          // flux-node Lagrange basis at xi = 0 and xi = 1
    double dphi[GL_MAXQ * GL_MAXQ];   // [q][l] derivative of flux-node basis l at flux node q
    double skew[GL_MAXQ * GL_MAXQ];   // S - S^T, S_ij = sum_q phi_i phi_j' w_q (operators.cpp:1440-1477)
    double wq[GL_MAXQ];               // flux-node weights on [0, 1]
    double P[GL_MAXQ * GL_MAXQ];      // chi M^-1 chi^T W: flux values -> projected -> flux values
    double haux[GL_MAXQ * GL_MAXQ];   // chi (M + K_aux)^-1 chi^T
    double pwa[GL_MAXD * GL_MAXQ];    // (M + K)^-1 chi^T W (nd x nq): the weight-adjusted inverse mass's projection
    double chm[GL_MAXQ * GL_MAXD];    // chi (M + K)^-1 (nq x nd): the transposed lift and the inverse mass in one
};

// Device buffers of the uncollocated path (per cell, reference units).
struct GlArgs {
    const GlTab* tab;
    double* t1;    // [nc][6][T1W][nq^2]: state at the face nodes (5), state of the projected entropy variables (5, split)
    double* t2;    // [nc][6][8][nq^2]: the cell's F_v(u, q) . e_dn at its face nodes (4) and its face-normal
                   // volume viscous flux interpolated to them, signed by the side (4)
    double* vis;   // [nc][4][nq^3]: W div(F_v) at the flux nodes, momentum and energy rows
    // curvilinear cells (nullptr on affine ones): at the volume flux nodes [nc][10][nq^3] the
    // cofactor C[k][d] (row k * 3 + d) and 1 / det J (row 9); at each face's flux nodes
    // [nc][6][3][nq^2] the face's metric column C[:, f / 2]
    const double* vmet;
    const double* fnrm;
    // boundary faces of a non-periodic mesh (nbr = -1 - k, a.btype[k]): [nb][4][nq^2] the outward
    // boundary viscous flux F*_v . n at the face nodes, written by the auxiliary kernel
    double* fb;
    double* proj;  // split form: [nc][5][nq^3] the state of the projected entropy variables at the flux nodes
};

// Boundary faces (out of line: only boundary face nodes call them, and the periodic path keeps its
// register allocation). The viscous boundary state of a face node (component s) from the cell's own
// face values (stride NF), for the auxiliary equation's lift.
static __device__ __noinline__ double gl_bnd_visc_state(int bt, const double* own, int NF, int s,
                                                        const PhysConst& pc) {
    double u[5], ub[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) u[k] = __ldg(&own[k * NF]);
    boundary_viscous_state<double>(bt, u, pc, ub, nullptr);
    return s == 0 ? ub[0] : s == 1 ? ub[1] : s == 2 ? ub[2] : s == 3 ? ub[3] : ub[4];
}
// The outward boundary viscous flux at a face node of face f (evaluate_auxiliary_flux on a boundary,
// viscous_numerical_flux.cpp:66-328): the viscous boundary state of us (the interpolated face state r,
// or the projected one), BR2 / SIPG with its gradient, the central flux with the interior one, no heat
// flux on an adiabatic 1001 wall; the interior side is r.
// Curvilinear faces (m = the face's metric column C[:, f / 2] at the node, else nullptr): the outward
// unit normal sg m / |m| and the flux scaled by |m|.
static __device__ __noinline__ void gl_bnd_visc_flux(int bt, const double r[5], const double us[5],
                                                     const double g[5][3], int f, const PhysConst& pc, double pen,
                                                     double out[4], const double* m) {
    Cst<double> cst; cst.load(pc);
    const int dn = f >> 1;
    const double sg = (f & 1) ? 1.0 : -1.0;
    double ub[5];
    boundary_viscous_state<double>(bt, us, pc, ub, nullptr);
    if (m) {
        const double Jf = sqrt(m[0] * m[0] + m[1] * m[1] + m[2] * m[2]);
        const double nv[3] = {sg * m[0] / Jf, sg * m[1] / Jf, sg * m[2] / Jf};
        const bool ad = bt == BC_WALL && !pc.bc_isothermal;
        double gb[5][3];
        for (int s = 0; s < 5; ++s)
            for (int e = 0; e < 3; ++e) gb[s][e] = (ad && s == 4) ? 0.0 : g[s][e];
        double Fi[3][4], Fe[3][4];
        viscous_flux<double>(r, g, pc.use_const_visc, cst, Fi, 7, nullptr, ad);
        viscous_flux<double>(ub, pc.diss_flux == DF_CENTRAL ? g : gb, pc.use_const_visc, cst, Fe, 7, nullptr, ad);
        for (int k = 0; k < 4; ++k) {
            const double fi = Fi[0][k] * nv[0] + Fi[1][k] * nv[1] + Fi[2][k] * nv[2];
            const double fe = Fe[0][k] * nv[0] + Fe[1][k] * nv[1] + Fe[2][k] * nv[2];
            out[k] = Jf * (0.5 * (fi + fe));
        }
        return;
    }
    const bool ad = bt == BC_WALL && !pc.bc_isothermal;
    double gb[5][3];
    for (int s = 0; s < 5; ++s)
        for (int e = 0; e < 3; ++e) gb[s][e] = (ad && s == 4) ? 0.0 : g[s][e];
    double Fi[3][4], Fe[3][4];
    viscous_flux<double>(r, g, pc.use_const_visc, cst, Fi, 7, nullptr, ad);
    viscous_flux<double>(ub, pc.diss_flux == DF_CENTRAL ? g : gb, pc.use_const_visc, cst, Fe, 7, nullptr, ad);
    for (int k = 0; k < 4; ++k) out[k] = 0.5 * (sg * Fi[dn][k] + sg * Fe[dn][k]);
    if (pc.diss_flux == DF_SIPG) {
        double J[5][3];
        for (int s = 0; s < 5; ++s)
            for (int e = 0; e < 3; ++e) J[s][e] = (e == dn) ? (r[s] - ub[s]) * sg : 0.0;
        viscous_flux<double>(r, J, pc.use_const_visc, cst, Fi, 7, nullptr, ad);
        viscous_flux<double>(ub, J, pc.use_const_visc, cst, Fe, 7, nullptr, ad);
        for (int k = 0; k < 4; ++k) out[k] = out[k] - pen * (0.5 * (sg * Fi[dn][k] + sg * Fe[dn][k]));
    }
}
// The convective boundary state of a face node (Euler::boundary_face_values) for outward normal
// sg e_dn of face f.
static __device__ __noinline__ void gl_bnd_state(int bt, const double r[5], int f, const PhysConst& pc,
                                                 double ub[5], unsigned* st, const double* nv = nullptr) {
    const int dn = f >> 1;
    const double sg = (f & 1) ? 1.0 : -1.0;
    double nrm[3] = {dn == 0 ? sg : 0.0, dn == 1 ? sg : 0.0, dn == 2 ? sg : 0.0};
    if (nv) { nrm[0] = sg * nv[0]; nrm[1] = sg * nv[1]; nrm[2] = sg * nv[2]; }   // curvilinear: sg times the unit m
    boundary_state<double>(bt, nrm, r, pc, ub, st);
}

template <bool SPLIT> __host__ __device__ constexpr int gl_t1_width() { return SPLIT ? 10 : 5; }
constexpr int GL_T2W = 8;

#ifndef PH_GL_PREFETCH
#define PH_GL_PREFETCH 1
#endif

// L2 prefetch of n doubles at p, one per 128-byte line, addresses clamped inside [p, p + n)
__device__ __forceinline__ void gl_prefetch_span(const double* p, int n, int i0, int stride) {
    const int nl = (n + 15) / 16;
    for (int i = i0; i < nl; i += stride) {
        const int e = i * 16;
        asm volatile("prefetch.global.L2 [%0];" ::"l"(p + (e < n ? e : n - 1)));
    }
}

// Warms L2 with the data a cell reads after its volume work: the neighbours' blocks of the
// face-value buffer (the auxiliary kernel: their states; the stage kernel: the whole blocks), and
// in the stage kernel its own face-value blocks, its own and its neighbours' viscous face blocks,
// its viscous volume rows and the RK registers of the epilogue. Each block is one the kernel
// itself reads; a prefetch writes nothing. Boundary faces (nbr < 0) have no neighbour block.
template <int NT, int NF, int D3, int Q3, int T1W, bool STAGE, bool VISC>
__device__ __forceinline__ void gl_prefetch_l2(const StageArgs& a, const GlArgs& g, int cell) {
    if (!PH_GL_PREFETCH) return;
    const int w = threadIdx.x >> 5, nw = NT / 32, lane = threadIdx.x & 31;
    // warp w takes the blocks w, w + nw, ...: 6 neighbour face-value blocks, then (stage: viscous)
    // 6 neighbour viscous face blocks, the own blocks, (viscous) the viscous rows, the RK registers
    constexpr int NB = STAGE ? 6 + (VISC ? 6 : 0) + 1 + (VISC ? 2 : 0) + 2 : 6;
    for (int b = w; b < NB; b += nw) {
        const double* p = nullptr;
        int n = 0;
        if (b < 6) {
            const int cn = __ldg(&a.nbr[cell * 6 + b]);
            if (cn >= 0) { p = g.t1 + ((size_t)cn * 6 + (b ^ 1)) * T1W * NF; n = (STAGE ? T1W : 5) * NF; }
        } else if (STAGE && VISC && b < 12) {
            const int f = b - 6, cn = __ldg(&a.nbr[cell * 6 + f]);
            if (cn >= 0) { p = g.t2 + ((size_t)cn * 6 + (f ^ 1)) * GL_T2W * NF; n = GL_T2W * NF; }
        } else {
            const int r = b - (STAGE && VISC ? 12 : 6);
            if (r == 0) { p = g.t1 + (size_t)cell * 6 * T1W * NF; n = 6 * T1W * NF; }
            else if (STAGE && VISC && r == 1) { p = g.t2 + (size_t)cell * 6 * GL_T2W * NF; n = 6 * GL_T2W * NF; }
            else if (STAGE && VISC && r == 2) { p = g.vis + (size_t)cell * 4 * Q3; n = 4 * Q3; }
            else if (STAGE && a.mode == 2) {
                const int k = r - (VISC ? 3 : 1);
                const double* base = k == 0 ? a.Un : a.acc_in;
                if (base) { p = base + (size_t)cell * 5 * D3; n = 5 * D3; }
            }
        }
        if (p) gl_prefetch_span(p, n, lane, 32);
    }
}

// temporaries of the sum-factorised passes on 5 components (and of the six faces' arrays)
template <int ND, int NQ> __host__ __device__ constexpr int gl_temp() {
    constexpr int a = 5 * NQ * NQ * NQ, b = 30 * NQ * NQ, c = 30 * NQ * ND, d = 30 * ND * ND;
    constexpr int ab = a > b ? a : b, cd = c > d ? c : d;
    return ab > cd ? ab : cd;
}

template <int NQ> __host__ __device__ constexpr int gl_threads() {
    return NQ * NQ * NQ <= 64 ? 64 : NQ * NQ * NQ <= 128 ? 128 : 256;
}

// Entropy variables of a conservative state (Euler::compute_entropy_variables, euler.cpp:811-830)
// and the conservative state of entropy variables (:833-855), FP64. The powers are taken through
// logarithms: s = log(p rho^-gamma) = log p - gamma log rho, and
// rho e = (gm1 / (-v4)^gamma)^(1/gm1) exp(-s / gm1) = exp((log gm1 - gamma log(-v4) - s) / gm1),
// one exponential and one or two logarithms instead of the powers' own logarithm-exponential
// pairs (the same values to rounding).
__device__ __forceinline__ void gl_entropy_vars(const double u[5], double gam, double gm1, double v[5],
                                                unsigned* st) {
    const double rho = u[0];
    double v2 = 0.0;
#pragma unroll
    for (int d = 0; d < 3; ++d) { const double w = u[1 + d] / rho; v2 = v2 + w * w; }
    const double p = positive<double>(gm1 * (u[4] - 0.5 * rho * v2), st);
    const double s = log(p) - gam * log(rho);
    const double rt = p / gm1;
    const double irt = 1.0 / rt;
    v[0] = (rt * (gam + 1.0 - s) - u[4]) * irt;
#pragma unroll
    for (int d = 0; d < 3; ++d) v[1 + d] = u[1 + d] * irt;
    v[4] = -rho * irt;
}
__device__ __forceinline__ void gl_cons_from_entropy(const double v[5], double gam, double gm1, double u[5]) {
    double vv = 0.0;
#pragma unroll
    for (int d = 0; d < 3; ++d) vv += v[1 + d] * v[1 + d];
    const double iv4 = 1.0 / v[4];
    const double s = gam - v[0] + 0.5 * vv * iv4;
    const double rt = exp((log(gm1) - gam * log(-v[4]) - s) / gm1);
    u[0] = -rt * v[4];
#pragma unroll
    for (int d = 0; d < 3; ++d) u[1 + d] = rt * v[1 + d];
    u[4] = rt * (1.0 - 0.5 * vv * iv4);
}

// One sum-factorised pass along direction d: out[s][o] (+)= scale * sum_l A[r * cols + l] in[s][o, r -> l]
// with r the output's coordinate along d. Input dims (n0, n1, n2), n_d = cols; output dims the
// same with n_d = rows. x is the fastest index.
template <int NT>
__device__ __forceinline__ void gl_pass(const double* A, int rows, int cols, int d, int n0, int n1, int n2,
                                            const double* in, int in_ss, double* out, int out_ss, int ns,
                                            double scale, bool acc) {
    const int m0 = d == 0 ? rows : n0, m1 = d == 1 ? rows : n1, m2 = d == 2 ? rows : n2;
    const int osz = m0 * m1 * m2;
    const int st = d == 0 ? 1 : d == 1 ? n0 : n0 * n1;
    for (int it = threadIdx.x; it < ns * osz; it += NT) {
        const int s = it / osz, o = it - s * osz;
        const int x = o % m0, y = (o / m0) % m1, z = o / (m0 * m1);
        const int r = d == 0 ? x : d == 1 ? y : z;
        const int base = ((d == 2 ? 0 : z) * n1 + (d == 1 ? 0 : y)) * n0 + (d == 0 ? 0 : x);
        const double* ip = in + s * in_ss + base;
        const double* ar = A + r * cols;
        double v = 0.0;
        for (int l = 0; l < cols; ++l) v += ar[l] * ip[l * st];
        double* op = out + s * out_ss + o;
        *op = acc ? *op + scale * v : scale * v;
    }
}

// ------------------------------------------------------------------------------------
// Compile-time sum-factorised passes
// ------------------------------------------------------------------------------------
// One pass along direction D of NS arrays with input extents (N0, N1, N2), N_D = COLS, and
// output extents the same with N_D = ROWS (x fastest): one thread per line reads the COLS
// inputs into registers and writes out[o] (+)= scale * sum_l A(o, l) in[l] for each of the ROWS
// outputs, A(o, l) = A[o * COLS + l], or A[l * ROWS + o] with TRANS (the transposed operator
// stored as cols x rows). Summation in ascending l from zero. A line's inputs are all read
// before its outputs are written, so in == out is allowed when ROWS == COLS.
template <int NT, int ROWS, int COLS, int D, int N0, int N1, int N2, int NS, bool TRANS = false>
__device__ __forceinline__ void gl_line(const double* __restrict__ A, const double* in, int in_ss, double* out,
                                        int out_ss, double scale, bool acc) {
    static_assert((D == 0 ? N0 : D == 1 ? N1 : N2) == COLS, "the input extent along D is COLS");
    constexpr int PA = D == 0 ? N1 : N0, PB = D == 2 ? N1 : N2;   // the other two extents, lower first
    constexpr int IST = D == 0 ? 1 : D == 1 ? N0 : N0 * N1;
    constexpr int M0 = D == 0 ? ROWS : N0, M1 = D == 1 ? ROWS : N1;
    constexpr int OST = D == 0 ? 1 : D == 1 ? M0 : M0 * M1;
    constexpr int NL = NS * PA * PB;
#pragma unroll 1
    for (int t = threadIdx.x; t < NL; t += NT) {
        const int s = t / (PA * PB), r = t - s * (PA * PB);
        const int ca = r % PA, cb = r / PA;
        int ib, ob;
        if constexpr (D == 0) { ib = (cb * N1 + ca) * N0; ob = (cb * M1 + ca) * M0; }
        else if constexpr (D == 1) { ib = cb * N1 * N0 + ca; ob = cb * M1 * M0 + ca; }
        else { ib = cb * N0 + ca; ob = ib; }
        const double* ip = in + s * in_ss + ib;
        double* op = out + s * out_ss + ob;
        double v[COLS];
#pragma unroll
        for (int l = 0; l < COLS; ++l) v[l] = ip[l * IST];
#pragma unroll
        for (int o = 0; o < ROWS; ++o) {
            double x = 0.0;
#pragma unroll
            for (int l = 0; l < COLS; ++l) x += (TRANS ? A[l * ROWS + o] : A[o * COLS + l]) * v[l];
            op[o * OST] = acc ? op[o * OST] + scale * x : scale * x;
        }
    }
}

// out = (A (x) A (x) A) in, x first (TRANS: the transpose of A stored NI x NO): input cubes of
// NI per direction, output NO per direction; t0, t1 hold NS NO NI^2 and NS NO^2 NI values.
// Ends with a barrier.
template <int NT, int NO, int NI, int NS, bool TRANS = false>
__device__ __forceinline__ void gl_apply3(const double* A, const double* in, int in_ss, double* out, int out_ss,
                                          double* t0, double* t1, double scale, bool acc) {
    constexpr int S0 = NO * NI * NI, S1 = NO * NO * NI;
    gl_line<NT, NO, NI, 0, NI, NI, NI, NS, TRANS>(A, in, in_ss, t0, S0, 1.0, false);
    __syncthreads();
    gl_line<NT, NO, NI, 1, NO, NI, NI, NS, TRANS>(A, t0, S0, t1, S1, 1.0, false);
    __syncthreads();
    gl_line<NT, NO, NI, 2, NO, NO, NI, NS, TRANS>(A, t1, S1, out, out_ss, scale, acc);
    __syncthreads();
}

// node index of position l along direction dn on the face-node line q2 = t2 * N + t1 (t1 < t2
// the tangential directions: the face-node order of both sides of a face)
template <int N> __device__ __forceinline__ int gl_line_node(int dn, int q2, int l) {
    const int t1c = q2 % N, t2c = q2 / N;
    return dn == 0 ? (t2c * N + t1c) * N + l : dn == 1 ? (t2c * N + l) * N + t1c : (l * N + t2c) * N + t1c;
}

// The two end values of a line of flux-node values: the flux-node basis at xi = 0 and 1. The solution
// basis is interpolated exactly by the flux-node basis (chis[side] = chi^T phis[side]), so a face value of a
// discrete function is one contraction along the normal of its flux-node values, and a face array is
// lifted by adding phis[side][l] times it to the flux-node array whose chi^T (x3) follows.
template <int NQ>
__device__ __forceinline__ void gl_line_ends(const GlTab& T, const double* ip, int st, double& v0, double& v1) {
    v0 = v1 = 0.0;
#pragma unroll
    for (int l = 0; l < NQ; ++l) {
        const double x = ip[l * st];
        v0 += T.phis[0][l] * x;
        v1 += T.phis[1][l] * x;
    }
}
// first node of line `line` (face-node order q2) along direction d and the line's stride
template <int NQ> __device__ __forceinline__ int gl_line_base(int d, int line, int& st) {
    const int a = line % NQ, b = line / NQ;
    st = d == 0 ? 1 : d == 1 ? NQ : NQ * NQ;
    return d == 0 ? NQ * line : d == 1 ? a + NQ * NQ * b : line;
}

// Shared-memory copy of the operator table (for the reads with run-time indices).
__device__ __forceinline__ void gl_load_tab(const GlTab* g, GlTab* s, int nt) {
    const double* src = reinterpret_cast<const double*>(g);
    double* dst = reinterpret_cast<double*>(s);
    for (int i = threadIdx.x; i < (int)(sizeof(GlTab) / sizeof(double)); i += nt) dst[i] = src[i];
}

// ------------------------------------------------------------------------------------
// Face values of the state (and of the projected entropy variables)
// ------------------------------------------------------------------------------------
template <int ND, int NQ, bool SPLIT>
struct GlTraceLayout {
    // the lines of five rows in one pass (80 at NQ = 4, 180 at NQ = 6)
    static constexpr int NT = NQ == 4 ? 96 : NQ == 6 ? 192 : gl_threads<NQ>();
    static constexpr int D3 = ND * ND * ND, Q3 = NQ * NQ * NQ;
    static constexpr int oQ = 0;                                    // 5 NQ^3 (flux-node values / entropy variables)
    static constexpr int nW = 5 * Q3;
    static constexpr int oW0 = oQ + 5 * Q3, oW1 = oW0 + nW;
    static constexpr int total = oW1 + nW;
    static constexpr size_t bytes = (size_t)total * sizeof(double);
};

template <int ND, int NQ, bool SPLIT>
__global__ void __launch_bounds__(GlTraceLayout<ND, NQ, SPLIT>::NT)
gl_trace_kernel(const StageArgs a, const GlArgs g, const __grid_constant__ GlTab T) {
    using L = GlTraceLayout<ND, NQ, SPLIT>;
    constexpr int NT = L::NT, D3 = L::D3, Q3 = L::Q3, NF = NQ * NQ, T1W = gl_t1_width<SPLIT>();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* sm = reinterpret_cast<double*>(smem_raw);
    double* sQ = sm + L::oQ;
    double* w0 = sm + L::oW0;
    double* w1 = sm + L::oW1;
    const int cell = a.cell_begin + blockIdx.x;
    for (int i = threadIdx.x; i < 5 * D3; i += NT) sQ[i] = __ldg(&a.U[(size_t)cell * 5 * D3 + i]);
    __syncthreads();
    gl_apply3<NT, NQ, ND, 5>(T.chi, sQ, D3, sQ, Q3, w0, w1, 1.0, false);
    double* out = g.t1 + (size_t)cell * 6 * T1W * NF;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        for (int it = threadIdx.x; it < 5 * NF; it += NT) {
            const int s = it / NF, line = it - s * NF;
            int st;
            const int base = gl_line_base<NQ>(d, line, st);
            double v0, v1;
            gl_line_ends<NQ>(T, sQ + s * Q3 + base, st, v0, v1);
            out[((2 * d) * T1W + s) * NF + line] = v0;
            out[((2 * d + 1) * T1W + s) * NF + line] = v1;
        }
    }
    if constexpr (SPLIT) {
        const double gam = a.pc.gam, gm1 = a.pc.gm1;
        __syncthreads();
        for (int q = threadIdx.x; q < Q3; q += NT) {
            double u[5], v[5];
#pragma unroll
            for (int s = 0; s < 5; ++s) u[s] = sQ[s * Q3 + q];
            gl_entropy_vars(u, gam, gm1, v, a.status);
#pragma unroll
            for (int s = 0; s < 5; ++s) sQ[s * Q3 + q] = v[s];
        }
        __syncthreads();
        gl_apply3<NT, NQ, NQ, 5>(T.P, sQ, Q3, sQ, Q3, w0, w1, 1.0, false);
        for (int it = threadIdx.x; it < Q3 + 3 * NF; it += NT) {
            if (it < Q3) {
                double v[5], u[5];
#pragma unroll
                for (int s = 0; s < 5; ++s) v[s] = sQ[s * Q3 + it];
                gl_cons_from_entropy(v, gam, gm1, u);
#pragma unroll
                for (int s = 0; s < 5; ++s) g.proj[((size_t)cell * 5 + s) * Q3 + it] = u[s];
            } else {   // the two face nodes of a line
                const int d = (it - Q3) / NF, line = (it - Q3) - d * NF;
                int st;
                const int base = gl_line_base<NQ>(d, line, st);
                double v[2][5], u[5];
#pragma unroll
                for (int s = 0; s < 5; ++s) gl_line_ends<NQ>(T, sQ + s * Q3 + base, st, v[0][s], v[1][s]);
#pragma unroll
                for (int side = 0; side < 2; ++side) {
                    gl_cons_from_entropy(v[side], gam, gm1, u);
#pragma unroll
                    for (int s = 0; s < 5; ++s) out[((2 * d + side) * T1W + 5 + s) * NF + line] = u[s];
                }
            }
        }
    }
}

// ------------------------------------------------------------------------------------
// Auxiliary equation and the viscous terms (Navier-Stokes)
// ------------------------------------------------------------------------------------
// The lifted gradient is formed at the flux nodes: with H = chi (M + K_aux)^-1 chi^T and
// chi_side = chi^T phi_side (the solution basis is interpolated exactly by the flux-node basis),
//   chi (x3) q_d = (1/h) (H (x) H (x) H) [W D_d (chi u) + sum_side phi_side (x) W_face (u* - u) n_d]
// which is the reference's q_d = (M_aux)^-1 [chi^T W D_d (chi u) + face lifts] taken to the
// flux nodes (strong_dg.cpp:498-1008, dg_base.cpp:4089-4260 with use_auxiliary_eq; C = h^2 I):
// four passes per direction instead of ten. The face values of q are the flux-node values along
// the normal contracted with phi_side (exact for the degree-p gradient).
template <int ND, int NQ, bool SPLIT>
struct GlAuxLayout {
    static constexpr int NT = gl_threads<NQ>();
    static constexpr int D3 = ND * ND * ND, Q3 = NQ * NQ * NQ, NF = NQ * NQ;
    static constexpr int nTab = (int)(sizeof(GlTab) / sizeof(double));
    static constexpr int oU = nTab;                      // 5 NQ^3: the state, later the projected state
    static constexpr int oQ = oU + 5 * Q3;               // 5 NQ^3: state at the flux nodes
    static constexpr int oAQ = oQ + 5 * Q3;              // 15 NQ^3: lifted gradient at the flux nodes
    static constexpr int oF = oAQ + 15 * Q3;             // 12 NQ^3: volume viscous flux
    static constexpr int nT = gl_temp<ND, NQ>();
    static constexpr int oT0 = oF + 12 * Q3, oT1 = oT0 + nT;
    static constexpr int total = oT1 + nT;
    static constexpr size_t bytes = (size_t)total * sizeof(double);
    static_assert(nT >= 30 * NF, "the six faces' terms fit a temporary");
};

// the lifted gradient of all three directions at once (see above), into sAQ[s * 3 + d][Q3]:
// the flux-node derivatives, the six faces' terms, the brackets, then H (x) H (x) H as three
// passes over all fifteen components in place (H is square: each line is read whole before it
// is written). Ends with a barrier.
template <int ND, int NQ, bool SPLIT, bool CURV = false, bool BND = false>
__device__ __forceinline__ void gl_aux_gradient(const StageArgs& a, const GlArgs& g, const GlTab& T,
                                                const GlTab* tab, int cell, const double* sQ, double* face,
                                                double* sAQ) {
    using L = GlAuxLayout<ND, NQ, SPLIT>;
    constexpr int NT = L::NT, Q3 = L::Q3, NF = L::NF, T1W = gl_t1_width<SPLIT>();
    gl_line<NT, NQ, NQ, 0, NQ, NQ, NQ, 5>(T.dphi, sQ, Q3, sAQ + 0 * Q3, 3 * Q3, 1.0, false);
    gl_line<NT, NQ, NQ, 1, NQ, NQ, NQ, 5>(T.dphi, sQ, Q3, sAQ + 1 * Q3, 3 * Q3, 1.0, false);
    gl_line<NT, NQ, NQ, 2, NQ, NQ, NQ, 5>(T.dphi, sQ, Q3, sAQ + 2 * Q3, 3 * Q3, 1.0, false);
    for (int it = threadIdx.x; it < 6 * 5 * NF; it += NT) {   // face[f][s][q2] = W_face (u* - u) n_{f/2}
        const int f = it / (5 * NF), s = (it / NF) % 5, q2 = it % NF;
        const int cn = __ldg(&a.nbr[cell * 6 + f]);
        const double uo = __ldg(&g.t1[(((size_t)cell * 6 + f) * T1W + s) * NF + q2]);
        const double ue = (!BND || cn >= 0) ? __ldg(&g.t1[(((size_t)cn * 6 + (f ^ 1)) * T1W + s) * NF + q2])
                                            : gl_bnd_visc_state(__ldg(&a.btype[-1 - cn]),
                                                                g.t1 + ((size_t)cell * 6 + f) * T1W * NF + q2, NF, s,
                                                                a.pc);
        const double sgn = (f & 1) ? 1.0 : -1.0;
        face[it] = tab->wq[q2 % NQ] * tab->wq[q2 / NQ] * ((0.5 * (uo + ue) - uo) * sgn);
    }
    __syncthreads();
    if constexpr (CURV) {
        // physical components: W sum_j C[d][j] D_j u at the volume flux nodes, and every face's
        // lift (u* - u) (C_face[:, dn])_d (each face reaches every component on a curved cell)
        const double* vm = g.vmet + (size_t)cell * 10 * Q3;
        const double* fm = g.fnrm + (size_t)cell * 18 * NF;
        for (int i = threadIdx.x; i < 5 * Q3; i += NT) {
            const int s = i / Q3, q = i - s * Q3;
            const int c[3] = {q % NQ, (q / NQ) % NQ, q / NF};
            const double W = tab->wq[c[0]] * tab->wq[c[1]] * tab->wq[c[2]];
            double r[3], b[3];
#pragma unroll
            for (int j = 0; j < 3; ++j) r[j] = sAQ[(s * 3 + j) * Q3 + q];
#pragma unroll
            for (int d = 0; d < 3; ++d)
                b[d] = W * (__ldg(&vm[(d * 3 + 0) * Q3 + q]) * r[0] + __ldg(&vm[(d * 3 + 1) * Q3 + q]) * r[1] +
                            __ldg(&vm[(d * 3 + 2) * Q3 + q]) * r[2]);
#pragma unroll
            for (int dn = 0; dn < 3; ++dn) {
                const int a1 = dn == 0 ? 1 : 0, a2 = dn == 2 ? 1 : 2;
                const int q2 = c[a2] * NQ + c[a1];
                const double l0 = tab->phis[0][c[dn]] * face[((2 * dn) * 5 + s) * NF + q2];
                const double l1 = tab->phis[1][c[dn]] * face[((2 * dn + 1) * 5 + s) * NF + q2];
#pragma unroll
                for (int d = 0; d < 3; ++d)
                    b[d] += l0 * __ldg(&fm[((2 * dn) * 3 + d) * NF + q2]) + l1 * __ldg(&fm[((2 * dn + 1) * 3 + d) * NF + q2]);
            }
#pragma unroll
            for (int d = 0; d < 3; ++d) sAQ[(s * 3 + d) * Q3 + q] = b[d];
        }
        __syncthreads();
        // the weight-adjusted inverse at the flux nodes: H (x3) [ (W / det J) H (x3) b ]
        gl_line<NT, NQ, NQ, 0, NQ, NQ, NQ, 15>(T.haux, sAQ, Q3, sAQ, Q3, 1.0, false);
        __syncthreads();
        gl_line<NT, NQ, NQ, 1, NQ, NQ, NQ, 15>(T.haux, sAQ, Q3, sAQ, Q3, 1.0, false);
        __syncthreads();
        gl_line<NT, NQ, NQ, 2, NQ, NQ, NQ, 15>(T.haux, sAQ, Q3, sAQ, Q3, 1.0, false);
        __syncthreads();
        for (int i = threadIdx.x; i < 15 * Q3; i += NT) {
            const int q = i % Q3;
            sAQ[i] *= tab->wq[q % NQ] * tab->wq[(q / NQ) % NQ] * tab->wq[q / NF] * __ldg(&vm[9 * Q3 + q]);
        }
        __syncthreads();
        gl_line<NT, NQ, NQ, 0, NQ, NQ, NQ, 15>(T.haux, sAQ, Q3, sAQ, Q3, 1.0, false);
        __syncthreads();
        gl_line<NT, NQ, NQ, 1, NQ, NQ, NQ, 15>(T.haux, sAQ, Q3, sAQ, Q3, 1.0, false);
        __syncthreads();
        gl_line<NT, NQ, NQ, 2, NQ, NQ, NQ, 15>(T.haux, sAQ, Q3, sAQ, Q3, 1.0, false);
        __syncthreads();
        return;
    }
    for (int i = threadIdx.x; i < 15 * Q3; i += NT) {
        const int k = i / Q3, q = i - k * Q3, s = k / 3, d = k - 3 * s;
        const int c[3] = {q % NQ, (q / NQ) % NQ, q / NF};
        const int a1 = d == 0 ? 1 : 0, a2 = d == 2 ? 1 : 2;
        const int q2 = c[a2] * NQ + c[a1];
        sAQ[i] = tab->wq[c[0]] * tab->wq[c[1]] * tab->wq[c[2]] * sAQ[i] +
                 tab->phis[0][c[d]] * face[((2 * d) * 5 + s) * NF + q2] +
                 tab->phis[1][c[d]] * face[((2 * d + 1) * 5 + s) * NF + q2];
    }
    __syncthreads();
    gl_line<NT, NQ, NQ, 0, NQ, NQ, NQ, 15>(T.haux, sAQ, Q3, sAQ, Q3, 1.0, false);
    __syncthreads();
    gl_line<NT, NQ, NQ, 1, NQ, NQ, NQ, 15>(T.haux, sAQ, Q3, sAQ, Q3, 1.0, false);
    __syncthreads();
    gl_line<NT, NQ, NQ, 2, NQ, NQ, NQ, 15>(T.haux, sAQ, Q3, sAQ, Q3, a.inv_h, false);
    __syncthreads();
}

// the contravariant viscous flux F~_j = sum_m C[m][j] F_m at volume flux node q (curvilinear)
__device__ __forceinline__ void gl_contravariant(const double* vm, int q, int Q3, double F[3][4]) {
    double C[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) C[i] = __ldg(&vm[i * Q3 + q]);
    double Ft[3][4];
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int k = 0; k < 4; ++k) Ft[j][k] = C[0 * 3 + j] * F[0][k] + C[1 * 3 + j] * F[1][k] + C[2 * 3 + j] * F[2][k];
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int k = 0; k < 4; ++k) F[j][k] = Ft[j][k];
}

// CURV: curvilinear cells (the metric at the flux nodes, g.vmet / g.fnrm): the physical
// gradient through the weight-adjusted inverse (gl_aux_gradient), contravariant volume fluxes,
// and each face node's F_v . C_face[:, dn] (the metric-scaled normal flux)
// BND: the cells with a boundary face (a tile list of them), the boundary states in the lift and the
// boundary viscous fluxes stored for the stage kernel
template <int ND, int NQ, bool SPLIT, bool CURV = false, bool BND = false>
__global__ void __launch_bounds__(gl_threads<NQ>(), 2)
gl_aux_kernel(const StageArgs a, const GlArgs g, const __grid_constant__ GlTab T) {
    using L = GlAuxLayout<ND, NQ, SPLIT>;
    constexpr int NT = L::NT, D3 = L::D3, Q3 = L::Q3, NF = L::NF, T1W = gl_t1_width<SPLIT>();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* sm = reinterpret_cast<double*>(smem_raw);
    GlTab* tab = reinterpret_cast<GlTab*>(sm);
    double* sU = sm + L::oU;
    double* sQ = sm + L::oQ;
    double* sAQ = sm + L::oAQ;
    double* sF = sm + L::oF;
    double* t0 = sm + L::oT0;
    double* t1 = sm + L::oT1;
    const int cell = a.tiles ? __ldg(&a.tiles[blockIdx.x]) : a.cell_begin + (int)blockIdx.x;
    Cst<double> cst; cst.load(a.pc);
    const int ucv = a.pc.use_const_visc;
    gl_load_tab(g.tab, tab, NT);
    for (int i = threadIdx.x; i < 5 * D3; i += NT) sU[i] = __ldg(&a.U[(size_t)cell * 5 * D3 + i]);
    gl_prefetch_l2<NT, NF, D3, Q3, T1W, false, true>(a, g, cell);
    __syncthreads();
    gl_apply3<NT, NQ, ND, 5>(T.chi, sU, D3, sQ, Q3, t0, t1, 1.0, false);
    gl_aux_gradient<ND, NQ, SPLIT, CURV, BND>(a, g, T, tab, cell, sQ, t0, sAQ);
    const double* vm = CURV ? g.vmet + (size_t)cell * 10 * Q3 : nullptr;
    // per face node of the cell: F_v(u, q) . e_dn with the state's and the gradient's face values
    // (each side's half of the dissipative numerical flux, strong_dg.cpp:3354-3452)
    double* tout = g.t2 + (size_t)cell * 6 * GL_T2W * NF;
    for (int it = threadIdx.x; it < 6 * NF; it += NT) {
        const int f = it / NF, q2 = it - f * NF, dn = f >> 1, side = f & 1;
        const double* rw = tab->phis[side];
        double gq[5][3], r[5];
#pragma unroll
        for (int s = 0; s < 5; ++s) {
            r[s] = __ldg(&g.t1[(((size_t)cell * 6 + f) * T1W + s) * NF + q2]);
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const double* row = sAQ + (s * 3 + d) * Q3;
                double v = 0.0;
#pragma unroll
                for (int l = 0; l < NQ; ++l) v += rw[l] * row[gl_line_node<NQ>(dn, q2, l)];
                gq[s][d] = v;
            }
        }
        if constexpr (BND) {   // a boundary face: its outward boundary viscous flux for the stage kernel
            const int cn = __ldg(&a.nbr[cell * 6 + f]);
            if (cn < 0) {
                double us[5], out[4];
#pragma unroll
                for (int s = 0; s < 5; ++s) us[s] = r[s];
                if (SPLIT && a.pc.bc_projected) {   // the face state of the projected entropy variables
#pragma unroll
                    for (int s = 0; s < 5; ++s) us[s] = __ldg(&g.t1[(((size_t)cell * 6 + f) * T1W + 5 + s) * NF + q2]);
                }
                double mc[3];
                if constexpr (CURV) {
                    const double* m = g.fnrm + ((size_t)cell * 6 + f) * 3 * NF + q2;
                    mc[0] = __ldg(&m[0]); mc[1] = __ldg(&m[NF]); mc[2] = __ldg(&m[2 * NF]);
                }
                gl_bnd_visc_flux(__ldg(&a.btype[-1 - cn]), r, us, gq, f, a.pc, a.pen, out, CURV ? mc : nullptr);
#pragma unroll
                for (int k = 0; k < 4; ++k) g.fb[((size_t)(-1 - cn) * 4 + k) * NF + q2] = out[k];
            }
        }
        double F[3][4];
        if constexpr (CURV) {   // F_v . C_face[:, dn]
            viscous_flux<double>(r, gq, ucv, cst, F, 7, nullptr);
            const double* m = g.fnrm + ((size_t)cell * 6 + f) * 3 * NF + q2;
            const double m0 = __ldg(&m[0]), m1 = __ldg(&m[NF]), m2 = __ldg(&m[2 * NF]);
#pragma unroll
            for (int k = 0; k < 4; ++k) tout[(f * GL_T2W + k) * NF + q2] = m0 * F[0][k] + m1 * F[1][k] + m2 * F[2][k];
            continue;
        }
        viscous_flux<double>(r, gq, ucv, cst, F, 1 << dn, nullptr);
#pragma unroll
        for (int k = 0; k < 4; ++k)   // (selects, not a run-time index, keep F in registers)
            tout[(f * GL_T2W + k) * NF + q2] = dn == 0 ? F[0][k] : dn == 1 ? F[1][k] : F[2][k];
    }
    // the split form evaluates the volume viscous flux at the entropy-projected state
    // (strong_dg.cpp:1328 before :1392); the face-normal flux interpolated to the faces uses
    // the state itself (:2836-3041)
    // sF: [d][k][Q3] volume viscous flux
    for (int q = threadIdx.x; q < Q3; q += NT) {
        double u[5], gq[5][3];
#pragma unroll
        for (int s = 0; s < 5; ++s) {
            u[s] = SPLIT ? __ldg(&g.proj[((size_t)cell * 5 + s) * Q3 + q]) : sQ[s * Q3 + q];
#pragma unroll
            for (int d = 0; d < 3; ++d) gq[s][d] = sAQ[(s * 3 + d) * Q3 + q];
        }
        double F[3][4];
        viscous_flux<double>(u, gq, ucv, cst, F, 7, nullptr);
        if constexpr (CURV) gl_contravariant(vm, q, Q3, F);
#pragma unroll
        for (int d = 0; d < 3; ++d)
#pragma unroll
            for (int k = 0; k < 4; ++k) sF[(d * 4 + k) * Q3 + q] = F[d][k];
    }
    __syncthreads();
    // W sum_d D_d F_d, momentum and energy rows
    gl_line<NT, NQ, NQ, 0, NQ, NQ, NQ, 4>(T.dphi, sF, Q3, t0, Q3, 1.0, false);
    __syncthreads();
    gl_line<NT, NQ, NQ, 1, NQ, NQ, NQ, 4>(T.dphi, sF + 4 * Q3, Q3, t0, Q3, 1.0, true);
    __syncthreads();
    gl_line<NT, NQ, NQ, 2, NQ, NQ, NQ, 4>(T.dphi, sF + 8 * Q3, Q3, t0, Q3, 1.0, true);
    __syncthreads();
    for (int i = threadIdx.x; i < 4 * Q3; i += NT) {
        const int q = i % Q3;
        g.vis[(size_t)cell * 4 * Q3 + i] = t0[i] * (tab->wq[q % NQ] * tab->wq[(q / NQ) % NQ] * tab->wq[q / NF]);
    }
    // face-normal volume viscous flux at the faces: n_dn sum_l phi_l(side) F_dn(u_l) (state not
    // projected)
    if constexpr (SPLIT) {
        __syncthreads();
        for (int q = threadIdx.x; q < Q3; q += NT) {
            double u[5], gq[5][3];
#pragma unroll
            for (int s = 0; s < 5; ++s) {
                u[s] = sQ[s * Q3 + q];
#pragma unroll
                for (int d = 0; d < 3; ++d) gq[s][d] = sAQ[(s * 3 + d) * Q3 + q];
            }
            double F[3][4];
            viscous_flux<double>(u, gq, ucv, cst, F, 7, nullptr);
            if constexpr (CURV) gl_contravariant(vm, q, Q3, F);
#pragma unroll
            for (int d = 0; d < 3; ++d)
#pragma unroll
                for (int k = 0; k < 4; ++k) sF[(d * 4 + k) * Q3 + q] = F[d][k];
        }
    }
    __syncthreads();
    for (int it = threadIdx.x; it < 6 * 4 * NF; it += NT) {
        const int f = it / (4 * NF), k = (it / NF) % 4, q2 = it % NF;
        const int dn = f >> 1, side = f & 1;
        const double* rw = tab->phis[side];
        const double* row = sF + (dn * 4 + k) * Q3;
        double v = 0.0;
#pragma unroll
        for (int l = 0; l < NQ; ++l) v += rw[l] * row[gl_line_node<NQ>(dn, q2, l)];
        tout[(f * GL_T2W + 4 + k) * NF + q2] = side ? v : -v;
    }
}

// The same on affine cells without boundary faces, line by line: the derivative pass adds the weights and
// the faces' lifts as it writes, a face node's gradient is contracted once for both ends of its line,
// and each direction's flux lines give the face-normal fluxes at their ends and are replaced by their
// derivatives (summed as they are stored). gl_aux_kernel, which serves the other cells, is bound by index
// arithmetic and shared-memory traffic: 136 us at 12^3 cells of p = 5, here 83 us (FP64 pipe 34 % busy,
// shared memory 50 %, three CTAs per SM by registers). 192 threads at NQ = 6 take the 180 lines of a
// direction's five rows in one pass.
template <int ND, int NQ, bool SPLIT>
struct GlAuxLineLayout {
    static constexpr int NT = NQ <= 3 ? 64 : NQ == 4 ? 96 : NQ == 5 ? 128 : NQ == 6 ? 192 : 256;
    static constexpr int D3 = ND * ND * ND, Q3 = NQ * NQ * NQ, NF = NQ * NQ;
    static constexpr int oQ = 0;                          // 5 NQ^3 state at the flux nodes
    static constexpr int oG = oQ + 5 * Q3;                // 15 NQ^3 lifted gradient, later flux rows d * 4 + k
    static constexpr int nR = SPLIT && 12 * Q3 > 30 * NF ? 12 * Q3 : 30 * NF;
    static constexpr int oR = oG + 15 * Q3;               // [d][s][2][NF] face terms, later (split) the state's own flux
    static constexpr int total = oR + nR;
    static constexpr size_t bytes = (size_t)total * sizeof(double);
    // CTAs per SM asked of the register allocator (96 registers at NQ = 6)
    static constexpr int MINB = NQ <= 3 ? 8 : NQ == 4 ? 5 : NQ == 5 ? 4 : NQ == 6 ? 3 : 2;
};

template <int ND, int NQ, bool SPLIT>
__global__ void __launch_bounds__(GlAuxLineLayout<ND, NQ, SPLIT>::NT, GlAuxLineLayout<ND, NQ, SPLIT>::MINB)
gl_aux_line_kernel(const StageArgs a, const GlArgs g, const __grid_constant__ GlTab T) {
    using L = GlAuxLineLayout<ND, NQ, SPLIT>;
    constexpr int NT = L::NT, D3 = L::D3, Q3 = L::Q3, NF = L::NF, T1W = gl_t1_width<SPLIT>();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double wq[NQ];
    double* sm = reinterpret_cast<double*>(smem_raw);
    double* sQ = sm + L::oQ;
    double* sG = sm + L::oG;
    double* sR = sm + L::oR;
    const int cell = a.tiles ? __ldg(&a.tiles[blockIdx.x]) : a.cell_begin + (int)blockIdx.x;
    const int tid = threadIdx.x;
    Cst<double> cst; cst.load(a.pc);
    const int ucv = a.pc.use_const_visc;
    if (tid < NQ) wq[tid] = g.tab->wq[tid];
    for (int i = tid; i < 5 * D3; i += NT) sQ[i] = __ldg(&a.U[(size_t)cell * 5 * D3 + i]);
    if constexpr (SPLIT) {   // read after the gradient: to L2 meanwhile
        const char* pj = reinterpret_cast<const char*>(g.proj + (size_t)cell * 5 * Q3);
        for (int i = tid * 128; i < 5 * Q3 * 8; i += NT * 128)
            asm volatile("prefetch.global.L2 [%0];" ::"l"(pj + i));
    }
    // faces: (u* - u) n at the two ends of every line, all loads in flight before the first store (with
    // the prefetch above 4.86 against 5.12 ms a step of 24^3 cells, p = 5; 151 against 160 us, 12^3, p = 3)
    {
        constexpr int NI = 30 * NF, IT = (NI + NT - 1) / NT;
        double uo[IT], ue[IT];
#pragma unroll
        for (int j = 0; j < IT; ++j) {
            const int it = tid + j * NT < NI ? tid + j * NT : 0;
            const int d = it / (10 * NF), s = (it / (2 * NF)) % 5, side = (it / NF) & 1, q2 = it % NF, f = 2 * d + side;
            const int cn = __ldg(&a.nbr[cell * 6 + f]);
            uo[j] = __ldg(&g.t1[(((size_t)cell * 6 + f) * T1W + s) * NF + q2]);
            ue[j] = __ldg(&g.t1[(((size_t)cn * 6 + (f ^ 1)) * T1W + s) * NF + q2]);
        }
#pragma unroll
        for (int j = 0; j < IT; ++j) {
            const int it = tid + j * NT;
            if (it < NI) sR[it] = (0.5 * (uo[j] + ue[j]) - uo[j]) * (((it / NF) & 1) ? 1.0 : -1.0);
        }
    }
    __syncthreads();
    gl_apply3<NT, NQ, ND, 5>(T.chi, sQ, D3, sQ, Q3, sG, sG + 5 * Q3, 1.0, false);
    // W D_d u + the faces' lifts, into row d * 5 + s: one thread per line
#pragma unroll
    for (int d = 0; d < 3; ++d)
        for (int it = tid; it < 5 * NF; it += NT) {
            const int s = it / NF, line = it - s * NF;
            int st;
            const int base = gl_line_base<NQ>(d, line, st);
            const double* ip = sQ + s * Q3 + base;
            double* op = sG + (d * 5 + s) * Q3 + base;
            const double f0 = sR[d * 10 * NF + s * 2 * NF + line], f1 = sR[d * 10 * NF + s * 2 * NF + NF + line];
            const double wab = wq[line % NQ] * wq[line / NQ];
            double v[NQ];
#pragma unroll
            for (int l = 0; l < NQ; ++l) v[l] = ip[l * st];
#pragma unroll
            for (int o = 0; o < NQ; ++o) {
                double x = 0.0;
#pragma unroll
                for (int l = 0; l < NQ; ++l) x += T.dphi[o * NQ + l] * v[l];
                op[o * st] = wab * (T.wq[o] * x + (T.phis[0][o] * f0 + T.phis[1][o] * f1));
            }
        }
    __syncthreads();
    gl_line<NT, NQ, NQ, 0, NQ, NQ, NQ, 15>(T.haux, sG, Q3, sG, Q3, 1.0, false);
    __syncthreads();
    gl_line<NT, NQ, NQ, 1, NQ, NQ, NQ, 15>(T.haux, sG, Q3, sG, Q3, 1.0, false);
    __syncthreads();
    gl_line<NT, NQ, NQ, 2, NQ, NQ, NQ, 15>(T.haux, sG, Q3, sG, Q3, a.inv_h, false);
    __syncthreads();
    // per face node of the cell: F_v(u, q) . e_d with the state's and the gradient's face values
    double* tout = g.t2 + (size_t)cell * 6 * GL_T2W * NF;
#pragma unroll 1
    for (int it = tid; it < 3 * NF; it += NT) {
        const int d = it / NF, line = it - d * NF;
        int st;
        const int base = gl_line_base<NQ>(d, line, st);
        double gq[2][5][3];
#pragma unroll
        for (int e = 0; e < 3; ++e)
#pragma unroll
            for (int s = 0; s < 5; ++s)
                gl_line_ends<NQ>(T, sG + (e * 5 + s) * Q3 + base, st, gq[0][s][e], gq[1][s][e]);
#pragma unroll
        for (int side = 0; side < 2; ++side) {
            double r[5], F[3][4];
#pragma unroll
            for (int s = 0; s < 5; ++s) r[s] = __ldg(&g.t1[(((size_t)cell * 6 + 2 * d + side) * T1W + s) * NF + line]);
            viscous_flux<double>(r, gq[side], ucv, cst, F, 7, nullptr);
#pragma unroll
            for (int k = 0; k < 4; ++k)
                tout[((2 * d + side) * GL_T2W + k) * NF + line] = d == 0 ? F[0][k] : d == 1 ? F[1][k] : F[2][k];
        }
    }
    __syncthreads();   // (the gradient rows are overwritten below)
    // nodal fluxes: the split form evaluates the volume term at the entropy-projected state
    // (strong_dg.cpp:1328 before :1392), the face-normal flux with the state itself (:2836-3041)
#pragma unroll 1
    for (int q = tid; q < Q3; q += NT) {
        double u[5], gq[5][3], F[3][4];
#pragma unroll
        for (int s = 0; s < 5; ++s) {
            u[s] = sQ[s * Q3 + q];
#pragma unroll
            for (int e = 0; e < 3; ++e) gq[s][e] = sG[(e * 5 + s) * Q3 + q];
        }
        viscous_flux<double>(u, gq, ucv, cst, F, 7, nullptr);
        double* R = (SPLIT ? sR : sG) + q;
#pragma unroll
        for (int e = 0; e < 3; ++e)
#pragma unroll
            for (int k = 0; k < 4; ++k) R[(e * 4 + k) * Q3] = F[e][k];
        if constexpr (SPLIT) {
#pragma unroll
            for (int s = 0; s < 5; ++s) u[s] = __ldg(&g.proj[((size_t)cell * 5 + s) * Q3 + q]);
            viscous_flux<double>(u, gq, ucv, cst, F, 7, nullptr);
#pragma unroll
            for (int e = 0; e < 3; ++e)
#pragma unroll
                for (int k = 0; k < 4; ++k) sG[(e * 4 + k) * Q3 + q] = F[e][k];
        }
    }
    __syncthreads();
    // the face-normal fluxes at the lines' ends, and D_d F_d in place of F_d
#pragma unroll
    for (int d = 0; d < 3; ++d)
        for (int it = tid; it < 4 * NF; it += NT) {
            const int k = it / NF, line = it - k * NF;
            int st;
            const int base = gl_line_base<NQ>(d, line, st);
            double* fp = sG + (d * 4 + k) * Q3 + base;
            double v[NQ], e0, e1;
#pragma unroll
            for (int l = 0; l < NQ; ++l) v[l] = fp[l * st];
            if constexpr (SPLIT) {
                gl_line_ends<NQ>(T, sR + (d * 4 + k) * Q3 + base, st, e0, e1);
            } else {
                e0 = e1 = 0.0;
#pragma unroll
                for (int l = 0; l < NQ; ++l) { e0 += T.phis[0][l] * v[l]; e1 += T.phis[1][l] * v[l]; }
            }
            tout[((2 * d) * GL_T2W + 4 + k) * NF + line] = -e0;
            tout[((2 * d + 1) * GL_T2W + 4 + k) * NF + line] = e1;
#pragma unroll
            for (int o = 0; o < NQ; ++o) {
                double x = 0.0;
#pragma unroll
                for (int l = 0; l < NQ; ++l) x += T.dphi[o * NQ + l] * v[l];
                fp[o * st] = x;
            }
        }
    __syncthreads();
    for (int q = tid; q < Q3; q += NT) {   // W sum_d D_d F_d, momentum and energy rows
        const double W = wq[q % NQ] * wq[(q / NQ) % NQ] * wq[q / NF];
#pragma unroll
        for (int k = 0; k < 4; ++k)
            g.vis[((size_t)cell * 4 + k) * Q3 + q] =
                W * ((sG[k * Q3 + q] + sG[(4 + k) * Q3 + q]) + sG[(8 + k) * Q3 + q]);
    }
}

// ------------------------------------------------------------------------------------
// Residual (+ mass inverse + RK epilogue)
// ------------------------------------------------------------------------------------
template <int ND, int NQ, bool VISC, bool SPLIT, bool CURV = false>
struct GlStageLayout {
    static constexpr int NT = gl_threads<NQ>();
    static constexpr int D3 = ND * ND * ND, Q3 = NQ * NQ * NQ, NF = NQ * NQ;
    static constexpr int nTab = (int)(sizeof(GlTab) / sizeof(double));
    static constexpr int oU = nTab;                       // 5 ND^3 state, later the right-hand side
    static constexpr int oQ = oU + 5 * D3;                // 5 NQ^3 state at the flux nodes (split: projected)
    static constexpr int oN = oQ + 5 * Q3;                // node quantities (11 NQ^3) or fluxes (15 NQ^3)
    static constexpr int oDiv = oN + 15 * Q3;             // 5 NQ^3 volume divergence (+ hybrid volume terms)
    static constexpr int oF = oDiv + 5 * Q3;              // 6 x 5 x NF face arrays
    static constexpr int nT = gl_temp<ND, NQ>();
    static constexpr int oT0 = oF + 30 * NF, oT1 = oT0 + nT;
    static constexpr int oQF = oT1 + nT;                 // split: the node quantities of two faces' nodes
    static constexpr int oM = oQF + (SPLIT ? 2 * NF * 11 : 0);   // curvilinear: 9 NQ^3 metric cofactor
    static constexpr int total = oM + (CURV ? 9 * Q3 : 0);
    static constexpr size_t bytes = (size_t)total * sizeof(double);
    static_assert(2 * nT >= 2 * NF * NQ * 5, "the hybrid pair fluxes of one direction fit the temporaries");
};

// The volume terms at the flux nodes minus the face arrays' lift (see gl_line_ends), plus the viscous
// divergence. Ends with a barrier.
template <int NT, int NQ, bool VISC>
__device__ __forceinline__ void gl_add_faces(const GlTab& T, const GlArgs& g, int cell, const double* sF,
                                             double* sDiv) {
    constexpr int NF = NQ * NQ, Q3 = NF * NQ;
    __shared__ double ph[2][NQ];   // (read with run-time indices)
    if (threadIdx.x < 2 * NQ) ph[threadIdx.x / NQ][threadIdx.x % NQ] = g.tab->phis[threadIdx.x / NQ][threadIdx.x % NQ];
    __syncthreads();
    for (int q = threadIdx.x; q < Q3; q += NT) {
        const int c[3] = {q % NQ, (q / NQ) % NQ, q / NF};
        double r[5];
#pragma unroll
        for (int s = 0; s < 5; ++s) r[s] = sDiv[s * Q3 + q];
        if constexpr (VISC) {
#pragma unroll
            for (int k = 0; k < 4; ++k) r[1 + k] += __ldg(&g.vis[((size_t)cell * 4 + k) * Q3 + q]);
        }
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const double p0 = ph[0][c[d]], p1 = ph[1][c[d]];
            const double* f = sF + 2 * d * 5 * NF + c[d == 2 ? 1 : 2] * NQ + c[d == 0 ? 1 : 0];
#pragma unroll
            for (int s = 0; s < 5; ++s) r[s] -= p0 * f[s * NF] + p1 * f[(5 + s) * NF];
        }
#pragma unroll
        for (int s = 0; s < 5; ++s) sDiv[s * Q3 + q] = r[s];
    }
    __syncthreads();
}

// Butcher RK stage (as the collocated kernel's epilogue) of one cell from its time derivative sK
template <int NT, int D3>
__device__ __forceinline__ void gl_rk_epilogue(const StageArgs& a, int cell, const double* sK) {
    for (int i = threadIdx.x; i < 5 * D3; i += NT) {
        const size_t dof = (size_t)cell * 5 * D3 + i;
        const double k = sK[i];
        const double un = a.Un[dof];
        const double bs = a.acc_in ? a.acc_in[dof] : (a.inc_mode ? 0.0 : un);
        const double sum = bs + a.c_acc * k;
        if (a.acc_out) a.acc_out[dof] = sum;
        if (a.final_out) a.final_out[dof] = a.inc_mode ? un + sum : sum;
        if (a.next) {
            const double cin = a.carry_in ? a.carry_in[dof] : 0.0;
            a.next[dof] = (cin + a.a_next * k) * a.dt + un;
        }
        if (a.carry_out) a.carry_out[dof] = a.a_carry * k;
    }
}

// CURV (split or conservative Euler on curvilinear cells): the volume two-point fluxes are dotted
// with the metric average 1/2 (C_i[:, d] + C_j[:, d]) and the conservative fluxes with C[:, d]
// (strong_dg.cpp:1235-1578), the face fluxes use the face's unit normal C[:, dn] / |C[:, dn]|
// scaled by |C[:, dn]| and the hybrid terms 1/2 (C_face[:, dn] + C_vol[:, dn]) (:3144-3452), and
// the inverse mass is the weight-adjusted P diag(1 / (W det J)) P^T, P = (M+K)^-1 chi^T W
// (dg_base.cpp:4217-4249, operators.cpp:1909-1932). The residual is then in physical units.
template <int ND, int NQ, bool VISC, bool SPLIT, bool CURV = false, bool BND = false>
__global__ void __launch_bounds__(gl_threads<NQ>(), 2)
gl_stage_kernel(const StageArgs a, const GlArgs g, const __grid_constant__ GlTab T) {
    using L = GlStageLayout<ND, NQ, VISC, SPLIT, CURV>;
    constexpr int NT = L::NT, D3 = L::D3, Q3 = L::Q3, NF = L::NF, T1W = gl_t1_width<SPLIT>();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* sm = reinterpret_cast<double*>(smem_raw);
    GlTab* tab = reinterpret_cast<GlTab*>(sm);
    double* sU = sm + L::oU;
    double* sQ = sm + L::oQ;
    double* sN = sm + L::oN;
    double* sDiv = sm + L::oDiv;
    double* sF = sm + L::oF;
    double* t0 = sm + L::oT0;
    double* t1 = sm + L::oT1;
    const int cell = a.tiles ? __ldg(&a.tiles[blockIdx.x]) : a.cell_begin + (int)blockIdx.x;
    Cst<double> cst; cst.load(a.pc);
    const int tp = a.pc.two_point, cf = a.pc.conv_flux, df = a.pc.diss_flux, ucv = a.pc.use_const_visc;
    double* sM = sm + L::oM;   // curvilinear: the cofactor at the flux nodes, [k * 3 + d][Q3]
    gl_load_tab(g.tab, tab, NT);
    if constexpr (!SPLIT)
        for (int i = threadIdx.x; i < 5 * D3; i += NT) sU[i] = __ldg(&a.U[(size_t)cell * 5 * D3 + i]);
    if constexpr (CURV)
        for (int i = threadIdx.x; i < 9 * Q3; i += NT) sM[i] = __ldg(&g.vmet[(size_t)cell * 10 * Q3 + i]);
    gl_prefetch_l2<NT, NF, D3, Q3, T1W, true, VISC>(a, g, cell);
    __syncthreads();
    if constexpr (!SPLIT) gl_apply3<NT, NQ, ND, 5>(T.chi, sU, D3, sQ, Q3, t0, t1, 1.0, false);
    if constexpr (SPLIT) {
        // the entropy-projected state u(P (x3) v(chi u)) at the flux nodes (strong_dg.cpp:1235-1330)
        for (int q = threadIdx.x; q < Q3; q += NT) {
            double u[5];
#pragma unroll
            for (int s = 0; s < 5; ++s) u[s] = __ldg(&g.proj[((size_t)cell * 5 + s) * Q3 + q]);
            NodeQ<double> nq;
            node_prepare<double>(u, tp, cst.gm1, nq, a.status);
            store_q<double>(sN, Q3, q, nq);
        }
        __syncthreads();
        // two-point volume term: sum over the node's three flux-node lines of
        // skew[x_d][l] w_a w_b F(u_i, u_l) . e_d   (operators.cpp:983-1062), pair-symmetric on
        // warp segments as in the collocated kernel: segments of NQ lanes own the lines along
        // rd; lane pos evaluates the pairs (pos, pos + k), k = 1 .. NQ / 2, in the frame whose x
        // axis is e_rd and receives the pair (pos - k, pos) from lane pos - k of its segment (the
        // two-point fluxes are symmetric); w_a w_b, the same along a line, scales the sum.
        constexpr int SPW = 32 / NQ, NSEG = (NT / 32) * SPW;
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        const int lseg = lane / NQ, pos = lane - lseg * NQ, segbase = lseg * NQ;
#pragma unroll 1
        for (int rd = 0; rd < 3; ++rd) {
            const int st = rd == 0 ? 1 : rd == 1 ? NQ : NF;
#pragma unroll 1
            for (int l0 = 0; l0 < NF; l0 += NSEG) {
                const int lt = l0 + warp * SPW + lseg;
                const bool valid = lseg < SPW && lt < NF;
                const int node = gl_line_node<NQ>(rd, valid ? lt : 0, pos);
                const int base = node - pos * st;
                double acc[5];
                if constexpr (CURV) {   // the pair flux dotted with the averaged metric column
                    NodeQ<double> qi;
                    load_q<double>(sN, Q3, node, qi);
                    const double mi[3] = {sM[(0 * 3 + rd) * Q3 + node], sM[(1 * 3 + rd) * Q3 + node],
                                          sM[(2 * 3 + rd) * Q3 + node]};
#pragma unroll
                    for (int s = 0; s < 5; ++s) acc[s] = 0.0;
#pragma unroll
                    for (int k = 1; k <= NQ / 2; ++k) {
                        const int jp = pos + k < NQ ? pos + k : pos + k - NQ;
                        const int jm = pos - k >= 0 ? pos - k : pos - k + NQ;
                        const bool dup = ((NQ & 1) == 0) && (2 * k == NQ);
                        const int nj = base + jp * st;
                        NodeQ<double> qj;
                        load_q<double>(sN, Q3, nj, qj);
                        const double nv[3] = {0.5 * (mi[0] + sM[(0 * 3 + rd) * Q3 + nj]),
                                              0.5 * (mi[1] + sM[(1 * 3 + rd) * Q3 + nj]),
                                              0.5 * (mi[2] + sM[(2 * 3 + rd) * Q3 + nj])};
                        double F[5];
                        two_point_n<double>(qi, qj, nv, tp, cst, F);
                        const double cj = tab->skew[pos * NQ + jp], cr = tab->skew[pos * NQ + jm];
#pragma unroll
                        for (int s = 0; s < 5; ++s) {
                            const double fr = __shfl_sync(0xffffffffu, F[s], segbase + jm);
                            acc[s] += cj * F[s];
                            if (!dup) acc[s] += cr * fr;
                        }
                    }
                } else {
                    NodeQ<double> qi;
                    load_q_rot<double>(sN, Q3, node, rd, qi);
                    double accr[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
#pragma unroll
                    for (int k = 1; k <= NQ / 2; ++k) {
                        const int jp = pos + k < NQ ? pos + k : pos + k - NQ;   // (pos + k) mod NQ
                        const int jm = pos - k >= 0 ? pos - k : pos - k + NQ;   // (pos - k) mod NQ
                        const bool dup = ((NQ & 1) == 0) && (2 * k == NQ);
                        NodeQ<double> qj;
                        load_q_rot<double>(sN, Q3, base + jp * st, rd, qj);
                        double F[5];
                        two_point_dir<double, 0>(qi, qj, tp, cst, F);
                        const double cj = tab->skew[pos * NQ + jp], cr = tab->skew[pos * NQ + jm];
#pragma unroll
                        for (int s = 0; s < 5; ++s) {
                            const double fr = __shfl_sync(0xffffffffu, F[s], segbase + jm);
                            accr[s] += cj * F[s];
                            if (!dup) accr[s] += cr * fr;
                        }
                    }
                    // back to (x, y, z) components by selects (a run-time index would put acc in
                    // local memory)
                    acc[0] = accr[0]; acc[4] = accr[4];
                    acc[1] = rd == 0 ? accr[1] : rd == 1 ? accr[3] : accr[2];
                    acc[2] = rd == 0 ? accr[2] : rd == 1 ? accr[1] : accr[3];
                    acc[3] = rd == 0 ? accr[3] : rd == 1 ? accr[2] : accr[1];
                }
                if (valid) {
                    const int t1c = lt % NQ, t2c = lt / NQ;
                    const double wab = tab->wq[t1c] * tab->wq[t2c];
#pragma unroll
                    for (int s = 0; s < 5; ++s) {
                        double* o = sDiv + s * Q3 + node;
                        *o = rd == 0 ? wab * acc[s] : *o + wab * acc[s];
                    }
                }
            }
            __syncthreads();
        }
    } else {
        // conservative: W div(F(chi u)) by the flux-node derivative   (strong_dg.cpp:1546)
        for (int q = threadIdx.x; q < Q3; q += NT) {
            double u[5];
#pragma unroll
            for (int s = 0; s < 5; ++s) u[s] = sQ[s * Q3 + q];
            NodeQ<double> nq;
            node_prepare<double>(u, TP_KG, cst.gm1, nq, a.status);
#pragma unroll
            for (int d = 0; d < 3; ++d) {   // affine: F . e_d; curvilinear: the contravariant F . C[:, d]
                const double nv[3] = {CURV ? sM[(0 * 3 + d) * Q3 + q] : d == 0 ? 1.0 : 0.0,
                                      CURV ? sM[(1 * 3 + d) * Q3 + q] : d == 1 ? 1.0 : 0.0,
                                      CURV ? sM[(2 * 3 + d) * Q3 + q] : d == 2 ? 1.0 : 0.0};
                double F[5];
                conv_flux_n<double>(nq, nv, 0.0, F);
#pragma unroll
                for (int s = 0; s < 5; ++s) sN[(d * 5 + s) * Q3 + q] = F[s];
            }
        }
        __syncthreads();
        gl_line<NT, NQ, NQ, 0, NQ, NQ, NQ, 5>(T.dphi, sN, Q3, sDiv, Q3, 1.0, false);
        __syncthreads();
        gl_line<NT, NQ, NQ, 1, NQ, NQ, NQ, 5>(T.dphi, sN + 5 * Q3, Q3, sDiv, Q3, 1.0, true);
        __syncthreads();
        gl_line<NT, NQ, NQ, 2, NQ, NQ, NQ, 5>(T.dphi, sN + 10 * Q3, Q3, sDiv, Q3, 1.0, true);
        __syncthreads();
        for (int i = threadIdx.x; i < 5 * Q3; i += NT) {
            const int q = i % Q3;
            sDiv[i] *= tab->wq[q % NQ] * tab->wq[(q / NQ) % NQ] * tab->wq[q / NF];
        }
        __syncthreads();
    }

    // ---- faces: numerical fluxes (canonical orientation: the left state is the cell whose
    // +e_dn face it is, the normal +e_dn), and this cell's face array
    // W_face (F_vol.n + F_v,vol.n -/+ F*_conv -/+ F*_diss) [- hybrid surface terms]
    for (int it = threadIdx.x; it < 6 * NF; it += NT) {
        const int f = it / NF, q2 = it % NF;
        const int dn = f >> 1, side = f & 1;
        const double sgn = side ? 1.0 : -1.0;
        const int cn = __ldg(&a.nbr[cell * 6 + f]);
        const bool bnd = BND && cn < 0;   // a boundary face (assemble_boundary_term_strong, strong_dg.cpp:1582-2366)
        const double* to = g.t1 + ((size_t)cell * 6 + f) * T1W * NF + q2;
        const double* te = g.t1 + ((size_t)(bnd ? cell : cn) * 6 + (f ^ 1)) * T1W * NF + q2;
        double uo[5], ue[5], ro[5], re[5];
#pragma unroll
        for (int s = 0; s < 5; ++s) { ro[s] = __ldg(&to[s * NF]); re[s] = __ldg(&te[s * NF]); }
        if (bnd) {
            // the convective flux between the interpolated face state (the projected one with
            // use_projected_entropy_variables_for_nsfr_boundary_term, :2255-2273) and its boundary state
            double ub[5];
#pragma unroll
            for (int s = 0; s < 5; ++s) uo[s] = ro[s];
            if (SPLIT && a.pc.bc_projected) {
#pragma unroll
                for (int s = 0; s < 5; ++s) uo[s] = __ldg(&to[(5 + s) * NF]);
            }
            double mnv[3];
            if constexpr (CURV) {   // the face's unit metric normal C[:, dn] / |C[:, dn]|
                const double* m = g.fnrm + ((size_t)cell * 6 + f) * 3 * NF + q2;
                const double m0 = __ldg(&m[0]), m1 = __ldg(&m[NF]), m2 = __ldg(&m[2 * NF]);
                const double J = sqrt(m0 * m0 + m1 * m1 + m2 * m2);
                mnv[0] = m0 / J; mnv[1] = m1 / J; mnv[2] = m2 / J;
            }
            gl_bnd_state(__ldg(&a.btype[-1 - cn]), uo, f, a.pc, ub, a.status, CURV ? mnv : nullptr);
#pragma unroll
            for (int s = 0; s < 5; ++s) ue[s] = ub[s];
        } else if constexpr (SPLIT) {
#pragma unroll
            for (int s = 0; s < 5; ++s) { uo[s] = __ldg(&to[(5 + s) * NF]); ue[s] = __ldg(&te[(5 + s) * NF]); }
        } else {
#pragma unroll
            for (int s = 0; s < 5; ++s) { uo[s] = ro[s]; ue[s] = re[s]; }
        }
        double nv[3] = {dn == 0 ? 1.0 : 0.0, dn == 1 ? 1.0 : 0.0, dn == 2 ? 1.0 : 0.0};
        double Jf = 1.0;
        if constexpr (CURV) {   // the face's unit normal and |C[:, dn]|
            const double* m = g.fnrm + ((size_t)cell * 6 + f) * 3 * NF + q2;
            const double m0 = __ldg(&m[0]), m1 = __ldg(&m[NF]), m2 = __ldg(&m[2 * NF]);
            Jf = sqrt(m0 * m0 + m1 * m1 + m2 * m2);
            nv[0] = m0 / Jf; nv[1] = m1 / Jf; nv[2] = m2 / Jf;
        }
        const double* uL = side ? uo : ue;
        const double* uR = side ? ue : uo;
        NodeQ<double> qL, qR;
        node_prepare<double>(uL, tp, cst.gm1, qL, nullptr);
        node_prepare<double>(uR, tp, cst.gm1, qR, nullptr);
        double Fc[5];
        conv_num_flux_n<double>(uL, uR, qL, qR, nv, tp, cf, cst, Fc);
        double term[5];
#pragma unroll
        for (int s = 0; s < 5; ++s) term[s] = -sgn * (CURV ? Jf * Fc[s] : Fc[s]);
        if constexpr (VISC) {
            // each side's F_v(u, q) . e_dn at the face node, from the auxiliary kernel
            const double* ao = g.t2 + ((size_t)cell * 6 + f) * GL_T2W * NF + q2;
            const double* ae = g.t2 + ((size_t)(bnd ? cell : cn) * 6 + (f ^ 1)) * GL_T2W * NF + q2;
            double Fo[4], Fe[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) { Fo[k] = __ldg(&ao[k * NF]); Fe[k] = __ldg(&ae[k * NF]); }
            const double* rL = side ? ro : re;
            const double* rR = side ? re : ro;
            const double* FL = side ? Fo : Fe;
            const double* FR = side ? Fe : Fo;
            double Fd[4];
#pragma unroll
            for (int k = 0; k < 4; ++k)   // boundary: F*_v . e_dn = sgn (F*_v . n_out) of the auxiliary kernel
                Fd[k] = bnd ? sgn * __ldg(&g.fb[((size_t)(-1 - cn) * 4 + k) * NF + q2]) : 0.5 * (FL[k] + FR[k]);
            if (df == DF_SIPG && !bnd) {
                double jump[5][3];
#pragma unroll
                for (int s = 0; s < 5; ++s)
#pragma unroll
                    for (int d = 0; d < 3; ++d) jump[s][d] = d == dn ? rL[s] - rR[s] : 0.0;
                double AL[3][4], AR[3][4];
                viscous_flux<double>(rL, jump, ucv, cst, AL, 1 << dn, nullptr);
                viscous_flux<double>(rR, jump, ucv, cst, AR, 1 << dn, nullptr);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const double al = dn == 0 ? AL[0][k] : dn == 1 ? AL[1][k] : AL[2][k];
                    const double ar = dn == 0 ? AR[0][k] : dn == 1 ? AR[1][k] : AR[2][k];
                    Fd[k] = Fd[k] - a.pen * (0.5 * (al + ar));
                }
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) term[1 + k] += -sgn * Fd[k] + __ldg(&ao[(4 + k) * NF]);
        }
        if constexpr (!SPLIT) {   // the cell's own convective volume flux at the face: n . sum_l phi_l F(u_l)
            const double* rw = tab->phis[side];
#pragma unroll
            for (int s = 0; s < 5; ++s) {
                const double* row = sN + (dn * 5 + s) * Q3;
                double v = 0.0;
#pragma unroll
                for (int l = 0; l < NQ; ++l) v += rw[l] * row[gl_line_node<NQ>(dn, q2, l)];
                term[s] += sgn * v;
            }
        }
        const double wf = tab->wq[q2 % NQ] * tab->wq[q2 / NQ];
#pragma unroll
        for (int s = 0; s < 5; ++s) sF[(f * 5 + s) * NF + q2] = wf * term[s];
    }
    __syncthreads();
    if constexpr (SPLIT) {
        // hybrid surface-volume two-point terms (strong_dg.cpp:3144-3350): between each face node
        // (its projected state) and the flux nodes of the normal line through it. One direction at
        // a time (its two faces share the volume nodes): the face nodes' quantities, then every
        // (face node, line node) pair flux, then the face sums and the volume sums, in the order
        // face 2 dn before face 2 dn + 1 and line position by position.
        double* sQF = sm + L::oQF;   // [11][2 NF]
        double* s2 = t0;             // [2][NF][NQ][5] (t0 and t1 are contiguous)
#pragma unroll 1
        for (int dn = 0; dn < 3; ++dn) {
            const double nv[3] = {dn == 0 ? 1.0 : 0.0, dn == 1 ? 1.0 : 0.0, dn == 2 ? 1.0 : 0.0};
            for (int it = threadIdx.x; it < 2 * NF; it += NT) {
                const int side = it / NF, q2 = it % NF;
                const double* to = g.t1 + ((size_t)cell * 6 + 2 * dn + side) * T1W * NF + q2;
                double uf[5];
#pragma unroll
                for (int s = 0; s < 5; ++s) uf[s] = __ldg(&to[(5 + s) * NF]);
                NodeQ<double> qf;
                node_prepare<double>(uf, tp, cst.gm1, qf, nullptr);
                store_q<double>(sQF, 2 * NF, it, qf);
            }
            __syncthreads();
            for (int it = threadIdx.x; it < 2 * NF * NQ; it += NT) {
                const int side = it / (NF * NQ), r = it % (NF * NQ), q2 = r / NQ, l = r % NQ;
                const int node = gl_line_node<NQ>(dn, q2, l);
                NodeQ<double> qv, qf;
                load_q<double>(sN, Q3, node, qv);
                load_q<double>(sQF, 2 * NF, side * NF + q2, qf);
                double F[5];
                if constexpr (CURV) {   // 1/2 (C_face[:, dn] + C_vol[:, dn])
                    const double* m = g.fnrm + ((size_t)cell * 6 + 2 * dn + side) * 3 * NF + q2;
                    const double mv[3] = {0.5 * (__ldg(&m[0]) + sM[(0 * 3 + dn) * Q3 + node]),
                                          0.5 * (__ldg(&m[NF]) + sM[(1 * 3 + dn) * Q3 + node]),
                                          0.5 * (__ldg(&m[2 * NF]) + sM[(2 * 3 + dn) * Q3 + node])};
                    two_point_n<double>(qv, qf, mv, tp, cst, F);
                } else {
                    two_point_n<double>(qv, qf, nv, tp, cst, F);
                }
#pragma unroll
                for (int s = 0; s < 5; ++s) s2[(size_t)it * 5 + s] = F[s];
            }
            __syncthreads();
            for (int it = threadIdx.x; it < 2 * NF; it += NT) {   // face sums
                const int side = it / NF, q2 = it % NF, f = 2 * dn + side;
                const double sgn = side ? 1.0 : -1.0;
                const double wf = tab->wq[q2 % NQ] * tab->wq[q2 / NQ];
                double hs[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
#pragma unroll
                for (int l = 0; l < NQ; ++l) {
                    const double Hop = tab->phis[side][l] * wf * sgn;
                    const double* F = s2 + ((size_t)(side * NF + q2) * NQ + l) * 5;
#pragma unroll
                    for (int s = 0; s < 5; ++s) hs[s] -= Hop * F[s];
                }
#pragma unroll
                for (int s = 0; s < 5; ++s) sF[(f * 5 + s) * NF + q2] -= hs[s];
            }
            for (int it = threadIdx.x; it < NF * NQ; it += NT) {   // volume sums (other outputs)
                const int q2 = it / NQ, l = it % NQ;
                const int t1c = q2 % NQ, t2c = q2 / NQ;
                const int node = gl_line_node<NQ>(dn, q2, l);
                const double wf = tab->wq[t1c] * tab->wq[t2c];
#pragma unroll
                for (int side = 0; side < 2; ++side) {
                    const double Hop = tab->phis[side][l] * wf * (side ? 1.0 : -1.0);
                    const double* F = s2 + ((size_t)(side * NF + q2) * NQ + l) * 5;
#pragma unroll
                    for (int s = 0; s < 5; ++s) sDiv[s * Q3 + node] += Hop * F[s];
                }
            }
            __syncthreads();
        }
    }
    // ---- assembly: r = -chi^T (x3) [div (+ hybrid) + viscous divergence - sum_f phis[side] (x) face array],
    // or, on affine cells, k = M^-1 R straight away: (1/h) (M+K)^-1 (x3) folded into the same passes
    gl_add_faces<NT, NQ, VISC>(T, g, cell, sF, sDiv);
    if (CURV || a.mode == 0) {
        gl_apply3<NT, ND, NQ, 5, true>(T.chi, sDiv, Q3, sU, D3, t0, t1, -1.0, false);
        // affine: sU = R / h^2 (the affine metric C = h^2 I and J = h^2 factored out); curvilinear: R
        if (a.mode == 0) {
            const double h2 = CURV ? 1.0 : a.h * a.h;
            for (int i = threadIdx.x; i < 5 * D3; i += NT) a.out[(size_t)cell * 5 * D3 + i] = h2 * sU[i];
            return;
        }
        // curvilinear: k = P (x3) [ (1 / (W det J)) P^T (x3) R ]
        gl_apply3<NT, NQ, ND, 5, true>(T.pwa, sU, D3, sDiv, Q3, t0, t1, 1.0, false);
        const double* iJ = g.vmet + ((size_t)cell * 10 + 9) * Q3;
        for (int i = threadIdx.x; i < 5 * Q3; i += NT) {
            const int q = i % Q3;
            sDiv[i] *= __ldg(&iJ[q]) / (tab->wq[q % NQ] * tab->wq[(q / NQ) % NQ] * tab->wq[q / NF]);
        }
        __syncthreads();
        gl_apply3<NT, ND, NQ, 5>(T.pwa, sDiv, Q3, sQ, D3, t0, t1, 1.0, false);
    } else {
        gl_apply3<NT, ND, NQ, 5, true>(T.chm, sDiv, Q3, sQ, D3, t0, t1, -a.inv_h, false);
    }
    if (a.mode == 1) {
        for (int i = threadIdx.x; i < 5 * D3; i += NT) a.out[(size_t)cell * 5 * D3 + i] = sQ[i];
        return;
    }
    if (a.mode == 3) {   // low-storage 3S* / 3S*+ stage (as the collocated kernel's)
        double err2 = 0.0;
        for (int i = threadIdx.x; i < 5 * D3; i += NT) ls_stage_dof(a, (size_t)cell * 5 * D3 + i, sQ[i], err2);
        if (a.err_partial) ls_tile_error<NT>(err2, &a.err_partial[cell]);
        return;
    }
    if (a.ent_partial) {
        // relaxation RK: this cell's v_hat^T M k, v_hat the entropy variables of the stage input
        // projected on the solution basis (compute_entropy_vars, runge_kutta_store_entropy.cpp:30-100)
        // and M = chi^T W J chi (compute_entropy_change_estimate, root_finding_rrk_ode_solver.cpp:353-388):
        // the sum over the flux nodes of W J (chi v_hat)(chi k), chi v_hat = (chi M^-1 chi^T W) v(chi u)
        for (int i = threadIdx.x; i < 5 * D3; i += NT) sU[i] = __ldg(&a.U[(size_t)cell * 5 * D3 + i]);
        __syncthreads();
        gl_apply3<NT, NQ, ND, 5>(T.chi, sU, D3, sDiv, Q3, t0, t1, 1.0, false);
        for (int q = threadIdx.x; q < Q3; q += NT) {
            double u[5], v[5];
#pragma unroll
            for (int s = 0; s < 5; ++s) u[s] = sDiv[s * Q3 + q];
            gl_entropy_vars(u, cst.gam, cst.gm1, v, nullptr);
#pragma unroll
            for (int s = 0; s < 5; ++s) sDiv[s * Q3 + q] = v[s];
        }
        __syncthreads();
        gl_apply3<NT, NQ, NQ, 5>(T.P, sDiv, Q3, sN, Q3, t0, t1, 1.0, false);
        gl_apply3<NT, NQ, ND, 5>(T.chi, sQ, D3, sDiv, Q3, t0, t1, 1.0, false);
        const double h3 = a.h * a.h * a.h;
        double ent = 0.0;
        for (int i = threadIdx.x; i < 5 * Q3; i += NT) {
            const int q = i % Q3;
            const double W = tab->wq[q % NQ] * tab->wq[(q / NQ) % NQ] * tab->wq[q / NF];
            const double J = CURV ? 1.0 / __ldg(&g.vmet[((size_t)cell * 10 + 9) * Q3 + q]) : h3;
            ent += W * J * sN[i] * sDiv[i];
        }
        __shared__ double ered[32];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ent += __shfl_down_sync(0xffffffffu, ent, o);
        if ((threadIdx.x & 31) == 0) ered[threadIdx.x >> 5] = ent;
        __syncthreads();
        if (threadIdx.x == 0) {
            double t = 0.0;
            for (int w = 0; w < (NT + 31) / 32; ++w) t += ered[w];
            a.ent_partial[cell] = t;
        }
    }
    gl_rk_epilogue<NT, D3>(a, cell, sQ);
}

// The last part of the affine stage kernels (as gl_stage_kernel's): lifts, transposed interpolation with the
// inverse mass, and the result or the RK stage. Overwrites sDiv.
template <int NT, int ND, int NQ, bool VISC>
__device__ __forceinline__ void gl_finish(const StageArgs& a, const GlTab& T, const GlArgs& g, int cell,
                                          const double* sF, double* sDiv, double* t0, double* t1) {
    constexpr int D3 = ND * ND * ND, Q3 = NQ * NQ * NQ;
    gl_add_faces<NT, NQ, VISC>(T, g, cell, sF, sDiv);
    if (a.mode == 0) {
        gl_apply3<NT, ND, NQ, 5, true>(T.chi, sDiv, Q3, sDiv, D3, t0, t1, -1.0, false);
        const double h2 = a.h * a.h;
        for (int i = threadIdx.x; i < 5 * D3; i += NT) a.out[(size_t)cell * 5 * D3 + i] = h2 * sDiv[i];
        return;
    }
    gl_apply3<NT, ND, NQ, 5, true>(T.chm, sDiv, Q3, sDiv, D3, t0, t1, -a.inv_h, false);
    if (a.mode == 1) {
        for (int i = threadIdx.x; i < 5 * D3; i += NT) a.out[(size_t)cell * 5 * D3 + i] = sDiv[i];
        return;
    }
    if (a.mode == 3) {   // low-storage 3S* / 3S*+ stage
        double err2 = 0.0;
        for (int i = threadIdx.x; i < 5 * D3; i += NT) ls_stage_dof(a, (size_t)cell * 5 * D3 + i, sDiv[i], err2);
        if (a.err_partial) ls_tile_error<NT>(err2, &a.err_partial[cell]);
        return;
    }
    gl_rk_epilogue<NT, D3>(a, cell, sDiv);
}

// ------------------------------------------------------------------------------------
// Residual (+ mass inverse + RK epilogue), conservative form, affine cells without boundary faces
// ------------------------------------------------------------------------------------
// One CTA per cell with a thread per line of one direction's five rows. A direction's flux lines give
// the volume flux at their ends and are replaced by their derivatives in one pass, the numerical fluxes
// are evaluated in the face's frame (the normal's axis first, so that the penalty's jump has one
// direction), and the state, the fluxes and the temporaries share their space (14 KB at NQ = 4). Bound by
// latency: a step of 12^3 cells of p = 3 (Roe, SIPG, three stages) takes 160 us where gl_stage_kernel with two
// warps of 236 registers a cell took 228.
template <int ND, int NQ>
struct GlConsLayout {
    static constexpr int NT = NQ <= 3 ? 64 : NQ == 4 ? 96 : NQ == 5 ? 160 : NQ == 6 ? 224 : 256;
    static constexpr int MINB = 512 / NT;                 // 128 registers
    static constexpr int D3 = ND * ND * ND, Q3 = NQ * NQ * NQ, NF = NQ * NQ;
    static constexpr int oQ = 0;                          // 5 NQ^3 state at the flux nodes, later the volume terms
    static constexpr int oN = oQ + 5 * Q3;                // [d][s][Q3] fluxes, then derivatives; temporaries
    static constexpr int oF = oN + 15 * Q3;               // [face][5][NF] face arrays
    static constexpr int total = oF + 30 * NF;
    static constexpr size_t bytes = (size_t)total * sizeof(double);
};

template <int ND, int NQ, bool VISC>
__global__ void __launch_bounds__(GlConsLayout<ND, NQ>::NT, GlConsLayout<ND, NQ>::MINB)
gl_cons_stage_kernel(const StageArgs a, const GlArgs g, const __grid_constant__ GlTab T) {
    using L = GlConsLayout<ND, NQ>;
    constexpr int NT = L::NT, D3 = L::D3, Q3 = L::Q3, NF = L::NF, T1W = gl_t1_width<false>();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double wq[NQ];
    double* sm = reinterpret_cast<double*>(smem_raw);
    double* sQ = sm + L::oQ;
    double* sN = sm + L::oN;
    double* sF = sm + L::oF;
    double* t0 = sN;
    double* t1 = sN + 5 * Q3;
    const int cell = a.tiles ? __ldg(&a.tiles[blockIdx.x]) : a.cell_begin + (int)blockIdx.x;
    const int tid = threadIdx.x;
    Cst<double> cst; cst.load(a.pc);
    const int tp = a.pc.two_point, cf = a.pc.conv_flux, df = a.pc.diss_flux, ucv = a.pc.use_const_visc;
    if (tid < NQ) wq[tid] = g.tab->wq[tid];
    for (int i = tid; i < 5 * D3; i += NT) sQ[i] = __ldg(&a.U[(size_t)cell * 5 * D3 + i]);
    gl_prefetch_l2<NT, NF, D3, Q3, T1W, true, VISC>(a, g, cell);
    __syncthreads();
    gl_apply3<NT, NQ, ND, 5>(T.chi, sQ, D3, sQ, Q3, t0, t1, 1.0, false);
    for (int q = tid; q < Q3; q += NT) {
        double u[5];
#pragma unroll
        for (int s = 0; s < 5; ++s) u[s] = sQ[s * Q3 + q];
        NodeQ<double> nq;
        node_prepare<double>(u, TP_KG, cst.gm1, nq, a.status);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const double nv[3] = {d == 0 ? 1.0 : 0.0, d == 1 ? 1.0 : 0.0, d == 2 ? 1.0 : 0.0};
            double F[5];
            conv_flux_n<double>(nq, nv, 0.0, F);
#pragma unroll
            for (int s = 0; s < 5; ++s) sN[(d * 5 + s) * Q3 + q] = F[s];
        }
    }
    __syncthreads();
    // D_d F_d in place of F_d, and the cell's own flux n . F at the lines' ends   (strong_dg.cpp:1546)
#pragma unroll
    for (int d = 0; d < 3; ++d)
        for (int it = tid; it < 5 * NF; it += NT) {
            const int s = it / NF, line = it - s * NF;
            int st;
            double* fp = sN + (d * 5 + s) * Q3 + gl_line_base<NQ>(d, line, st);
            double v[NQ], e0 = 0.0, e1 = 0.0;
#pragma unroll
            for (int l = 0; l < NQ; ++l) v[l] = fp[l * st];
#pragma unroll
            for (int l = 0; l < NQ; ++l) { e0 += T.phis[0][l] * v[l]; e1 += T.phis[1][l] * v[l]; }
            sF[(2 * d * 5 + s) * NF + line] = -e0;
            sF[((2 * d + 1) * 5 + s) * NF + line] = e1;
#pragma unroll
            for (int o = 0; o < NQ; ++o) {
                double x = 0.0;
#pragma unroll
                for (int l = 0; l < NQ; ++l) x += T.dphi[o * NQ + l] * v[l];
                fp[o * st] = x;
            }
        }
    __syncthreads();
    for (int q = tid; q < Q3; q += NT) {
        const double W = wq[q % NQ] * wq[(q / NQ) % NQ] * wq[q / NF];
#pragma unroll
        for (int s = 0; s < 5; ++s)
            sQ[s * Q3 + q] = W * ((sN[s * Q3 + q] + sN[(5 + s) * Q3 + q]) + sN[(10 + s) * Q3 + q]);
    }
    // numerical fluxes (canonical orientation: the left state is the cell whose +e_d face it is)
#pragma unroll 1
    for (int it = tid; it < 6 * NF; it += NT) {
        const int f = it / NF, q2 = it - f * NF;
        const int d = f >> 1, side = f & 1;
        const int d2 = d == 2 ? 0 : d + 1, d3 = d == 0 ? 2 : d - 1;
        const double sgn = side ? 1.0 : -1.0;
        const int cn = __ldg(&a.nbr[cell * 6 + f]);
        const double* to = g.t1 + ((size_t)cell * 6 + f) * T1W * NF + q2;
        const double* te = g.t1 + ((size_t)cn * 6 + (f ^ 1)) * T1W * NF + q2;
        const int row[5] = {0, 1 + d, 1 + d2, 1 + d3, 4};
        double uL[5], uR[5], term[5];
#pragma unroll
        for (int s = 0; s < 5; ++s) {
            const double uo = __ldg(&to[row[s] * NF]), ue = __ldg(&te[row[s] * NF]);
            uL[s] = side ? uo : ue;
            uR[s] = side ? ue : uo;
        }
        NodeQ<double> qL, qR;
        node_prepare<double>(uL, tp, cst.gm1, qL, nullptr);
        node_prepare<double>(uR, tp, cst.gm1, qR, nullptr);
        conv_num_flux<double, 0>(uL, uR, qL, qR, tp, cf, cst, term);
        if constexpr (VISC) {   // each side's F_v(u, q) . e_d at the face node, from the auxiliary kernel
            const double* ao = g.t2 + ((size_t)cell * 6 + f) * GL_T2W * NF + q2;
            const double* ae = g.t2 + ((size_t)cn * 6 + (f ^ 1)) * GL_T2W * NF + q2;
            const int kr[4] = {d, d2, d3, 3};
            double Fd[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) Fd[k] = 0.5 * (__ldg(&ao[kr[k] * NF]) + __ldg(&ae[kr[k] * NF]));
            if (df == DF_SIPG) {
                double jump[5][3], AL[3][4], AR[3][4];
#pragma unroll
                for (int s = 0; s < 5; ++s) { jump[s][0] = uL[s] - uR[s]; jump[s][1] = jump[s][2] = 0.0; }
                viscous_flux<double>(uL, jump, ucv, cst, AL, 1, nullptr);
                viscous_flux<double>(uR, jump, ucv, cst, AR, 1, nullptr);
#pragma unroll
                for (int k = 0; k < 4; ++k) Fd[k] -= a.pen * (0.5 * (AL[0][k] + AR[0][k]));
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) term[1 + k] += Fd[k] - sgn * __ldg(&ao[(4 + kr[k]) * NF]);
        }
        const double wf = wq[q2 % NQ] * wq[q2 / NQ];
#pragma unroll
        for (int s = 0; s < 5; ++s) {
            double* o = sF + (f * 5 + row[s]) * NF + q2;
            *o = wf * (*o - sgn * term[s]);
        }
    }
    gl_finish<NT, ND, NQ, VISC>(a, T, g, cell, sF, sQ, t0, t1);
}

// ------------------------------------------------------------------------------------
// Residual (+ mass inverse + RK epilogue), Chandrashekar + EC/Roe (+ BR2) flux set, affine cells
// without boundary faces
// ------------------------------------------------------------------------------------
// One CTA per cell of as many warps as one direction's lines take (four at NQ = 6). The two-point
// volume terms run on line segments (line_pairs), and the hybrid surface-volume terms with them:
// a lane evaluates the pairs of its own nodes with the line's two face nodes, adds them to its
// nodes' sums and hands the face sums to the line's first lane, so no pair flux passes through
// memory. The numerical face fluxes, whose operands come from the face-value buffers, are evaluated
// while the node quantities are formed. The temporaries of the final passes reuse the space of the
// quantities (48 KB at NQ = 6: four CTAs per SM). At 12^3 cells of p = 5 it takes 86 us
// (FP64 pipe 37 % busy, the rest latency), 97 us while the faces were lifted one after the other after
// the last interpolation. An RK4 step of 24^3 such cells: 11.9 ms with the node form, 7.7 with
// this kernel and the states projected once, 4.9 with the line form of the other two kernels.
template <int ND, int NQ>
struct GlLineLayout {
    static constexpr int D3 = ND * ND * ND, Q3 = NQ * NQ * NQ, NF = NQ * NQ;
    static constexpr int LNT = (NF + line_spw<NQ>() - 1) / line_spw<NQ>() * 32;
    static constexpr int NT = LNT < 64 ? 64 : LNT;
    static constexpr int ZP = NQ == 6 ? NF + 1 : NQ == 4 ? NF + 3 : NF;   // as LineLayout
    static constexpr int NS = ZP * (NQ - 1) + NF;
    static constexpr int nTab = (int)(sizeof(GlTab) / sizeof(double));
    static constexpr int oQ = nTab;                       // rho/2, v/2 (3), b, |v|^2/4, log rho, log b
    static constexpr int oQF = oQ + 8 * NS;               // [face][8][NF] the same at the face nodes
    static constexpr int nT = gl_temp<ND, NQ>();
    static constexpr int oT0 = oQ, oT1 = oQ + nT;
    static constexpr int nQ = 8 * NS + 48 * NF > 2 * nT ? 8 * NS + 48 * NF : 2 * nT;
    static constexpr int oF = oQ + nQ;                    // [face][5][NF] face arrays
    static constexpr int oDiv = oF + 30 * NF;             // 5 NQ^3 volume terms, later the result
    static constexpr int total = oDiv + 5 * Q3;
    static constexpr size_t bytes = (size_t)total * sizeof(double);
    static constexpr int MINB = NT <= 128 ? 512 / NT : NT <= 256 ? 2 : 1;   // 128 registers (65536 / 512 threads)
};

template <int ND, int NQ, bool VISC>
__global__ void __launch_bounds__(GlLineLayout<ND, NQ>::NT, GlLineLayout<ND, NQ>::MINB)
gl_line_stage_kernel(const StageArgs a, const GlArgs g, const __grid_constant__ GlTab T) {
    using L = GlLineLayout<ND, NQ>;
    constexpr int NT = L::NT, D3 = L::D3, Q3 = L::Q3, NF = L::NF, NS = L::NS, ZP = L::ZP, T1W = gl_t1_width<true>();
    constexpr int NPL = line_npl<NQ>(), H = line_lanes<NQ>(), SPW = line_spw<NQ>();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int span[4];
    double* sm = reinterpret_cast<double*>(smem_raw);
    GlTab* tab = reinterpret_cast<GlTab*>(sm);
    double* sQ = sm + L::oQ;
    double* sQF = sm + L::oQF;
    double* sF = sm + L::oF;
    double* sDiv = sm + L::oDiv;
    double* t0 = sm + L::oT0;
    double* t1 = sm + L::oT1;
    const int cell = a.tiles ? __ldg(&a.tiles[blockIdx.x]) : a.cell_begin + (int)blockIdx.x;
    const int tid = threadIdx.x;
    Cst<double> cst; cst.load(a.pc);
    constexpr int tp = (int)TP_CH, cf = (int)CF_EC_ROE;
    if (tid < 4) span[tid] = (tid & 1) ? (int)0x80000000 : 0x7fffffff;
    gl_load_tab(g.tab, tab, NT);
    gl_prefetch_l2<NT, NF, D3, Q3, T1W, true, VISC>(a, g, cell);
    __syncthreads();

    // ---- node quantities of the projected state
    int lo_r = 0x7fffffff, hi_r = (int)0x80000000, lo_b = lo_r, hi_b = hi_r;
    auto widen = [&](const NodeQ<double>& q) {
        lo_r = min(lo_r, hi_word(q.rho)); hi_r = max(hi_r, hi_word(q.rho));
        lo_b = min(lo_b, hi_word(q.b)); hi_b = max(hi_b, hi_word(q.b));
    };
    for (int q = tid; q < Q3; q += NT) {
        double u[5];
#pragma unroll
        for (int s = 0; s < 5; ++s) u[s] = __ldg(&g.proj[((size_t)cell * 5 + s) * Q3 + q]);
        NodeQ<double> nq;
        node_prepare<double, LOG_HERE>(u, tp, cst.gm1, nq, a.status);
        double* Q = sQ + q + (q / NF) * (ZP - NF);
        Q[0] = 0.5 * nq.rho; Q[NS] = 0.5 * nq.v[0]; Q[2 * NS] = 0.5 * nq.v[1]; Q[3 * NS] = 0.5 * nq.v[2];
        Q[4 * NS] = nq.b; Q[5 * NS] = 0.25 * nq.vsq;
        widen(nq);
    }
    // ---- faces: numerical fluxes (canonical orientation, the normal's axis first), and this cell's
    // face array W_face (-/+ F*_conv -/+ F*_diss + F_v,vol.n)
#pragma unroll 1
    for (int it = tid; it < 6 * NF; it += NT) {
        const int f = it / NF, q2 = it - f * NF;
        const int d = f >> 1, side = f & 1;
        const int d2 = d == 2 ? 0 : d + 1, d3 = d == 0 ? 2 : d - 1;
        const double sgn = side ? 1.0 : -1.0;
        const int cn = __ldg(&a.nbr[cell * 6 + f]);
        const double* to = g.t1 + (((size_t)cell * 6 + f) * T1W + 5) * NF + q2;
        const double* te = g.t1 + (((size_t)cn * 6 + (f ^ 1)) * T1W + 5) * NF + q2;
        const int row[5] = {0, 1 + d, 1 + d2, 1 + d3, 4};
        double uo[5], ue[5];
#pragma unroll
        for (int s = 0; s < 5; ++s) { uo[s] = __ldg(&to[row[s] * NF]); ue[s] = __ldg(&te[row[s] * NF]); }
        NodeQ<double> qo, qe;
        node_prepare<double, LOG_HERE>(uo, tp, cst.gm1, qo, nullptr);
        node_prepare<double, LOG_HERE>(ue, tp, cst.gm1, qe, nullptr);
        double* QF = sQF + f * 8 * NF + q2;
        QF[0] = 0.5 * qo.rho; QF[(1 + d) * NF] = 0.5 * qo.v[0]; QF[(1 + d2) * NF] = 0.5 * qo.v[1];
        QF[(1 + d3) * NF] = 0.5 * qo.v[2]; QF[4 * NF] = qo.b; QF[5 * NF] = 0.25 * qo.vsq;
        widen(qo);
        NodeQ<double> ql = qo, qr = qe;   // (the conservative states are not read by this flux set)
        if (!side) { ql = qe; qr = qo; }
        double term[5];
        conv_num_flux<double, 0, LOG_HERE>(uo, uo, ql, qr, tp, cf, cst, term);
#pragma unroll
        for (int s = 0; s < 5; ++s) term[s] *= -sgn;
        if constexpr (VISC) {   // each side's F_v(u, q) . e_d at the face node, from the auxiliary kernel
            const double* ao = g.t2 + ((size_t)cell * 6 + f) * GL_T2W * NF + q2;
            const double* ae = g.t2 + ((size_t)cn * 6 + (f ^ 1)) * GL_T2W * NF + q2;
            const int kr[4] = {d, d2, d3, 3};
#pragma unroll
            for (int k = 0; k < 4; ++k)
                term[1 + k] += __ldg(&ao[(4 + kr[k]) * NF]) -
                               sgn * (0.5 * (__ldg(&ao[kr[k] * NF]) + __ldg(&ae[kr[k] * NF])));
        }
        const double wf = tab->wq[q2 % NQ] * tab->wq[q2 / NQ];
#pragma unroll
        for (int s = 0; s < 5; ++s) sF[(f * 5 + row[s]) * NF + q2] = wf * term[s];
    }
    lo_r = __reduce_min_sync(0xffffffffu, lo_r); hi_r = __reduce_max_sync(0xffffffffu, hi_r);
    lo_b = __reduce_min_sync(0xffffffffu, lo_b); hi_b = __reduce_max_sync(0xffffffffu, hi_b);
    if ((tid & 31) == 0) {
        atomicMin(&span[0], lo_r); atomicMax(&span[1], hi_r);
        atomicMin(&span[2], lo_b); atomicMax(&span[3], hi_b);
    }
    __syncthreads();
    const bool smooth = series_span<double>(span[0], span[1]) && series_span<double>(span[2], span[3]);
    if (!smooth) {   // strong gradients in the cell: the logarithms of every node
        for (int q = tid; q < Q3 + 6 * NF; q += NT) {
            const bool vol = q < Q3;
            const int r = q - Q3;
            double* Q = vol ? sQ + q + (q / NF) * (ZP - NF) : sQF + (r / NF) * 8 * NF + r % NF;
            const int pitch = vol ? NS : NF;
            Q[6 * pitch] = log(2.0 * Q[0]);
            Q[7 * pitch] = log(Q[4 * pitch]);
        }
        __syncthreads();
    }

    // ---- volume and hybrid two-point terms, direction by direction. Up to four flux nodes one warp takes all lines
    // of a direction (the block's other warp waits below) and keeps the directions apart by itself: a block
    // barrier that both warps meet takes 0.4 to 1.8 % more of a step (20^3 cells, p = 2, Euler: 426 against 421 us)
    static_assert(L::LNT == 32 || NT == L::LNT, "one warp works, or every thread meets the barriers");
    {
        const int lane = tid & 31;
        const int pos = lane / SPW < H ? lane / SPW : 0, seg = lane % SPW;
        const int lineid = (tid >> 5) * SPW + seg;
        const bool lvalid = lane < H * SPW && lineid < NF;   // (idle lanes run along on line 0)
        const int line = lvalid ? lineid : 0, la = line % NQ, lb = line / NQ;
        const double wab = tab->wq[la] * tab->wq[lb];
        auto directions = [&](auto lm) {
            constexpr int LM = decltype(lm)::value;
#pragma unroll 1
            for (int d = 0; d < 3; ++d) {
                const int d2 = d == 2 ? 0 : d + 1, d3 = d == 0 ? 2 : d - 1;
                const int st = d == 0 ? 1 : d == 1 ? NQ : ZP;
                const int base = d == 0 ? NQ * la + ZP * lb : d == 1 ? la + ZP * lb : la + NQ * lb;
                const int r1 = (1 + d) * NS, r2 = (1 + d2) * NS, r3 = (1 + d3) * NS;
                double acc[NPL][5], hs[2][5];
                line_pairs<double, NQ, NS, false, LM>(
                    LineRows<double>{sQ, sQ + 4 * NS, sQ + 6 * NS, nullptr, r1, r2, r3}, base, st, pos, seg, tab->skew, cst,
                    acc);
                // hybrid terms: this lane's nodes with the line's two face nodes
#pragma unroll
                for (int side = 0; side < 2; ++side) {
                    const double* QF = sQF + (2 * d + side) * 8 * NF + line;
                    HalfQ<double> qf;
                    qf.hr = QF[0]; qf.hv[0] = QF[(1 + d) * NF]; qf.hv[1] = QF[(1 + d2) * NF]; qf.hv[2] = QF[(1 + d3) * NF];
                    qf.b = QF[4 * NF]; qf.q4 = QF[5 * NF];
                    if constexpr (LM == LOG_STORED) { qf.la = QF[6 * NF]; qf.lb = QF[7 * NF]; }
#pragma unroll
                    for (int s = 0; s < 5; ++s) hs[side][s] = 0.0;
#pragma unroll
                    for (int e = 0; e < NPL; ++e) {
                        const int i = NPL * pos + e, o = base + i * st;
                        HalfQ<double> qv;
                        qv.hr = sQ[o]; qv.hv[0] = sQ[r1 + o]; qv.hv[1] = sQ[r2 + o]; qv.hv[2] = sQ[r3 + o];
                        qv.b = sQ[4 * NS + o]; qv.q4 = sQ[5 * NS + o];
                        if constexpr (LM == LOG_STORED) { qv.la = sQ[6 * NS + o]; qv.lb = sQ[7 * NS + o]; }
                        double F[5];
                        ch_pair_axis<double, LM>(qv, qf, cst, F);
                        const double ph = tab->phis[side][i];
                        const double hp = side ? ph : -ph;
#pragma unroll
                        for (int s = 0; s < 5; ++s) { hs[side][s] += ph * F[s]; acc[e][s] += hp * F[s]; }
                    }
                }
                // the face sums of the line: lanes in the order of their places
#pragma unroll
                for (int side = 0; side < 2; ++side)
#pragma unroll
                    for (int s = 0; s < 5; ++s) {
                        double t = hs[side][s];
#pragma unroll
                        for (int j = 1; j < H; ++j) t += __shfl_sync(0xffffffffu, hs[side][s], j * SPW + seg);
                        hs[side][s] = t;
                    }
                const int row[5] = {0, 1 + d, 1 + d2, 1 + d3, 4};
                if (d > 0) {   // the previous direction's terms are in place
                    if constexpr (L::LNT == 32) __syncwarp();
                    else __syncthreads();
                }
                if (lvalid) {
                    const int su = d == 0 ? 1 : d == 1 ? NQ : NF;
                    double* A = sDiv + gl_line_node<NQ>(d, line, 0) + NPL * pos * su;
#pragma unroll
                    for (int e = 0; e < NPL; ++e)
#pragma unroll
                        for (int s = 0; s < 5; ++s) {
                            double* o = A + row[s] * Q3 + e * su;
                            *o = d == 0 ? wab * acc[e][s] : *o + wab * acc[e][s];
                        }
                    if (pos == 0) {
#pragma unroll
                        for (int side = 0; side < 2; ++side)
#pragma unroll
                            for (int s = 0; s < 5; ++s)
                                sF[((2 * d + side) * 5 + row[s]) * NF + line] += (side ? wab : -wab) * hs[side][s];
                    }
                }
            }
        };
        if (NT == L::LNT || tid < L::LNT) {   // (`smooth` is the same for the whole block)
            if (smooth) directions(std::integral_constant<int, LOG_NONE>());
            else directions(std::integral_constant<int, LOG_STORED>());
        }
    }
    __syncthreads();
    gl_finish<NT, ND, NQ, VISC>(a, T, g, cell, sF, sDiv, t0, t1);
}

// ------------------------------------------------------------------------------------
// Relaxation RK on uncollocated flux nodes: the integrated numerical entropy of
// u_n + gamma (u_1 - u_n), the state interpolated to the flux nodes
// (compute_integrated_numerical_entropy, root_finding_rrk_ode_solver.cpp:211-350): per-cell partials
// ------------------------------------------------------------------------------------
template <int ND, int NQ>
struct GlEntropyLayout {
    static constexpr int D3 = ND * ND * ND, Q3 = NQ * NQ * NQ, nT = gl_temp<ND, NQ>();
    static constexpr int oU = 0, oQ = oU + 5 * D3, oT0 = oQ + 5 * Q3, oT1 = oT0 + nT, total = oT1 + nT;
    static constexpr size_t bytes = (size_t)total * sizeof(double);
};

template <int ND, int NQ>
__global__ void __launch_bounds__(gl_threads<NQ>())
gl_rrk_entropy_kernel(const double* __restrict__ Un, const double* __restrict__ U1, double gamma,
                      const __grid_constant__ GlTab T, double h3, const double* __restrict__ vmet, double gam,
                      double* __restrict__ partial) {
    using L = GlEntropyLayout<ND, NQ>;
    constexpr int NT = gl_threads<NQ>(), D3 = L::D3, Q3 = L::Q3, NF = NQ * NQ;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* sm = reinterpret_cast<double*>(smem_raw);
    double* sU = sm + L::oU;
    double* sQ = sm + L::oQ;
    const int cell = blockIdx.x;
    for (int i = threadIdx.x; i < 5 * D3; i += NT) {
        const size_t k = (size_t)cell * 5 * D3 + i;
        sU[i] = Un[k] + gamma * (U1[k] - Un[k]);
    }
    __syncthreads();
    gl_apply3<NT, NQ, ND, 5>(T.chi, sU, D3, sQ, Q3, sm + L::oT0, sm + L::oT1, 1.0, false);
    double e = 0.0;
    for (int q = threadIdx.x; q < Q3; q += NT) {
        double u[5];
#pragma unroll
        for (int s = 0; s < 5; ++s) u[s] = sQ[s * Q3 + q];
        const double W = T.wq[q % NQ] * T.wq[(q / NQ) % NQ] * T.wq[q / NF];
        const double J = vmet ? 1.0 / vmet[((size_t)cell * 10 + 9) * Q3 + q] : h3;
        e += W * J * numerical_entropy_fn(u, gam);
    }
    __shared__ double red[32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) e += __shfl_down_sync(0xffffffffu, e, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = e;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < (NT + 31) / 32; ++w) t += red[w];
        partial[cell] = t;
    }
}

// ------------------------------------------------------------------------------------
// The weight-adjusted inverse mass on curvilinear cells on its own (ph_apply_inverse_mass):
// out = P (x3) [ (1 / (W det J)) P^T (x3) in ], one CTA per cell (a.U = in, a.out = out)
// ------------------------------------------------------------------------------------
template <int ND, int NQ>
struct GlMinvLayout {
    static constexpr int NT = gl_threads<NQ>();
    static constexpr int D3 = ND * ND * ND, Q3 = NQ * NQ * NQ;
    static constexpr int nTab = (int)(sizeof(GlTab) / sizeof(double));
    static constexpr int oU = nTab, oQ = oU + 5 * Q3;
    static constexpr int nT = gl_temp<ND, NQ>();
    static constexpr int oT0 = oQ + 5 * Q3, oT1 = oT0 + nT;
    static constexpr int total = oT1 + nT;
    static constexpr size_t bytes = (size_t)total * sizeof(double);
};

template <int ND, int NQ>
__global__ void __launch_bounds__(gl_threads<NQ>())
gl_minv_kernel(const StageArgs a, const GlArgs g, const __grid_constant__ GlTab T) {
    using L = GlMinvLayout<ND, NQ>;
    constexpr int NT = L::NT, D3 = L::D3, Q3 = L::Q3, NF = NQ * NQ;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* sm = reinterpret_cast<double*>(smem_raw);
    GlTab* tab = reinterpret_cast<GlTab*>(sm);
    double* sU = sm + L::oU;
    double* sQ = sm + L::oQ;
    double* t0 = sm + L::oT0;
    double* t1 = sm + L::oT1;
    const int cell = a.cell_begin + blockIdx.x;
    gl_load_tab(g.tab, tab, NT);
    for (int i = threadIdx.x; i < 5 * D3; i += NT) sU[i] = __ldg(&a.U[(size_t)cell * 5 * D3 + i]);
    __syncthreads();
    gl_apply3<NT, NQ, ND, 5, true>(T.pwa, sU, D3, sQ, Q3, t0, t1, 1.0, false);
    const double* iJ = g.vmet + ((size_t)cell * 10 + 9) * Q3;
    for (int i = threadIdx.x; i < 5 * Q3; i += NT) {
        const int q = i % Q3;
        sQ[i] *= __ldg(&iJ[q]) / (tab->wq[q % NQ] * tab->wq[(q / NQ) % NQ] * tab->wq[q / NF]);
    }
    __syncthreads();
    gl_apply3<NT, ND, NQ, 5>(T.pwa, sQ, Q3, a.out + (size_t)cell * 5 * D3, D3, t0, t1, 1.0, false);
}

} // namespace ph
