// Stage kernel of the split form on collocated GLL nodes with the Chandrashekar + EC/Roe (+ BR2)
// flux set, affine or curvilinear cells without boundary faces.
//
// Work decomposition. A CTA owns CPC cells. A 1-D line of N1 nodes belongs to a segment of lanes:
// two neighbouring nodes per lane when N1 is even, one when it is odd, so that every unordered pair
// of the line is evaluated once and every lane evaluates equally many (N1 = 6: five pairs on each of
// three lanes, its own pair and the four with the next lane's nodes; a pair's flux goes to the
// next lane by shuffles). The three directions run one after the other through one copy of the code.
// A neighbour's face values are read where the face fluxes are evaluated, and those go through shared memory
// once, as lifted terms.
//
// Why this split, against the node-per-lane form (residual_kernel): no pair of an even line is
// evaluated twice (15 instead of 18 per line at N1 = 6), the logarithms of the means are taken only in
// tiles whose gradients need them, halved node quantities save six operations per pair, the
// neighbour traces take no shared memory, and the rolled direction loop keeps the code in the
// instruction caches. The operations and their order per node are the same, so in FP64 both kernels give
// the same bits. What bounds it: FP64 operations with dependent latencies (FP64 pipe 44 %, issue 53 %, 19
// of 64 warps at 24^3 cells, p = 5); in the precision form issue slots (70 %).
// One stage, viscous, B200, node-per-lane form -> this kernel (FP64 / precision form, ms):
//   24^3 cells p = 5  0.488 -> 0.320 / 0.269 -> 0.215    32^3 p = 3  0.385 -> 0.224 / 0.215 -> 0.142
//   24^3 p = 4        0.305 -> 0.217 / 0.176 -> 0.132    30^3 p = 2  0.183 -> 0.105 / 0.111 -> 0.070
//   16^3 p = 6        0.401 -> 0.282                     32^3 p = 1  0.084 -> 0.048
// and 24^3 p = 4 curved 0.416 -> 0.253 (FP64). Measured and left out: one thread per line (15 pairs
// in registers: 0.433 ms at p = 5, its registers leave 12 warps per SM), the neighbour values copied
// ahead by cp.async (0.355), an L2 prefetch for the CTAs of the next wave (0.339).
#pragma once
#include "ph_kernels.cuh"

namespace ph {

template <int N1> constexpr int line_cells() {
    return N1 == 2 ? 16 : N1 == 3 ? 4 : N1 == 4 ? 4 : 1;
}

// nodes per lane, lanes per line, lines per warp (lane = place on the line * SPW + line of the warp)
template <int N1> __host__ __device__ constexpr int line_npl() { return N1 % 2 == 0 ? 2 : 1; }
template <int N1> __host__ __device__ constexpr int line_lanes() { return N1 / line_npl<N1>(); }
template <int N1> __host__ __device__ constexpr int line_spw() { return 32 / line_lanes<N1>(); }

template <typename R, int N1, int CPC, bool CURV, bool WIDE = false>
struct LineLayout {
    static constexpr int NP = N1 * N1 * N1, NF = N1 * N1;
    static constexpr int NPL = line_npl<N1>(), H = line_lanes<N1>(), SPW = line_spw<N1>();
    static constexpr int LNT = (CPC * NF + SPW - 1) / SPW * 32;   // threads of one direction's lines
    static constexpr int NT = (WIDE ? 3 : 1) * LNT;
    static constexpr int NA = WIDE ? 15 : 5;                  // rows of volume terms (wide: each direction its own)
    static constexpr int NQ = 8 + (CURV ? 9 : 0);   // rho/2 v/2 (3) p E b |v|^2/4 (+ half the metric cofactor)
    static constexpr bool F32 = sizeof(R) == 4;
    // nodes of a cell in shared memory: x + N1 y + ZP z. A padded z pitch and lanes ordered by their place on
    // the line first keep the lines' accesses in all three directions near one pass per bank
    // (N1 = 6: 1.8 passes instead of 2.3, N1 = 4 in FP64: 1.3 instead of 2.0, counted over all warps)
    static constexpr int ZP = N1 == 6 ? NF + 1 : N1 == 4 && !F32 ? NF + 3 : NF;
    static constexpr int NS = ZP * (N1 - 1) + NF;             // a row of nodes
    static constexpr int oS = 0;                              // skew operator, 1 / w_end
    static constexpr int oB = oS + N1 * N1 + N1;              // (M+K)^-1 diag(w)
    static constexpr int oQ = (oB + N1 * N1 + 1) & ~1;
    static constexpr int oL = oQ + CPC * NQ * NS;             // [c][2][NS] logarithms of rho and b
    static constexpr int oA = oL + CPC * 2 * NS;              // [c][NA][NS] volume terms
    static constexpr int oT = oA + CPC * NA * NS;             // [c][face][5][NF] lifted face terms
    static constexpr int total = oT + CPC * 30 * NF;
    static constexpr size_t bytes = (size_t)total * sizeof(R);
    // CTAs per SM asked of the register allocator, from timing one stage on B200 (viscous, affine):
    // N1 = 6 FP64 5 (96 registers; 0.320 ms at 24^3 cells, 4: 0.334, 6: 0.345), FP32 8 (64 registers;
    // 0.215 ms, 10: 0.227); N1 = 4 FP64 4 (0.224 ms at 32^3 cells, 5: 0.261), FP32 8 (0.142 ms); N1 = 5 FP64
    // 4 (0.217 ms at 24^3 cells, 3: 0.254), FP32 8 (0.132 ms, 6: 0.142); N1 = 3 FP64 5 (0.105 ms at 30^3
    // cells, 4: 0.113). Curvilinear cells' rows leave room for fewer CTAs at N1 = 4 and 6.
    static constexpr int ASKED = F32 ? (N1 == 7 ? 2 : 8)
                               : N1 == 7 ? 1 : N1 == 2 ? 7 : N1 == 3 ? 5 : N1 == 6 ? (CURV ? 4 : 5) : CURV && N1 == 4 ? 3 : 4;
    static constexpr int MINB = WIDE ? (NT <= 160 ? 3 : 1) : ASKED;
    // The batched kernel's own: its arguments come from shared memory, not from the parameter bank, which takes
    // registers, and its tiles may be wider. Timed on B200, one stage of 24^3 cells (16^3 from N1 = 5), us,
    // affine / curved, the single kernel's request -> this one, where they differ:
    //   precision form  N1 = 3, 8 cells 56 / 83 -> 41 / 60   N1 = 4, 2 cells 82 / 138 -> 71 / 111, 4 cells 74 / 122 -> 72 / 115
    //                   N1 = 5, 2 cells 71 / 99 -> 58 / 82   N1 = 6 80 / 133 -> 78 / 122   N1 = 7 157 / 227 -> 154 / 202
    //   FP64            N1 = 2 25 -> 23 (affine)             N1 = 3, 4 cells 60 / 94 -> 58 / 89, 8 cells 80 / 122 -> 60 / 93
    //                   N1 = 4, 2 cells 144 / 258 -> 105 / 192   N1 = 5, 1 cell 76 / 121 -> 74 / 119, 2 cells 85 / 136 -> 80 / 121
    //                   N1 = 6 119 -> 115 (affine)           N1 = 7 303 / 486 -> 227 / 337
    // Some of these spill (FP64 up to 230 bytes of local memory a thread at N1 = 3, 5 and 7): the requests that do
    // not leave too few warps (N1 = 5, 1 cell, FP64: none at 2 CTAs per SM, 109 us; 120 bytes at 5, 74 us).
    static constexpr int BATCHED =
        N1 == 2 ? (F32 ? 8 : CURV ? 5 : 6)
        : N1 == 3 ? (CPC == 4 ? (F32 ? (CURV ? 8 : 7) : 6) : F32 ? 4 : 3)
        : N1 == 4 ? (CPC == 2 ? (F32 ? (CURV ? 12 : 14) : CURV ? 6 : 8) : F32 ? (CURV ? 6 : 7) : CURV ? 3 : 4)
        : N1 == 5 ? (CPC == 1 ? (F32 ? 8 : 5) : F32 ? 4 : 3)
        : N1 == 6 ? (F32 ? (CURV ? 7 : 6) : 4) : F32 ? 3 : 2;
};

__device__ __forceinline__ int hi_word(double x) { return __double2hiint(x); }
__device__ __forceinline__ int hi_word(float x) { return __float_as_int(x); }
// true when any two of the values whose high words span [lo, hi] have |a - b| / (a + b) < 0.1, so
// every logarithmic mean among them takes its series branch (u = f^2 < 1e-2). The high words of
// positive numbers are ordered and piecewise linear: a span below 0.17 of a binade keeps
// |a - b| / (a + b) below 0.17 / 1.83 = 0.093 even across a power of two. Negative numbers and NaN
// against a number span far more.
template <typename R> __device__ __forceinline__ bool series_span(int lo, int hi) {
    constexpr unsigned lim = sizeof(R) == 8 ? (unsigned)(0.17 * (1 << 20)) : (unsigned)(0.17 * (1 << 23));
    return lo > 0 && (unsigned)hi - (unsigned)lo < lim;
}

// Where a cell's halved node quantities are: rho / 2 and the velocity rows at q (+ r1..r3: the rows of
// the line's frame), b and |v|^2 / 4 from qb, the logarithms from l, the halved metric column from m.
template <typename R> struct LineRows {
    const R* q;
    const R* qb;
    const R* l;
    const R* m;   // rows 0, 3, 6 of it (curvilinear cells)
    int r1, r2, r3;
};

// The two-point terms of one line on its segment of lanes: acc[e][s] = sum_j S[i][j] F(i, j) for this lane's
// nodes i = NPL pos + e, momentum in the line's frame (curvilinear: in x, y, z). Node i is at offset
// base + i st of the rows (row pitch NS); sS the operator, row-major; pos, seg: the lane's place on the
// line and its line of the warp. All lanes of the warp call it.
template <typename R, int N1, int NS, bool CURV, int LM>
__device__ __forceinline__ void line_pairs(const LineRows<R>& rw, int base, int st, int pos, int seg, const R* sS,
                                           const Cst<R>& cst, R (&acc)[line_npl<N1>()][5]) {
    constexpr int NPL = line_npl<N1>(), H = line_lanes<N1>(), SPW = line_spw<N1>();
    const int prev = (pos == 0 ? H - 1 : pos - 1) * SPW + seg;
    auto node = [&](int i, HalfQ<R>& q, R m[3]) {
        const int o = base + i * st;
        q.hr = rw.q[o]; q.hv[0] = rw.q[rw.r1 + o]; q.hv[1] = rw.q[rw.r2 + o]; q.hv[2] = rw.q[rw.r3 + o];
        q.b = rw.qb[o]; q.q4 = rw.qb[NS + o];
        if constexpr (LM == LOG_STORED) { q.la = rw.l[o]; q.lb = rw.l[NS + o]; }
        if constexpr (CURV) {
#pragma unroll
            for (int k = 0; k < 3; ++k) m[k] = rw.m[3 * k * NS + o];
        }
    };
    auto pair = [&](const HalfQ<R>& qi, const R mi[3], const HalfQ<R>& qj, const R mj[3], R F[5]) {
        if constexpr (CURV) {
            const R nv[3] = {mi[0] + mj[0], mi[1] + mj[1], mi[2] + mj[2]};
            ch_pair_n<R, LM>(qi, qj, nv, cst, F);
        } else {
            ch_pair_axis<R, LM>(qi, qj, cst, F);
        }
    };
    // the flux that the previous lane evaluated (towards this lane's nodes)
    auto from_prev = [&](const R F[5], R G[5]) {
#pragma unroll
        for (int s = 0; s < 5; ++s) G[s] = __shfl_sync(0xffffffffu, F[s], prev);
    };
    auto add = [&](R a[5], R c, const R F[5]) {
#pragma unroll
        for (int s = 0; s < 5; ++s) a[s] += c * F[s];
    };
#pragma unroll
    for (int e = 0; e < NPL; ++e)
#pragma unroll
        for (int s = 0; s < 5; ++s) acc[e][s] = R(0);
    if constexpr (NPL == 2) {
        // this lane's nodes i0, i1; the next lane's j0, j1; the previous lane's h0, h1. A node adds its
        // pairs in the order (i, i+1), (i-1, i), (i, i+2), (i-2, i), ..., opposite node last
        const int i0 = 2 * pos, i1 = i0 + 1;
        const int j0 = pos + 1 < H ? i0 + 2 : 0, j1 = j0 + 1;
        const int h0 = pos > 0 ? i0 - 2 : N1 - 2, h1 = h0 + 1;
        const R* c0 = sS + i0 * N1;
        const R* c1 = sS + i1 * N1;
        R* a0 = acc[0];
        R* a1 = acc[NPL - 1];
        HalfQ<R> q0, q1;
        R m0[3], m1[3];
        node(i0, q0, m0);
        node(i1, q1, m1);
        R F[5], G[5];
        if constexpr (N1 == 2) {
            pair(q0, m0, q1, m1, F);
            add(a0, c0[i1], F);
            add(a1, c1[i0], F);
        } else if constexpr (N1 == 4) {
            HalfQ<R> qj;
            R mj[3], E[5];
            pair(q0, m0, q1, m1, F);            // k = 1
            add(a0, c0[i1], F);
            node(j0, qj, mj);
            pair(q1, m1, qj, mj, E);
            from_prev(E, G);
            add(a0, c0[h1], G);
            add(a1, c1[j0], E);
            add(a1, c1[i0], F);
            // k = 2: the opposite pairs (0, 2) and (1, 3), one on each of the two lanes: lane 0's first
            // nodes, lane 1's second nodes
            HalfQ<R> qa = pos == 0 ? q0 : q1, qb;
            R ma[3], mb[3];
            if constexpr (CURV) {
#pragma unroll
                for (int e = 0; e < 3; ++e) ma[e] = pos == 0 ? m0[e] : m1[e];
            }
            node(pos == 0 ? j0 : j1, qb, mb);
            pair(qa, ma, qb, mb, F);
            from_prev(F, G);
            const R ce = c0[j0], cg = c1[j1];
#pragma unroll
            for (int s = 0; s < 5; ++s) {
                const R x = pos == 0 ? F[s] : G[s], y = pos == 0 ? G[s] : F[s];
                a0[s] += ce * x;
                a1[s] += cg * y;
            }
        } else {
            static_assert(N1 == 6 || N1 == 4 || N1 == 2, "even lines of 2, 4 or 6 nodes");
            HalfQ<R> q2;
            R m2[3], E[5];
            pair(q0, m0, q1, m1, F);            // k = 1
            add(a0, c0[i1], F);
            node(j0, q2, m2);
            pair(q1, m1, q2, m2, E);
            from_prev(E, G);
            add(a0, c0[h1], G);
            add(a1, c1[j0], E);
            add(a1, c1[i0], F);
            pair(q0, m0, q2, m2, F);            // k = 2
            from_prev(F, G);
            add(a0, c0[j0], F);
            add(a0, c0[h0], G);
            node(j1, q2, m2);
            pair(q1, m1, q2, m2, F);
            from_prev(F, G);
            add(a1, c1[j1], F);
            add(a1, c1[h1], G);
            pair(q0, m0, q2, m2, F);            // k = 3
            from_prev(F, G);
            add(a0, c0[j1], F);
            add(a1, c1[h0], G);
        }
    } else {
        // one node per lane: pair (i, i + k) on lane i, k = 1 .. (N1 - 1) / 2
        HalfQ<R> qi;
        R mi[3];
        node(pos, qi, mi);
#pragma unroll
        for (int k = 1; k <= N1 / 2; ++k) {
            const int jp = pos + k < N1 ? pos + k : pos + k - N1, jm = pos - k >= 0 ? pos - k : pos - k + N1;
            HalfQ<R> qj;
            R mj[3], F[5];
            node(jp, qj, mj);
            pair(qi, mi, qj, mj, F);
            const R cj = sS[pos * N1 + jp], cr = sS[pos * N1 + jm];
#pragma unroll
            for (int s = 0; s < 5; ++s) {
                const R g = __shfl_sync(0xffffffffu, F[s], jm * SPW + seg);
                acc[0][s] += cj * F[s];
                acc[0][s] += cr * g;
            }
        }
    }
}

// The five DOFs of one node in a Butcher RK stage: the running sum, u_{n+1} and the next stage's input
// from the stage's time derivative k (un: u_n, bs: the sum so far).
template <int NP>
__device__ __forceinline__ void rk_node(const StageArgs& a, size_t o5, const double k[5], const double un[5],
                                        const double bs[5]) {
#pragma unroll
    for (int s = 0; s < 5; ++s) {
        const size_t dof = o5 + s * NP;
        const double sum = bs[s] + a.c_acc * k[s];
        if (a.acc_out) a.acc_out[dof] = sum;
        if (a.final_out) {
            if (a.comp) {   // compensated u_{n+1} = u_n + increment
                const double y = sum - a.comp[dof];
                const double t = un[s] + y;
                a.comp[dof] = (t - un[s]) - y;
                a.final_out[dof] = t;
            } else {
                a.final_out[dof] = a.inc_mode ? un[s] + sum : sum;
            }
        }
        if (a.next) {
            const double cin = a.carry_in ? a.carry_in[dof] : 0.0;
            a.next[dof] = (cin + a.a_next * k[s]) * a.dt + un[s];
        }
        if (a.carry_out) a.carry_out[dof] = a.a_carry * k[s];
    }
}

// what the threads of a tile share beside the rows: the cell of each slot (-1: none) and the span of the
// nodes' high words of rho and b (min, max each)
template <int CPC> struct LineShared {
    int cell[CPC];
    int span[4];
};

template <typename R, int N1, int CPC, bool VISC, bool CURV, bool WIDE = false>
__device__ __forceinline__ void line_tile(const StageArgs& a, LineShared<CPC>& sh) {
    using L = LineLayout<R, N1, CPC, CURV, WIDE>;
    constexpr int NA = L::NA;
    constexpr int NP = L::NP, NF = L::NF, NT = L::NT, NQ = L::NQ, H = L::H, NPL = L::NPL, NS = L::NS, ZP = L::ZP;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    R* sm = reinterpret_cast<R*>(smem_raw);
    R* sS = sm + L::oS;
    R* sW = sS + N1 * N1;
    R* sB = sm + L::oB;
    R* sQ = sm + L::oQ;
    R* sL = sm + L::oL;
    R* sA = sm + L::oA;
    R* sT = sm + L::oT;
    const int* scell = sh.cell;
    Cst<R> cst; cst.load(a.pc);
    constexpr int tp = (int)TP_CH, cf = (int)CF_EC_ROE;
    const int tid = threadIdx.x;

    // L2 prefetch of what the epilogue reads, FP64 (0.224 against 0.230 ms at 32^3 cells, p = 3; the
    // precision form is faster without: 0.142 against 0.150 ms)
    if constexpr (!L::F32) {
        for (int c = 0; c < CPC; ++c) {
            if (scell[c] < 0) continue;
            const size_t o = (size_t)scell[c] * 5 * NP;
            constexpr int nl = (5 * NP + 15) / 16;
            if (a.mode == 2) {
                for (int i = tid; i < (a.acc_in ? 2 : 1) * nl; i += NT) {
                    const double* b = i < nl ? a.Un : a.acc_in;
                    const int e = (i < nl ? i : i - nl) * 16;
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(b + o + (e < 5 * NP ? e : 5 * NP - 1)));
                }
            }
            if constexpr (VISC) {
                constexpr int VT = viscous_terms_per_cell<N1>();
                const R* fb = static_cast<const R*>(a.Fv) + (size_t)scell[c] * VT;
                for (int i = tid; i < (VT + 15) / 16; i += NT)
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(fb + (i * 16 < VT ? i * 16 : VT - 1)));
            }
        }
    }
    for (int i = tid; i < N1 * N1; i += NT) {
        sS[i] = (R)a.ops->Dsk[(i / N1) * MAXN1 + (i % N1)];
        sB[i] = (R)a.ops->B[(i / N1) * MAXN1 + (i % N1)];
    }
    if (tid == 0) sW[0] = R(1) / (R)a.ops->w[0];   // 1 / w_end

    // ---- node quantities
    int lo_r = 0x7fffffff, hi_r = (int)0x80000000, lo_b = lo_r, hi_b = hi_r;
#pragma unroll
    for (int it = tid; it < CPC * NP; it += NT) {
        const int c = it / NP, node = it - c * NP;
        const int cc = scell[c];
        if (cc < 0) continue;
        double ud[5];
#pragma unroll
        for (int s = 0; s < 5; ++s) ud[s] = __ldg(&a.U[((size_t)cc * 5 + s) * NP + node]);
        if constexpr (!L::F32) {
            if (ud[0] < 0.0) atomicOr(a.status, ST_NONPHYSICAL);
        } else {
            check_state_fp64(ud, a.pc.gm1, a.status);
        }
        R u[5];
#pragma unroll
        for (int s = 0; s < 5; ++s) u[s] = (R)ud[s];
        NodeQ<R> q;
        node_prepare<R, LOG_HERE>(u, tp, cst.gm1, q, L::F32 ? nullptr : a.status);
        R* Q = sQ + c * NQ * NS + node + (node / NF) * (ZP - NF);
        Q[0] = R(0.5) * q.rho; Q[NS] = R(0.5) * q.v[0]; Q[2 * NS] = R(0.5) * q.v[1]; Q[3 * NS] = R(0.5) * q.v[2];
        Q[4 * NS] = q.p; Q[5 * NS] = q.E; Q[6 * NS] = q.b; Q[7 * NS] = R(0.25) * q.vsq;
        lo_r = min(lo_r, hi_word(q.rho)); hi_r = max(hi_r, hi_word(q.rho));
        lo_b = min(lo_b, hi_word(q.b)); hi_b = max(hi_b, hi_word(q.b));
        if constexpr (CURV) {
#pragma unroll
            for (int i = 0; i < 9; ++i)
                Q[(8 + i) * NS] = R(0.5) * (R)__ldg(&a.metric[((size_t)cc * 10 + i) * NP + node]);
        }
    }
    lo_r = __reduce_min_sync(0xffffffffu, lo_r); hi_r = __reduce_max_sync(0xffffffffu, hi_r);
    lo_b = __reduce_min_sync(0xffffffffu, lo_b); hi_b = __reduce_max_sync(0xffffffffu, hi_b);
    if ((tid & 31) == 0) {
        atomicMin(&sh.span[0], lo_r); atomicMax(&sh.span[1], hi_r);
        atomicMin(&sh.span[2], lo_b); atomicMax(&sh.span[3], hi_b);
    }
    __syncthreads();
    const bool smooth = series_span<R>(sh.span[0], sh.span[1]) && series_span<R>(sh.span[2], sh.span[3]);
    if (!smooth) {   // strong gradients somewhere in the tile: the logarithms of every node
        for (int it = tid; it < CPC * NP; it += NT) {
            const int c = it / NP, node = it - c * NP;
            if (scell[c] < 0) continue;
            const int o = node + (node / NF) * (ZP - NF);
            const R* Q = sQ + c * NQ * NS + o;
            sL[c * 2 * NS + o] = rlog<R>(R(2) * Q[0]);
            sL[c * 2 * NS + NS + o] = rlog<R>(Q[6 * NS]);
        }
        __syncthreads();
    }

    // ---- the numerical fluxes at the face nodes (canonical orientation: the left cell is the interior
    // side), lifted into this cell with 1 / w_end. The neighbour's values come straight from its rows
    // (gathering them ahead, into registers or by asynchronous copies, cost more CTAs per SM than its
    // latency: 0.355 ms against 0.326 at 24^3 cells, p = 5 in FP64)
    {
        constexpr int FI = CPC * 6 * NF;
        const R inv_wend = sW[0];
#pragma unroll 1
        for (int it = tid; it < FI; it += NT) {
            const int fn = it % NF, f = (it / NF) % 6, c = it / (NF * 6);
            const int cell = scell[c];
            if (cell < 0) continue;
            const int d = f >> 1, side = f & 1;
            // the frame's axes: the face normal first on affine cells
            const int d1 = CURV ? 0 : d, d2 = CURV ? 1 : d == 2 ? 0 : d + 1, d3 = CURV ? 2 : d == 0 ? 2 : d - 1;
            const R sgn = side ? R(1) : R(-1);
            const int on = line_node<N1>(d, fn, side ? N1 - 1 : 0);
            const R* Q = sQ + c * NQ * NS + on + (on / NF) * (ZP - NF);
            const int cn = __ldg(&a.nbr[cell * 6 + f]);
            const double* ug = a.U + (size_t)cn * 5 * NP + line_node<N1>(d, fn, side ? 0 : N1 - 1);
            R re[5], vn[4];
            re[0] = (R)__ldg(&ug[0]); re[1] = (R)__ldg(&ug[(1 + d1) * NP]); re[2] = (R)__ldg(&ug[(1 + d2) * NP]);
            re[3] = (R)__ldg(&ug[(1 + d3) * NP]); re[4] = (R)__ldg(&ug[4 * NP]);
            if constexpr (VISC) {   // the neighbour's block of the opposite face: same node order
                const R* fb = static_cast<const R*>(a.Fv) + (size_t)cn * viscous_terms_per_cell<N1>() + 4 * NP +
                              (f ^ 1) * 4 * NF + fn;
                vn[0] = __ldg(&fb[d1 * NF]); vn[1] = __ldg(&fb[d2 * NF]); vn[2] = __ldg(&fb[d3 * NF]);
                vn[3] = __ldg(&fb[3 * NF]);
            }
            NodeQ<R> qo, qe;
            qo.rho = R(2) * Q[0]; qo.v[0] = R(2) * Q[(1 + d1) * NS]; qo.v[1] = R(2) * Q[(1 + d2) * NS];
            qo.v[2] = R(2) * Q[(1 + d3) * NS];
            qo.p = Q[4 * NS]; qo.E = Q[5 * NS]; qo.b = Q[6 * NS]; qo.vsq = R(4) * Q[7 * NS];
            node_prepare<R, LOG_HERE, N1 % 2 == 0>(re, tp, cst.gm1, qe, nullptr);
            R F[5], term[5];
            if constexpr (CURV) {
                const R m[3] = {R(2) * Q[(8 + 0 + d) * NS], R(2) * Q[(8 + 3 + d) * NS], R(2) * Q[(8 + 6 + d) * NS]};
                const R J = rsqrt_<R>(m[0] * m[0] + m[1] * m[1] + m[2] * m[2]);
                const R nrm[3] = {qdiv<R>(m[0], J), qdiv<R>(m[1], J), qdiv<R>(m[2], J)};
                NodeQ<R> ql = qo, qr = qe;
                if (!side) { ql = qe; qr = qo; }
                conv_num_flux_n<R, LOG_HERE>(re, re, ql, qr, nrm, tp, cf, cst, F);
#pragma unroll
                for (int s = 0; s < 5; ++s) term[s] = -sgn * J * F[s];
            } else {
                NodeQ<R> ql = qo, qr = qe;   // (re is not read by this flux set: the states enter through q)
                if (!side) { ql = qe; qr = qo; }
                conv_num_flux<R, 0, LOG_HERE>(re, re, ql, qr, tp, cf, cst, F);
#pragma unroll
                for (int s = 0; s < 5; ++s) term[s] = -sgn * F[s];
            }
            if constexpr (VISC) {
                const R* fv = static_cast<const R*>(a.Fv) + (size_t)cell * viscous_terms_per_cell<N1>() + 4 * NP +
                              f * 4 * NF + fn;
                const int dk[4] = {d1, d2, d3, 3};
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const R Fo = __ldg(&fv[dk[k] * NF]);
                    const R Fn = R(0.5) * (Fo + vn[k]);
                    term[1 + k] += sgn * (Fo - Fn);
                }
            }
            R* T = sT + (c * 6 + f) * 5 * NF + fn;
            T[0] = term[0] * inv_wend; T[(1 + d1) * NF] = term[1] * inv_wend;
            T[(1 + d2) * NF] = term[2] * inv_wend; T[(1 + d3) * NF] = term[3] * inv_wend;
            T[4 * NF] = term[4] * inv_wend;
        }
    }

    // ---- volume, direction by direction
    {
        const int lane = tid & 31;
        const int pos = lane / L::SPW < H ? lane / L::SPW : 0, seg = lane % L::SPW;   // place on the line, line
        const int dir = WIDE ? tid / L::LNT : 0;   // wide: the direction of this warp
        const int lineid = ((tid - dir * L::LNT) >> 5) * L::SPW + seg;
        const bool lvalid = lane < H * L::SPW && lineid < CPC * NF;   // (idle lanes run along on line 0)
        const int lc = lvalid ? lineid / NF : 0, line = lvalid ? lineid - lc * NF : 0;
        const R* Qc = sQ + lc * NQ * NS;
        const R* Lc = sL + lc * 2 * NS;
        R* Ac = sA + (lc * NA + 5 * dir) * NS;
        auto directions = [&](auto lm) {
            constexpr int LM = decltype(lm)::value;
#pragma unroll 1
            for (int d = dir; d < (WIDE ? dir + 1 : 3); ++d) {
                const int st = d == 0 ? 1 : d == 1 ? N1 : ZP;
                const int la = line % N1, lb = line / N1;
                const int base = d == 0 ? N1 * la + ZP * lb : d == 1 ? la + ZP * lb : la + N1 * lb;
                const int d1 = CURV ? 0 : d, d2 = CURV ? 1 : d == 2 ? 0 : d + 1, d3 = CURV ? 2 : d == 0 ? 2 : d - 1;
                const int r1 = (1 + d1) * NS, r2 = (1 + d2) * NS, r3 = (1 + d3) * NS;
                R acc[NPL][5];
                line_pairs<R, N1, NS, CURV, LM>(LineRows<R>{Qc, Qc + 6 * NS, Lc, Qc + (8 + d) * NS, r1, r2, r3}, base, st,
                                                pos, seg, sS, cst, acc);
                if (!WIDE && d > 0) __syncthreads();   // the previous direction's terms are in place
                if (lvalid) {
                    const int row[5] = {0, r1, r2, r3, 4 * NS};
#pragma unroll
                    for (int e = 0; e < NPL; ++e) {
                        R* A0 = Ac + base + (NPL * pos + e) * st;
#pragma unroll
                        for (int s = 0; s < 5; ++s) A0[row[s]] = WIDE || d == 0 ? acc[e][s] : A0[row[s]] + acc[e][s];
                    }
                }
            }
        };
        if (smooth) directions(std::integral_constant<int, LOG_NONE>());
        else directions(std::integral_constant<int, LOG_STORED>());
    }
    __syncthreads();

    // ---- per node: G = -volume - viscous divergence + lifted faces, mass inverse, outputs
    constexpr int PER = (CPC * NP + NT - 1) / NT;
    const bool inv = a.mode != 0 && a.fr;
#pragma unroll
    for (int r = 0; r < PER; ++r) {
        const int it = tid + r * NT;
        const int c = it / NP, node = it - c * NP;
        const int cc = it < CPC * NP ? scell[c] : -1;
        if (cc < 0) continue;
        const size_t o5 = (size_t)cc * 5 * NP + node;
        // this node's inputs in flight before anything is stored (outputs may alias them DOF by DOF)
        double un[5], bs[5];
        const bool rk = a.mode == 2 && !inv;
        if (rk) {
#pragma unroll
            for (int s = 0; s < 5; ++s) {
                un[s] = a.Un[o5 + s * NP];
                bs[s] = a.acc_in ? a.acc_in[o5 + s * NP] : (a.inc_mode ? 0.0 : un[s]);
            }
        }
        R dv[4];
        if constexpr (VISC) {
            const R* p = static_cast<const R*>(a.Fv) + (size_t)cc * viscous_terms_per_cell<N1>() + node;
#pragma unroll
            for (int k = 0; k < 4; ++k) dv[k] = __ldg(&p[k * NP]);
        }
        R* A = sA + c * NA * NS + node + (node / NF) * (ZP - NF);
        R G[5];
#pragma unroll
        for (int s = 0; s < 5; ++s) G[s] = WIDE ? -((A[s * NS] + A[(5 + s) * NS]) + A[(10 + s) * NS]) : -A[s * NS];
        if constexpr (VISC) {
#pragma unroll
            for (int k = 0; k < 4; ++k) G[1 + k] -= dv[k];
        }
        const int cx[3] = {node % N1, (node / N1) % N1, node / NF};
#pragma unroll
        for (int f = 0; f < 6; ++f) {
            const int dn = f >> 1;
            if (cx[dn] != ((f & 1) ? N1 - 1 : 0)) continue;
            const int t1 = dn == 0 ? 1 : 0, t2 = dn == 2 ? 1 : 2;
            const R* tr = sT + (c * 6 + f) * 5 * NF + cx[t2] * N1 + cx[t1];
#pragma unroll
            for (int s = 0; s < 5; ++s) G[s] += tr[s * NF];
        }
        if (inv) {
#pragma unroll
            for (int s = 0; s < 5; ++s) A[s * NS] = G[s];
            continue;
        }
        double k[5];
        if (a.mode == 0) {
            const double W = a.ops->w[cx[0]] * a.ops->w[cx[1]] * a.ops->w[cx[2]];
#pragma unroll
            for (int s = 0; s < 5; ++s) a.out[o5 + s * NP] = CURV ? W * (double)G[s] : W * a.h * a.h * (double)G[s];
            continue;
        }
        const double ij = CURV ? __ldg(&a.metric[((size_t)cc * 10 + 9) * NP + node]) : a.inv_h;
#pragma unroll
        for (int s = 0; s < 5; ++s) k[s] = (double)G[s] * ij;
        if (a.mode == 1) {
#pragma unroll
            for (int s = 0; s < 5; ++s) a.out[o5 + s * NP] = k[s];
            continue;
        }
        rk_node<NP>(a, o5, k, un, bs);
    }
    if (!inv) return;
    // FR mass inverse B (x) B (x) B, direction by direction, between the volume terms' rows and the
    // node quantities' rows (curvilinear: the weight-adjusted inverse, 1 / det J between two applications)
    constexpr int SRC = NA * NS, DST = NQ * NS;
    R* src = sA;
    R* dst = sQ;
    int ns = SRC, nd = DST;
    for (int rep = 0; rep < (CURV ? 2 : 1); ++rep) {
        if (rep == 1) {
            __syncthreads();
            for (int it = tid; it < CPC * NP; it += NT) {
                const int c = it / NP, node = it - c * NP;
                if (scell[c] < 0) continue;
                const double ij = __ldg(&a.metric[((size_t)scell[c] * 10 + 9) * NP + node]);
                const int o = c * ns + node + (node / NF) * (ZP - NF);
                for (int s = 0; s < 5; ++s) src[o + s * NS] = (R)((double)src[o + s * NS] * ij);
            }
        }
        for (int e = 0; e < 3; ++e) {
            __syncthreads();
            const int se = e == 0 ? 1 : e == 1 ? N1 : ZP, sd = e == 0 ? 1 : e == 1 ? N1 : NF;
            for (int it = tid; it < CPC * NP; it += NT) {
                const int c = it / NP, node = it - c * NP;
                if (scell[c] < 0) continue;
                const int pos = (node / sd) % N1, o = node + (node / NF) * (ZP - NF), b0 = o - pos * se;
                for (int s = 0; s < 5; ++s) {
                    R v = R(0);
                    for (int l = 0; l < N1; ++l) v += sB[pos * N1 + l] * src[c * ns + s * NS + b0 + l * se];
                    dst[c * nd + s * NS + o] = v;
                }
            }
            R* t = src; src = dst; dst = t;
            const int n = ns; ns = nd; nd = n;
        }
    }
    __syncthreads();
    for (int it = tid; it < CPC * NP; it += NT) {
        const int c = it / NP, node = it - c * NP;
        const int cc = scell[c];
        if (cc < 0) continue;
        const size_t o5 = (size_t)cc * 5 * NP + node;
        double k[5], un[5], bs[5];
#pragma unroll
        for (int s = 0; s < 5; ++s) {
            const double G = (double)src[c * ns + s * NS + node + (node / NF) * (ZP - NF)];
            k[s] = CURV ? G : G * a.inv_h;
        }
        if (a.mode == 1) {
#pragma unroll
            for (int s = 0; s < 5; ++s) a.out[o5 + s * NP] = k[s];
            continue;
        }
#pragma unroll
        for (int s = 0; s < 5; ++s) {
            un[s] = a.Un[o5 + s * NP];
            bs[s] = a.acc_in ? a.acc_in[o5 + s * NP] : (a.inc_mode ? 0.0 : un[s]);
        }
        rk_node<NP>(a, o5, k, un, bs);
    }
}

// cell of slot c of the CTA: cells in order, or from the tile list (tc cells per entry); -1 past the end
__device__ __forceinline__ int line_cell(const StageArgs& a, int slot, int tc) {
    if (!a.tiles) {
        const int cell = a.cell_begin + slot;
        return cell < a.nc ? cell : -1;
    }
    const int e = slot / tc;
    if (e >= a.ntiles) return -1;
    const int cell = __ldg(&a.tiles[e]) + slot - e * tc;
    return cell < a.nc ? cell : -1;
}

// Wide form: one warp group per direction instead of one after the other, for meshes whose cells do not fill
// the SMs with warps and whose time is one tile's chain of dependent operations.
template <typename R, int N1, int CPC, bool VISC, bool CURV, bool WIDE = false>
__global__ void __launch_bounds__(LineLayout<R, N1, CPC, CURV, WIDE>::NT, LineLayout<R, N1, CPC, CURV, WIDE>::MINB)
line_kernel(const StageArgs a, int tc) {
    __shared__ LineShared<CPC> sh;
    if (threadIdx.x < CPC) sh.cell[threadIdx.x] = line_cell(a, (int)blockIdx.x * CPC + (int)threadIdx.x, tc);
    if (threadIdx.x < 4) sh.span[threadIdx.x] = (threadIdx.x & 1) ? (int)0x80000000 : 0x7fffffff;
    __syncthreads();
    line_tile<R, N1, CPC, VISC, CURV, WIDE>(a, sh);
}

// The batched form (residual_kernel_batched's tile list and instance table) over the same tile.
template <typename R, int N1, int CPC, bool CURV>
__global__ void __launch_bounds__(LineLayout<R, N1, CPC, CURV>::NT, LineLayout<R, N1, CPC, CURV>::BATCHED)
line_kernel_batched(const StageArgs* __restrict__ inst, const BatchTile* __restrict__ tiles, int ntiles) {
    __shared__ __align__(16) StageArgs sa;
    __shared__ LineShared<CPC> sh;
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const BatchTile tile = tiles[t];
        const int* src = reinterpret_cast<const int*>(inst + tile.inst);
        int* dst = reinterpret_cast<int*>(&sa);
        for (int i = threadIdx.x; i < (int)(sizeof(StageArgs) / sizeof(int)); i += blockDim.x) dst[i] = src[i];
        if (threadIdx.x < 4) sh.span[threadIdx.x] = (threadIdx.x & 1) ? (int)0x80000000 : 0x7fffffff;
        __syncthreads();
        if (threadIdx.x < CPC)
            sh.cell[threadIdx.x] = tile.cell0 + (int)threadIdx.x < sa.nc ? tile.cell0 + (int)threadIdx.x : -1;
        __syncthreads();
        line_tile<R, N1, CPC, false, CURV>(sa, sh);
        __syncthreads();
    }
}

} // namespace ph
