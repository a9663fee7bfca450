// Taylor-Green integrated quantities with QGauss(p+11) over-integration
// (PeriodicTurbulence::compute_and_update_integrated_quantities,
// src/flow_solver/flow_solver_cases/periodic_turbulence.cpp:439-672).
//
// One CTA per cell. The solution is contracted with the 1-D basis in x once and kept
// in shared memory (value and x-derivative); each thread owns one (qx, qy) column of
// cubature points and walks qz, contracting y and z on the fly. Per-cell partial sums
// go to global memory and are summed on the host in cell order (deterministic).
//
// Curvilinear cells (CURV): the node coordinates are three more nodal fields carried
// through the same contractions; their derivatives at a cubature point are the mapping
// Jacobian there (the mapping has the solution's degree), which gives det J for the
// weights and J^-1 for the physical gradients.
//
// FULL: all nine quantities of the reference's IntegratedQuantitiesEnum
// (periodic_turbulence.h:176-186) with the integrands of navier_stokes.cpp:399-740 and
// euler.cpp:378-402. The palinstrophy needs the gradient of the vorticity after its L2
// projection onto the solution basis (vol_projection_operator, operators.cpp:1865-1889):
// each column thread accumulates the qz-projection of the vorticity while it walks qz,
// the qy and qx projections follow in shared memory, and a second pass over the
// cubature points differentiates the projected vorticity.
#pragma once
#include "ph_kernels.cuh"

namespace ph {

constexpr int MAXNE = 20;

struct IntegralTab {
    double B[MAXNE * MAXN1];
    double dB[MAXNE * MAXN1];
    double P[MAXN1 * MAXNE];   // 1-D L2 projection onto the solution basis, [node][cubature point]
    double w[MAXNE];
    double x[MAXNE];           // cubature points on [0, 1]
};

// Viscosity and gas constants of the integrands (the reference evaluates them with a
// NavierStokes physics object whatever the PDE).
struct IntegralConst {
    double h, gam, gm1, mach2, temp_ratio, const_visc;
    int use_const_visc;
};

// partial sums per cell: FULL = the nine quantities then the max wave speed;
// otherwise kinetic energy, enstrophy, max wave speed
template <bool FULL> __host__ __device__ constexpr int integral_partials() { return FULL ? 10 : 3; }

template <int N1, bool CURV, bool FULL>
__host__ __device__ constexpr size_t integrals_smem_bytes() {
    constexpr int NFLD = CURV ? 8 : 5;
    constexpr int NE = N1 + 10;
    constexpr size_t base = NFLD * N1 * N1 * N1 + 2 * NFLD * N1 * N1 * NE;
    constexpr size_t proj = FULL ? 3 * NE * NE * N1 + 3 * NE * N1 * N1 : 0;
    return sizeof(double) * (base + proj);
}

// Physical gradient of nf nodal fields at one cubature point from the x-contracted values
// and x-derivatives (sT0, sT1); fields listed in fld[].
template <int N1, int NE, int NF>
__device__ __forceinline__ void point_fields(const double* sT0, const double* sT1, const double* sB, const double* sdB,
                                             const int (&fld)[NF], int qx, int qy, int qz, double (&u)[NF],
                                             double (&g)[NF][3]) {
    constexpr int NT2 = N1 * N1 * NE;
#pragma unroll
    for (int f = 0; f < NF; ++f) {
        const int s = fld[f];
        double v = 0.0, gx = 0.0, gy = 0.0, gz = 0.0;
#pragma unroll
        for (int k = 0; k < N1; ++k) {
            double a0 = 0.0, a1 = 0.0, a2 = 0.0;
#pragma unroll
            for (int j = 0; j < N1; ++j) {
                const double t0 = sT0[s * NT2 + (k * N1 + j) * NE + qx];
                const double t1 = sT1[s * NT2 + (k * N1 + j) * NE + qx];
                a0 += sB[qy * N1 + j] * t0;
                a1 += sB[qy * N1 + j] * t1;
                a2 += sdB[qy * N1 + j] * t0;
            }
            const double b = sB[qz * N1 + k], db = sdB[qz * N1 + k];
            v += b * a0; gx += b * a1; gy += b * a2; gz += db * a0;
        }
        u[f] = v; g[f][0] = gx; g[f][1] = gy; g[f][2] = gz;
    }
}

// J^-1 and det J from the reference gradients of the three coordinate fields
// (J[m][j] = dX_m/dxi_j; physical gradient = reference gradient times J^-1).
__device__ __forceinline__ double inverse_jacobian(const double (&gx)[3][3], double (&I)[3][3]) {
    const double(&J)[3][3] = gx;
    const double dj = J[0][0] * (J[1][1] * J[2][2] - J[1][2] * J[2][1]) -
                      J[0][1] * (J[1][0] * J[2][2] - J[1][2] * J[2][0]) +
                      J[0][2] * (J[1][0] * J[2][1] - J[1][1] * J[2][0]);
    I[0][0] = (J[1][1] * J[2][2] - J[1][2] * J[2][1]) / dj;
    I[0][1] = (J[0][2] * J[2][1] - J[0][1] * J[2][2]) / dj;
    I[0][2] = (J[0][1] * J[1][2] - J[0][2] * J[1][1]) / dj;
    I[1][0] = (J[1][2] * J[2][0] - J[1][0] * J[2][2]) / dj;
    I[1][1] = (J[0][0] * J[2][2] - J[0][2] * J[2][0]) / dj;
    I[1][2] = (J[0][2] * J[1][0] - J[0][0] * J[1][2]) / dj;
    I[2][0] = (J[1][0] * J[2][1] - J[1][1] * J[2][0]) / dj;
    I[2][1] = (J[0][1] * J[2][0] - J[0][0] * J[2][1]) / dj;
    I[2][2] = (J[0][0] * J[1][1] - J[0][1] * J[1][0]) / dj;
    return dj;
}

template <int NF>
__device__ __forceinline__ void to_physical(double (&g)[NF][3], int nf, const double (&I)[3][3]) {
#pragma unroll
    for (int s = 0; s < NF; ++s) {
        if (s >= nf) break;
        const double r0 = g[s][0], r1 = g[s][1], r2 = g[s][2];
#pragma unroll
        for (int d = 0; d < 3; ++d) g[s][d] = r0 * I[0][d] + r1 * I[1][d] + r2 * I[2][d];
    }
}

template <int N1, bool CURV, bool FULL>
__global__ void integrals_kernel(const double* __restrict__ U, const double* __restrict__ X,
                                 const double* __restrict__ origin, const IntegralTab* tab, int nc, IntegralConst ic,
                                 double* __restrict__ partial) {
    constexpr int NE = N1 + 10;
    constexpr int NP = N1 * N1 * N1;
    constexpr int NT2 = N1 * N1 * NE;
    constexpr int NFLD = CURV ? 8 : 5;   // state (+ node coordinates)
    constexpr int NQ = integral_partials<FULL>();
    constexpr int NACC = FULL ? 9 : 2;   // summed quantities (the wave speed is a max)
    __shared__ double sB[NE * N1], sdB[NE * N1], sP[FULL ? N1 * NE : 1], sw[NE], sx[NE];
    __shared__ double red[NQ][32];
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* sU = reinterpret_cast<double*>(smem_raw);
    double* sT0 = sU + NFLD * NP;       // [s][(k*N1 + j)*NE + qx], x-contracted values
    double* sT1 = sT0 + NFLD * NT2;     // x-contracted x-derivatives
    double* sWz = sT1 + NFLD * NT2;     // FULL: vorticity projected in z, [c][qy*NE + qx][k]
    double* sWy = sWz + 3 * NE * NE * N1;   // FULL: ... and in y, [c][(k*N1 + j)*NE + qx]
    const int cell = blockIdx.x;
    const int tid = threadIdx.x;
    for (int i = tid; i < NE * N1; i += blockDim.x) { sB[i] = tab->B[i]; sdB[i] = tab->dB[i]; }
    if constexpr (FULL) {
        for (int i = tid; i < N1 * NE; i += blockDim.x) sP[i] = tab->P[i];
    }
    for (int i = tid; i < NE; i += blockDim.x) { sw[i] = tab->w[i]; sx[i] = tab->x[i]; }
    for (int i = tid; i < 5 * NP; i += blockDim.x) sU[i] = U[(size_t)cell * 5 * NP + i];
    if constexpr (CURV) {
        for (int i = tid; i < 3 * NP; i += blockDim.x) sU[5 * NP + i] = X[(size_t)cell * 3 * NP + i];
    }
    __syncthreads();
    for (int i = tid; i < NFLD * NT2; i += blockDim.x) {
        const int qx = i % NE, kj = (i / NE) % (N1 * N1), s = i / NT2;
        double v = 0.0, dv = 0.0;
        for (int a = 0; a < N1; ++a) {
            const double u = sU[s * NP + kj * N1 + a];
            v += sB[qx * N1 + a] * u;
            dv += sdB[qx * N1 + a] * u;
        }
        sT0[i] = v;
        sT1[i] = dv;
    }
    __syncthreads();
    const double h = ic.h, inv_h = 1.0 / h, detj = h * h * h;
    const double gam = ic.gam, gm1 = ic.gm1;
    double acc[NACC];
#pragma unroll
    for (int i = 0; i < NACC; ++i) acc[i] = 0.0;
    double wave = 0.0;
    double o0rg[3] = {0.0, 0.0, 0.0};
    if constexpr (FULL && !CURV) {
        for (int d = 0; d < 3; ++d) o0rg[d] = origin[3 * cell + d];
    }
    int fld[NFLD];
#pragma unroll
    for (int s = 0; s < NFLD; ++s) fld[s] = s;
    for (int col = tid; col < NE * NE; col += blockDim.x) {
        const int qx = col % NE, qy = col / NE;
        double zp[FULL ? 3 : 1][FULL ? N1 : 1];   // FULL: vorticity projected along this column
#pragma unroll
        for (int c = 0; c < (FULL ? 3 : 1); ++c)
#pragma unroll
            for (int k = 0; k < (FULL ? N1 : 1); ++k) zp[c][k] = 0.0;
        for (int qz = 0; qz < NE; ++qz) {
            double u[NFLD], g[NFLD][3];
            point_fields<N1, NE, NFLD>(sT0, sT1, sB, sdB, fld, qx, qy, qz, u, g);
            double wdet = detj;
            if constexpr (CURV) {
                const double gx[3][3] = {{g[5][0], g[5][1], g[5][2]}, {g[6][0], g[6][1], g[6][2]},
                                         {g[7][0], g[7][1], g[7][2]}};
                double I[3][3];
                wdet = inverse_jacobian(gx, I);
                to_physical<NFLD>(g, 5, I);
            } else {
#pragma unroll
                for (int s = 0; s < 5; ++s)
#pragma unroll
                    for (int d = 0; d < 3; ++d) g[s][d] *= inv_h;
            }
            const double rho = u[0];
            double v[3], v2 = 0.0;
#pragma unroll
            for (int d = 0; d < 3; ++d) { v[d] = u[1 + d] / rho; v2 += v[d] * v[d]; }
            double gv[3][3];
#pragma unroll
            for (int a = 0; a < 3; ++a)
#pragma unroll
                for (int d = 0; d < 3; ++d) gv[a][d] = (g[1 + a][d] - v[a] * g[0][d]) / rho;
            const double o0 = gv[2][1] - gv[1][2], o1 = gv[0][2] - gv[2][0], o2 = gv[1][0] - gv[0][1];
            const double om2 = o0 * o0 + o1 * o1 + o2 * o2;
            const double wt = sw[qx] * sw[qy] * sw[qz] * wdet;
            acc[0] += 0.5 * rho * v2 * wt;
            acc[1] += 0.5 * rho * om2 * wt;
            const double p = gm1 * (u[4] - 0.5 * rho * v2);
            if constexpr (FULL) {
                double S[3][3], dil = 0.0;
#pragma unroll
                for (int a = 0; a < 3; ++a)
#pragma unroll
                    for (int b = 0; b < 3; ++b) S[a][b] = 0.5 * (gv[a][b] + gv[b][a]);
#pragma unroll
                for (int d = 0; d < 3; ++d) dil += gv[d][d];
                double s2 = 0.0, sd2 = 0.0;
#pragma unroll
                for (int a = 0; a < 3; ++a)
#pragma unroll
                    for (int b = 0; b < 3; ++b) {
                        const double dv = S[a][b] - (a == b ? dil / 3.0 : 0.0);
                        s2 += S[a][b] * S[a][b];
                        sd2 += dv * dv;
                    }
                // Sutherland's law in the nondimensional temperature (navier_stokes.cpp:241-300)
                const double T = gam * ic.mach2 * (p / rho);
                const double mu = ic.use_const_visc ? 1.0 * ic.const_visc
                                                    : ((1.0 + ic.temp_ratio) / (T + ic.temp_ratio)) * pow(T, 1.5);
                double r2 = 0.0;
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    double xd;
                    if constexpr (CURV) xd = u[5 + d];
                    else xd = o0rg[d] + h * sx[d == 0 ? qx : d == 1 ? qy : qz];
                    r2 += xd * xd;
                }
                acc[2] += p * dil * wt;
                acc[3] += mu * sd2 * wt;
                acc[4] += mu * s2 * wt;
                acc[5] += 0.5 * v2 * wt;
                acc[6] += 0.5 * om2 * wt;
                acc[8] += 0.5 * r2 * sqrt(om2) * wt;
#pragma unroll
                for (int k = 0; k < N1; ++k) {
                    const double pk = sP[k * NE + qz];
                    zp[0][k] += pk * o0; zp[1][k] += pk * o1; zp[2][k] += pk * o2;
                }
            }
            const double c = sqrt(p * gam / rho);
            const double ws = sqrt(v2) + c;
            wave = ws > wave ? ws : wave;
        }
        if constexpr (FULL) {
#pragma unroll
            for (int c = 0; c < 3; ++c)
#pragma unroll
                for (int k = 0; k < N1; ++k) sWz[(c * NE * NE + col) * N1 + k] = zp[c][k];
        }
    }
    if constexpr (FULL) {
        __syncthreads();
        // projection in y: sWy[c][(k*N1 + j)*NE + qx] = sum_qy P[j][qy] sWz[c][qy*NE + qx][k]
        for (int i = tid; i < 3 * N1 * N1 * NE; i += blockDim.x) {
            const int qx = i % NE, j = (i / NE) % N1, k = (i / (NE * N1)) % N1, c = i / (NE * N1 * N1);
            double v = 0.0;
            for (int qy = 0; qy < NE; ++qy) v += sP[j * NE + qy] * sWz[(c * NE * NE + qy * NE + qx) * N1 + k];
            sWy[i] = v;
        }
        __syncthreads();
        // projection in x: coefficients into the (no longer needed) state slots 0..2 of sU
        for (int i = tid; i < 3 * NP; i += blockDim.x) {
            const int a = i % N1, kj = (i / N1) % (N1 * N1), c = i / NP;
            double v = 0.0;
            for (int qx = 0; qx < NE; ++qx) v += sP[a * NE + qx] * sWy[(c * N1 * N1 + kj) * NE + qx];
            sU[i] = v;
        }
        __syncthreads();
        // x-contraction of the projected vorticity into slots 0..2 (coordinates stay in 5..7)
        for (int i = tid; i < 3 * NT2; i += blockDim.x) {
            const int qx = i % NE, kj = (i / NE) % (N1 * N1), s = i / NT2;
            double v = 0.0, dv = 0.0;
            for (int a = 0; a < N1; ++a) {
                const double u = sU[s * NP + kj * N1 + a];
                v += sB[qx * N1 + a] * u;
                dv += sdB[qx * N1 + a] * u;
            }
            sT0[i] = v;
            sT1[i] = dv;
        }
        __syncthreads();
        constexpr int NF2 = CURV ? 6 : 3;
        int fld2[NF2];
#pragma unroll
        for (int f = 0; f < NF2; ++f) fld2[f] = f < 3 ? f : f + 2;
        double pal = 0.0;
        for (int pt = tid; pt < NE * NE * NE; pt += blockDim.x) {
            const int qx = pt % NE, qy = (pt / NE) % NE, qz = pt / (NE * NE);
            double u[NF2], g[NF2][3];
            point_fields<N1, NE, NF2>(sT0, sT1, sB, sdB, fld2, qx, qy, qz, u, g);
            double wdet = detj;
            if constexpr (CURV) {
                const double gx[3][3] = {{g[3][0], g[3][1], g[3][2]}, {g[4][0], g[4][1], g[4][2]},
                                         {g[5][0], g[5][1], g[5][2]}};
                double I[3][3];
                wdet = inverse_jacobian(gx, I);
                to_physical<NF2>(g, 3, I);
            } else {
#pragma unroll
                for (int s = 0; s < 3; ++s)
#pragma unroll
                    for (int d = 0; d < 3; ++d) g[s][d] *= inv_h;
            }
            double gg = 0.0;
#pragma unroll
            for (int s = 0; s < 3; ++s)
#pragma unroll
                for (int d = 0; d < 3; ++d) gg += g[s][d] * g[s][d];
            pal += 0.5 * gg * sw[qx] * sw[qy] * sw[qz] * wdet;
        }
        acc[7] = pal;
    }
    // block reduction in a fixed order (warp shuffles, then warp 0)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
        for (int i = 0; i < NACC; ++i) acc[i] += __shfl_down_sync(0xffffffffu, acc[i], o);
        const double wo = __shfl_down_sync(0xffffffffu, wave, o);
        wave = wo > wave ? wo : wave;
    }
    const int warp = tid >> 5, lane = tid & 31, nw = (blockDim.x + 31) >> 5;
    if (lane == 0) {
#pragma unroll
        for (int i = 0; i < NACC; ++i) red[i][warp] = acc[i];
        red[NQ - 1][warp] = wave;
    }
    __syncthreads();
    if (tid == 0) {
        double a[NQ];
#pragma unroll
        for (int i = 0; i < NQ; ++i) a[i] = 0.0;
        for (int w = 0; w < nw; ++w) {
#pragma unroll
            for (int i = 0; i < NACC; ++i) a[i] += red[i][w];
            a[NQ - 1] = red[NQ - 1][w] > a[NQ - 1] ? red[NQ - 1][w] : a[NQ - 1];
        }
#pragma unroll
        for (int i = 0; i < NQ; ++i) partial[(size_t)NQ * cell + i] = a[i];
    }
}

// Kinetic energy, enstrophy and wave speed on affine cells (the integrals_kernel's partials without FULL).
// One thread per column of cubature points: it contracts the x-contracted fields along y once, into
// registers, and walks z. Only what the three integrals need is carried: the values of the five
// fields, the x-derivatives of rho, m_y, m_z, the y-derivatives of rho, m_x, m_z and (from the values) the
// z-derivatives of rho, m_x, m_y. Gauss points and solution nodes are symmetric about the cell's
// centre, so the column is held as even and odd halves and two mirrored points share their sums:
// 4 operations per field and point at N1 = 6 instead of 6. The factors 1 / h and the cell's volume
// are taken out of the sums; the wave speed is compared squared (one root per point).
// Bound by FP64 operations of few warps with much independent work. One call at 16^3 cells on B200, its four numbers'
// way to the host included, field-by-field contraction at every point -> this kernel: p = 1 0.163 -> 0.090 ms, p = 2
// 0.222 -> 0.125, p = 3 0.345 -> 0.208, p = 4 0.579 -> 0.272, p = 5 0.641 -> 0.350, p = 6 1.35 -> 1.06 (its column of 77
// values does not fit the 168 registers that ten warps leave: 2.2 KB a thread are spilled).
template <int N1> struct IntegralsAffine {
    static constexpr int NE = N1 + 10, NP = N1 * N1 * N1, NT2 = N1 * N1 * NE;
    static constexpr int NT = (NE * NE + 31) / 32 * 32;
    static constexpr int KE = (N1 + 1) / 2, KO = N1 / 2, QH = (NE + 1) / 2;   // even / odd halves, mirrored point pairs
    static constexpr int oT0 = 5 * NP, oT1 = oT0 + 5 * NT2, total = oT1 + 3 * NT2;
    static constexpr size_t bytes = (size_t)total * sizeof(double);
};

template <int N1>
__global__ void __launch_bounds__(IntegralsAffine<N1>::NT)
integrals_affine_kernel(const double* __restrict__ U, const IntegralTab* tab, int nc, IntegralConst ic,
                        double* __restrict__ partial) {
    using L = IntegralsAffine<N1>;
    constexpr int NE = L::NE, NP = L::NP, NT2 = L::NT2, NT = L::NT, KE = L::KE, KO = L::KO, QH = L::QH;
    __shared__ double sB[NE * N1], sdB[NE * N1], sw[NE];
    // even / odd parts of B and dB in z: [pair q][k]
    __shared__ double sE[QH * KE], sO[QH * (KO > 0 ? KO : 1)], sdE[QH * KE], sdO[QH * (KO > 0 ? KO : 1)];
    __shared__ double red[3][32];
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* sU = reinterpret_cast<double*>(smem_raw);   // [5][NP]
    double* sT0 = sU + L::oT0;                          // [s][(k*N1 + j)*NE + qx] values
    double* sT1 = sU + L::oT1;                          // x-derivatives of rho, m_y, m_z
    const int cell = blockIdx.x, tid = threadIdx.x;
    for (int i = tid; i < NE * N1; i += NT) { sB[i] = tab->B[i]; sdB[i] = tab->dB[i]; }
    for (int i = tid; i < NE; i += NT) sw[i] = tab->w[i];
    for (int i = tid; i < 5 * NP; i += NT) sU[i] = U[(size_t)cell * 5 * NP + i];
    __syncthreads();
    for (int i = tid; i < QH * KE; i += NT) {
        const int q = i / KE, k = i - q * KE, m = N1 - 1 - k;
        const double f = k == m ? 0.5 : 1.0;   // the middle node is its own mirror
        sE[i] = f * 0.5 * (sB[q * N1 + k] + sB[q * N1 + m]);
        sdE[i] = f * 0.5 * (sdB[q * N1 + k] + sdB[q * N1 + m]);
        if (k < KO) {
            sO[q * KO + k] = 0.5 * (sB[q * N1 + k] - sB[q * N1 + m]);
            sdO[q * KO + k] = 0.5 * (sdB[q * N1 + k] - sdB[q * N1 + m]);
        }
    }
    for (int i = tid; i < 5 * NT2; i += NT) {
        const int qx = i % NE, kj = (i / NE) % (N1 * N1), s = i / NT2;
        const double* u = sU + s * NP + kj * N1;
        double v = 0.0, dv = 0.0;
#pragma unroll
        for (int a = 0; a < N1; ++a) { v += sB[qx * N1 + a] * u[a]; dv += sdB[qx * N1 + a] * u[a]; }
        sT0[i] = v;
        if (s != 1 && s != 4) sT1[(s == 0 ? 0 : s - 1) * NT2 + i - s * NT2] = dv;
    }
    __syncthreads();
    const double gam = ic.gam, gm1 = ic.gm1;
    double ke = 0.0, en = 0.0, w2 = 0.0;
    if (tid < NE * NE) {
        const int qx = tid % NE, qy = tid / NE;
        // even and odd parts along z of: 0-4 the values, 5-7 d/dx of rho, m_y, m_z, 8-10 d/dy of rho, m_x, m_z
        double ev[11][KE], od[11][KO > 0 ? KO : 1];
#pragma unroll
        for (int f = 0; f < 11; ++f) {
            const double* t = f < 5 ? sT0 + f * NT2 : f < 8 ? sT1 + (f - 5) * NT2
                                                            : sT0 + (f == 8 ? 0 : f == 9 ? 1 : 3) * NT2;
            const double* c = (f < 8 ? sB : sdB) + qy * N1;
#pragma unroll
            for (int k = 0; k < KE; ++k) {
                const int m = N1 - 1 - k;
                double x = 0.0, y = 0.0;
#pragma unroll
                for (int j = 0; j < N1; ++j) {
                    x += c[j] * t[(k * N1 + j) * NE + qx];
                    if (m != k) y += c[j] * t[(m * N1 + j) * NE + qx];
                }
                if (m == k) y = x;
                ev[f][k] = x + y;
                if (k < KO) od[f][k] = x - y;
            }
        }
#pragma unroll 1
        for (int q = 0; q < QH; ++q) {
            // the pair's two points: field f (0-10 as above, 11-13 d/dz of rho, m_x, m_y) at q and at its mirror
            auto points = [&](int f, double d[2]) {
                const int r = f < 11 ? f : f - 11;
                double e = 0.0, o = 0.0;
#pragma unroll
                for (int k = 0; k < KE; ++k) e += (f < 11 ? sE : sdE)[q * KE + k] * ev[r][k];
#pragma unroll
                for (int k = 0; k < KO; ++k) o += (f < 11 ? sO : sdO)[q * KO + k] * od[r][k];
                d[0] = e + o;
                d[1] = f < 11 ? e - o : o - e;
            };
            double rho[2], v[3][2], en_[2], om[3][2], d[2];
            points(0, rho); points(1, v[0]); points(2, v[1]); points(3, v[2]); points(4, en_);
            double ir[2], vv[2];
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                ir[m] = qrcp<double>(rho[m]);
#pragma unroll
                for (int c = 0; c < 3; ++c) v[c][m] *= ir[m];
                vv[m] = v[0][m] * v[0][m] + v[1][m] * v[1][m] + v[2][m] * v[2][m];
            }
            // om: rho times the vorticity (times h), derivative by derivative
            points(5, d);    // d rho / dx
#pragma unroll
            for (int m = 0; m < 2; ++m) { om[1][m] = v[2][m] * d[m]; om[2][m] = -(v[1][m] * d[m]); }
            points(6, d);    // d m_y / dx
#pragma unroll
            for (int m = 0; m < 2; ++m) om[2][m] += d[m];
            points(7, d);    // d m_z / dx
#pragma unroll
            for (int m = 0; m < 2; ++m) om[1][m] -= d[m];
            points(8, d);    // d rho / dy
#pragma unroll
            for (int m = 0; m < 2; ++m) { om[0][m] = -(v[2][m] * d[m]); om[2][m] += v[0][m] * d[m]; }
            points(9, d);    // d m_x / dy
#pragma unroll
            for (int m = 0; m < 2; ++m) om[2][m] -= d[m];
            points(10, d);   // d m_z / dy
#pragma unroll
            for (int m = 0; m < 2; ++m) om[0][m] += d[m];
            points(11, d);   // d rho / dz
#pragma unroll
            for (int m = 0; m < 2; ++m) { om[0][m] += v[1][m] * d[m]; om[1][m] -= v[0][m] * d[m]; }
            points(12, d);   // d m_x / dz
#pragma unroll
            for (int m = 0; m < 2; ++m) om[1][m] += d[m];
            points(13, d);   // d m_y / dz
#pragma unroll
            for (int m = 0; m < 2; ++m) om[0][m] -= d[m];
            const double wz = sw[q];
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                if (m && 2 * q + 1 == NE) continue;   // (the centre is its own mirror)
                ke += wz * (rho[m] * vv[m]);
                en += wz * ((om[0][m] * om[0][m] + om[1][m] * om[1][m] + om[2][m] * om[2][m]) * ir[m]);
                const double p = gm1 * (en_[m] - 0.5 * rho[m] * vv[m]), cc = gam * p * ir[m];
                const double s2 = (vv[m] + cc) + 2.0 * sqrt(vv[m] * cc);   // (|v| + c)^2
                w2 = s2 > w2 ? s2 : w2;
            }
        }
        const double wxy = 0.5 * (sw[qx] * sw[qy]);
        ke *= wxy * (ic.h * ic.h * ic.h);
        en *= wxy * ic.h;   // h^3 / h^2
    }
    // block reduction in a fixed order (warp shuffles, then the warps in order)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        ke += __shfl_down_sync(0xffffffffu, ke, o);
        en += __shfl_down_sync(0xffffffffu, en, o);
        const double wo = __shfl_down_sync(0xffffffffu, w2, o);
        w2 = wo > w2 ? wo : w2;
    }
    if ((tid & 31) == 0) { red[0][tid >> 5] = ke; red[1][tid >> 5] = en; red[2][tid >> 5] = w2; }
    __syncthreads();
    if (tid == 0) {
        double a0 = 0.0, a1 = 0.0, a2 = 0.0;
        for (int w = 0; w < NT / 32; ++w) {
            a0 += red[0][w]; a1 += red[1][w];
            a2 = red[2][w] > a2 ? red[2][w] : a2;
        }
        partial[(size_t)3 * cell] = a0;
        partial[(size_t)3 * cell + 1] = a1;
        partial[(size_t)3 * cell + 2] = sqrt(a2);
    }
}

// One row of the integrals table on the device: the per-cell partials of integrals_kernel
// (not FULL: kinetic energy, enstrophy, max wave speed per cell) reduced to
// {KE / V, enstrophy / V, 2 enstrophy / (Re V) (re > 0; zero otherwise), max wave speed}, the
// values ph_integrals returns. One block of ROW_THREADS: each thread sums a fixed strided share of the cells in
// order, then a fixed-order tree, so a row is the same on every run. The row index comes
// from a device counter that the kernel advances, so one captured launch serves every row.
constexpr int ROW_THREADS = 512;
static __global__ void __launch_bounds__(ROW_THREADS)
integrals_row_kernel(const double* __restrict__ partial, int nc, double vol, double re, int* __restrict__ counter,
                     int max_rows, double* __restrict__ table) {
    __shared__ double ske[ROW_THREADS], sen[ROW_THREADS], swv[ROW_THREADS];
    const int tid = threadIdx.x;
    double ke = 0.0, en = 0.0, wv = 0.0;
    for (int i = tid; i < nc; i += ROW_THREADS) {
        ke += partial[3 * (size_t)i];
        en += partial[3 * (size_t)i + 1];
        const double w = partial[3 * (size_t)i + 2];
        wv = w > wv ? w : wv;
    }
    ske[tid] = ke; sen[tid] = en; swv[tid] = wv;
    __syncthreads();
    for (int h = ROW_THREADS / 2; h > 0; h >>= 1) {
        if (tid < h) {
            ske[tid] += ske[tid + h];
            sen[tid] += sen[tid + h];
            swv[tid] = swv[tid + h] > swv[tid] ? swv[tid + h] : swv[tid];
        }
        __syncthreads();
    }
    if (tid == 0) {
        const int r = *counter;
        if (r < max_rows) {
            double* row = table + 4 * (size_t)r;
            row[0] = ske[0] / vol;
            row[1] = sen[0] / vol;
            row[2] = re > 0.0 ? 2.0 * row[1] / re : 0.0;
            row[3] = swv[0];
        }
        *counter = r + 1;
    }
}

// ------------------------------------------------------------------------------------
// Rate of change of the kinetic energy, dKE/dt = integral of dKE/dU . dU/dt over the cell with
// the same QGauss(p+11) cubature as the kinetic energy itself (so its time integral is that
// KE), from a state U and its time derivative K = M^-1 R(U): the integrand is
// v . K_m - |v|^2 / 2 K_rho (rho |v|^2 / 2 with m = rho v; the energy does not enter). Affine
// cells; per-cell partial sums (W det J included), summed on the host in cell order. One CTA
// per cell; one thread per (qx, qy) column walks qz.
// ------------------------------------------------------------------------------------
template <int N1> __host__ __device__ constexpr int ke_rate_threads() {
    return (N1 + 10) * (N1 + 10) <= 256 ? 256 : 512;
}
template <int N1> __host__ __device__ constexpr size_t ke_rate_smem() {
    constexpr int NE = N1 + 10;
    return sizeof(double) * (8 * (size_t)N1 * N1 * N1 + 8 * (size_t)N1 * N1 * NE + 8 * (size_t)N1 * NE * NE);
}

template <int N1>
__global__ void __launch_bounds__(ke_rate_threads<N1>())
ke_rate_kernel(const double* __restrict__ U, const double* __restrict__ K, const IntegralTab* __restrict__ tab,
               int nc, double h3, double* __restrict__ partial) {
    constexpr int NE = N1 + 10, NP = N1 * N1 * N1, NT = ke_rate_threads<N1>();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* sF = reinterpret_cast<double*>(smem_raw);   // [8][NP]: rho, m (3) of U, then of K
    double* t0 = sF + 8 * NP;                           // [8][N1][N1][NE] after x
    double* t1 = t0 + 8 * N1 * N1 * NE;                 // [8][N1][NE][NE] after y
    __shared__ double sB[NE * N1], sw[NE], red[NT / 32];
    const int cell = blockIdx.x, tid = threadIdx.x;
    for (int i = tid; i < NE * N1; i += NT) sB[i] = tab->B[i];
    for (int i = tid; i < NE; i += NT) sw[i] = tab->w[i];
    for (int i = tid; i < 8 * NP; i += NT) {
        const int f = i / NP, node = i % NP;
        const double* src = f < 4 ? U : K;
        sF[i] = src[((size_t)cell * 5 + (f % 4)) * NP + node];
    }
    __syncthreads();
    for (int i = tid; i < 8 * N1 * N1 * NE; i += NT) {   // x: [f][z][y][qx]
        const int qx = i % NE, r = i / NE;              // r = (f * N1 + z) * N1 + y
        double v = 0.0;
        for (int a = 0; a < N1; ++a) v += sB[qx * N1 + a] * sF[r * N1 + a];
        t0[i] = v;
    }
    __syncthreads();
    for (int i = tid; i < 8 * N1 * NE * NE; i += NT) {   // y: [f][z][qy][qx]
        const int qx = i % NE, qy = (i / NE) % NE, fz = i / (NE * NE);
        double v = 0.0;
        for (int b = 0; b < N1; ++b) v += sB[qy * N1 + b] * t0[(fz * N1 + b) * NE + qx];
        t1[i] = v;
    }
    __syncthreads();
    double acc = 0.0;
    for (int col = tid; col < NE * NE; col += NT) {
        const int qx = col % NE, qy = col / NE;
        for (int qz = 0; qz < NE; ++qz) {
            double f[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                double v = 0.0;
                for (int c = 0; c < N1; ++c) v += sB[qz * N1 + c] * t1[((k * N1 + c) * NE + qy) * NE + qx];
                f[k] = v;
            }
            const double v0 = f[1] / f[0], v1 = f[2] / f[0], v2 = f[3] / f[0];
            const double rate = v0 * f[5] + v1 * f[6] + v2 * f[7] - 0.5 * (v0 * v0 + v1 * v1 + v2 * v2) * f[4];
            acc += sw[qx] * sw[qy] * sw[qz] * rate;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if ((tid & 31) == 0) red[tid >> 5] = acc;
    __syncthreads();
    if (tid == 0) {
        double t = 0.0;
        for (int w = 0; w < NT / 32; ++w) t += red[w];
        partial[cell] = t * h3;
    }
}

} // namespace ph
