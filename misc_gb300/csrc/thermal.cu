// Thermal path: heat conduction (and capacitance in transient steps) of the brick8 and shell4
// elements, assembly into the reference's thermal CSR, thermal constraints, heat generation and a
// device solve.
//
// Reference: getThermalSolnLoad (Working/AStrO_commandFunctions.f90:16-72), r_getElRt /
// r_getElRtk / r_getElRtm (Working/AStrO_r_elementEqns.f90:2062-2204), the conductivity and
// specific heat staging (Working/AStrO_r_designPropertyFunctions.f90:129-186, 527-644),
// getThermalAppliedLoad's bodyHeatGen branch (commandFunctions :78-139, through r_getElBodyForce),
// getThermalConstraintLoad / scaleThermalMPC (:197-258), buildThermalMPC
// (Working/AStrO_bookKeeping.f90:614-752) and allocateThermalMat (:413-472).
//
// GB300 mapping: one DOF per node, so the thermal matrix lives as the values of the model's
// node-block pattern with 1 x 1 blocks, in rank order (the reference numbers thermal DOF by
// currentRank too).  Element kernels run one thread per element, their updates of shared entries colour
// by colour (no atomics, fixed summation order); the property stage (per element conductivity in the element frame,
// heat capacity, shell thickness) runs once per thermal setup.  The solve is a Jacobi-
// preconditioned conjugate gradient in FP64 on K_T + C^T C with its scalars kept on the device.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <vector>

#include "astro_internal.h"
#include "krylov_resident.cuh"
#include "shell_props.cuh"

namespace {

constexpr int kProps = 11;  // per element: conductivity 3x3 row-major, heat capacity, thickness

// The matrix of the thermal solve: slot-major rows (entry s of row r at s * ld + r) and penalty rows.
struct CgMat {
    int N, S, ld;
    const double *v;
    const int *col;
    const int *pp, *pc;  // penalty rows (null: none)
    const double *pv;
};

struct ThermPlan {
    int nMat = 0;
    DevBuf d_props, d_val, d_pos, d_rowStart, d_elMatId, d_matCond, d_matSH, d_layCond, d_laySH;
    int matSize = 0, haveMat = 0;
    // constraints: rows of (internal column, coefficient), unscaled and scaled
    int mpcDim = 0;
    std::vector<int> mRange, mCol;
    std::vector<double> mVal, mRhs, sVal, sRhs;
    int scaled = 0;
    DevBuf d_mRange, d_mCol, d_sVal, d_sRhs, d_penPtr, d_penCol, d_penVal;
    int penCount = 0;
    // constraint load: the rows' defects, and per constrained node its terms in row order
    DevBuf d_mDef, d_gPtr, d_gTerm, d_gRow, d_termRow;
    int targets = 0;
    DevBuf d_scr;  // bricks: the element stage's results of a chunk
    // the solve's slot-major copy of the matrix (entry s of row r at s * ld + r)
    DevBuf d_ell, d_ellCol;
    DevBuf d_words;  // exchanged by the resident solve
    int slots = 0, ld = 0, haveCols = 0;  // haveCols: d_ellCol is filled
    // the solve's vectors and a batch of its iterations as a graph, with the pointers it was captured with
    DevBuf d_cg[8];  // x, r, z, p, Ap, 1 / diagonal, partials, scalars
    cudaGraphExec_t cgExec = nullptr;
    CgMat cgMat = {};
    std::vector<int> rowStart;  // thermMatRange(0:N)
};

ThermPlan *plan_of(astro_ctx *ctx) { return static_cast<ThermPlan *>(ctx->thermal); }

// Inputs of the per-element thermal properties: the material (solids) or layer (shells) values
// as given, and the element design-variable maps.
struct ThPropArgs {
    int shell;
    const int *esec, *elMatId;
    const double *elDen;  // solid density, the real density design terms applied
    const double *matCond, *matSH;
    const int *layRange;
    const LayerDev *lay;
    const double *layCond, *laySH;
    const int *e2dR, *e2d;  // null: no design variables
    const double *e2c;
    const int *dcat, *dlay, *dcomp;
    const double *dval;
};

// One element's thermal properties with its design-variable terms, + i h on variable `pert`
// (0 = none): the conductivity tc in the element frame, the heat capacity sh (density x specific
// heat; per area for shells, the layers summed) and the shell section thickness secT.  Solids:
// r_getMaterialThermCond / r_getMaterialSpecHeat (Working/AStrO_r_designPropertyFunctions.f90:129-186)
// and r_getMaterialDensity (:82-103); shells: r_getShellThermCond / r_getShellSpecHeat
// (:527-644), every layer's conductivity, specific heat, density, thickness and angle with its
// 'layup' terms.  Each value takes its terms one at a time in the element's term order.
template <class T>
__device__ void th_props_t(const ThPropArgs &A, int e, int pert, double h, T tc[3][3], T &sh, T &secT) {
    auto add_terms = [&](T &v, int cat, int layerNum, int comp) {
        if (!A.e2dR) return;
        for (int q = A.e2dR[e]; q < A.e2dR[e + 1]; ++q) {
            const int d = A.e2d[q] - 1;
            if (A.dcat[d] != cat || (layerNum && A.dlay[d] != layerNum) || (comp && A.dcomp[d] != comp)) continue;
            T dv = T(A.dval[d]);
            if (d + 1 == pert) dv = dv + pert_i<T>(h);
            v = v + A.e2c[q] * dv;
        }
    };
    auto fill = [](T t[3][3], const T *v) {
        t[0][0] = v[0];
        t[1][1] = v[1];
        t[2][2] = v[2];
        t[0][1] = t[1][0] = v[3];
        t[0][2] = t[2][0] = v[4];
        t[1][2] = t[2][1] = v[5];
    };
    if (!A.shell) {
        const int mat = A.elMatId[e];
        T cv[6];
        for (int k = 0; k < 6; ++k) {
            cv[k] = T(A.matCond[6 * (mat - 1) + k]);
            add_terms(cv[k], ASTRO_DCAT_THERMAL_COND, 0, k + 1);
        }
        fill(tc, cv);
        T rho = T(A.elDen[e]);
        if (pert && A.e2dR)
            for (int q = A.e2dR[e]; q < A.e2dR[e + 1]; ++q)
                if (A.e2d[q] == pert && A.dcat[pert - 1] == ASTRO_DCAT_DENSITY) rho = rho + A.e2c[q] * pert_i<T>(h);
        T spec = T(A.matSH[mat - 1]);
        add_terms(spec, ASTRO_DCAT_SPEC_HEAT, 0, 0);
        sh = rho * spec;
        secT = T(0.0);
        return;
    }
    const int sec = A.esec[e];
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) tc[i][j] = T(0.0);
    sh = T(0.0);
    secT = T(0.0);
    for (int li = A.layRange[sec - 1], ln = 1; li < A.layRange[sec]; ++li, ++ln) {
        const LayerDev L = A.lay[li];
        T t = T(L.t), ang = T(L.angle), rho = T(L.rho), spec = T(A.laySH[li]), cv[6];
        add_terms(t, ASTRO_DCAT_LAYUP_THICKNESS, ln, 0);
        add_terms(ang, ASTRO_DCAT_LAYUP_ANGLE, ln, 0);
        add_terms(rho, ASTRO_DCAT_LAYUP_DENSITY, ln, 0);
        add_terms(spec, ASTRO_DCAT_LAYUP_SPEC_HEAT, ln, 0);
        for (int k = 0; k < 6; ++k) {
            cv[k] = T(A.layCond[6 * li + k]);
            add_terms(cv[k], ASTRO_DCAT_LAYUP_THERMAL_COND, ln, k + 1);
        }
        T tl[3][3], al[3][3], pr[3][3];
        fill(tl, cv);
        for (int i = 0; i < 3; ++i)
            for (int j = 0; j < 3; ++j) al[i][j] = T(0.0);
        al[2][2] = T(1.0);
        al[0][0] = a_cos(ang);
        al[1][0] = a_sin(ang);
        al[0][1] = -al[1][0];
        al[1][1] = al[0][0];
        for (int a = 0; a < 3; ++a)
            for (int b = 0; b < 3; ++b) {
                T v = T(0.0);
                for (int k = 0; k < 3; ++k) v = v + tl[a][k] * al[b][k];
                pr[a][b] = v;
            }
        for (int a = 0; a < 3; ++a)
            for (int b = 0; b < 3; ++b) {
                T v = T(0.0);
                for (int k = 0; k < 3; ++k) v = v + al[a][k] * pr[k][b];
                tc[a][b] = tc[a][b] + t * v;
            }
        sh = sh + t * rho * spec;
        secT = secT + t;
    }
}

// per element: conductivity in the element frame, heat capacity and shell thickness (real values
// of the design variables applied)
__global__ void k_th_props(ThPropArgs A, int E, double *__restrict__ out) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= E) return;
    double tc[3][3], sh, secT;
    th_props_t<double>(A, e, 0, 0.0, tc, sh, secT);
    double *o = out + (size_t)kProps * e;
    for (int i = 0; i < 9; ++i) o[i] = tc[i / 3][i % 3];
    o[9] = sh;
    o[10] = secT;
}

// Gauss point g of the element: shape functions, their global gradient in the element frame and
// w detJ (r_getIntPtData; shells with dxds(3,3) = 1).  r3 is the Gauss abscissa (the real path's
// 1/sqrt(3) or the complex path's single-precision literal); the shape functions are real, the
// geometry T.
template <class T>
__device__ __forceinline__ void th_point_t(int shell, const T Xl[8][3], double r3, int g, double N[8], T Nx[8][3],
                                           T &wdet) {
    const int npe = shell ? 4 : 8;
    double dN[8][3];
    if (shell) {
        const double s1 = (g & 1) ? r3 : -r3, s2 = (g & 2) ? r3 : -r3;
        const double sx[4] = {-1.0, 1.0, 1.0, -1.0}, sy[4] = {-1.0, -1.0, 1.0, 1.0};
        for (int n = 0; n < 4; ++n) {
            N[n] = 0.25 * (1.0 + sx[n] * s1) * (1.0 + sy[n] * s2);
            dN[n][0] = 0.25 * sx[n] * (1.0 + sy[n] * s2);
            dN[n][1] = 0.25 * sy[n] * (1.0 + sx[n] * s1);
            dN[n][2] = 0.0;
        }
    } else {
        const double s1 = (g & 1) ? r3 : -r3, s2 = (g & 2) ? r3 : -r3, s3 = (g & 4) ? r3 : -r3;
        const double sx[8] = {-1, 1, 1, -1, -1, 1, 1, -1}, sy[8] = {-1, -1, 1, 1, -1, -1, 1, 1},
                     sz[8] = {-1, -1, -1, -1, 1, 1, 1, 1};
        for (int n = 0; n < 8; ++n) {
            const double a1 = 1.0 + sx[n] * s1, a2 = 1.0 + sy[n] * s2, a3 = 1.0 + sz[n] * s3;
            N[n] = 0.125 * a1 * a2 * a3;
            dN[n][0] = 0.125 * sx[n] * a2 * a3;
            dN[n][1] = 0.125 * sy[n] * a1 * a3;
            dN[n][2] = 0.125 * sz[n] * a1 * a2;
        }
    }
    T J[3][3];
    for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b) {
            T s = T(0.0);
            for (int n = 0; n < npe; ++n) s = s + Xl[n][a] * dN[n][b];
            J[a][b] = s;
        }
    if (shell) J[2][2] = T(1.0);
    const T c11 = J[1][1] * J[2][2] - J[1][2] * J[2][1];
    const T c12 = J[1][2] * J[2][0] - J[1][0] * J[2][2];
    const T c13 = J[1][0] * J[2][1] - J[1][1] * J[2][0];
    const T det = J[0][0] * c11 + J[0][1] * c12 + J[0][2] * c13;
    const T di = T(1.0) / det;
    T I[3][3];
    I[0][0] = di * c11;
    I[1][0] = di * c12;
    I[2][0] = di * c13;
    I[0][1] = di * (J[0][2] * J[2][1] - J[0][1] * J[2][2]);
    I[1][1] = di * (J[0][0] * J[2][2] - J[0][2] * J[2][0]);
    I[2][1] = di * (J[0][1] * J[2][0] - J[0][0] * J[2][1]);
    I[0][2] = di * (J[0][1] * J[1][2] - J[0][2] * J[1][1]);
    I[1][2] = di * (J[0][2] * J[1][0] - J[0][0] * J[1][2]);
    I[2][2] = di * (J[0][0] * J[1][1] - J[0][1] * J[1][0]);
    for (int n = 0; n < npe; ++n)
        for (int b = 0; b < 3; ++b) Nx[n][b] = dN[n][0] * I[0][b] + dN[n][1] * I[1][b] + dN[n][2] * I[2][b];
    wdet = det;  // unit weights
}

__device__ __forceinline__ void th_point(int shell, const double Xl[8][3], int g, double N[8], double Nx[8][3],
                                         double &wdet) {
    th_point_t<double>(shell, Xl, AK<double>::rt3, g, N, Nx, wdet);
}

struct ThArgs {
    const double *nodes, *orient;  // bricks: per element column-major; shells: ShellProps
    const ShellProps *sprops;
    const int *elist, *rank, *els, *elBlk;
    const double *props;
    const double *temp, *ptemp, *ptdot;
    int count, shell, dynamic, buildMat;
    double gamma, delT;
    double *load, *val;
    double *scr;  // bricks: per listed element kThScr doubles (the element stage's results)
    int q0;       // bricks, scatter: the colour's first element in the list
    int repeats;  // bricks, scatter: elements may name a node twice
};

template <int NPE>
__device__ __forceinline__ void th_frame(const ThArgs &A, int e, double Xl[8][3], int rk[8]) {
    double Or[3][3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j)
            Or[i][j] = NPE == 4 ? A.sprops[e].orient[3 * i + j] : A.orient[9 * (size_t)e + 3 * j + i];
#pragma unroll
    for (int a = 0; a < NPE; ++a) {
        const int nd = A.elist[8 * (size_t)e + a] - 1;
        rk[a] = A.rank[nd] - 1;
        const double X0 = A.nodes[3 * (size_t)nd], X1 = A.nodes[3 * (size_t)nd + 1], X2 = A.nodes[3 * (size_t)nd + 2];
#pragma unroll
        for (int i = 0; i < 3; ++i) Xl[a][i] = Or[i][0] * X0 + Or[i][1] * X1 + Or[i][2] * X2;
    }
}

// ---- bricks: sum factorisation ------------------------------------------------------------------
// On the 2 x 2 x 2 Gauss points a trilinear shape function is a product of N_s(t) = (1 + s t) / 2 with
// values p = (1 + r) / 2 (node and point on the same side) and q = (1 - r) / 2, so with
// Q = (1 / det J) adj(J) k adj(J)^T per point
//   K_ab = 1/4 ( sx sx' U1[y y'][z z'] + ... + sx sy' W12[x'][y][z z'] + sy sx' W12[x][y'][z z'] + ... )
// where U1 sums Q11 over the points against N_y N_y' N_z N_z' (a node pair enters a direction in three
// ways), W12 sums Q12 against N_x N_y and N_z N_z', and so on: 63 sums of 8 terms for the 36 entries.
// J itself comes from the 12 edge differences the same way.  About 1,800 FP64 operations an element;
// gradients and products point by point are 4,700 (GB300 issues 1.7 FP64 lanes a clock and SM, which is
// what bounds this kernel).  One thread per element of all colours at once into scratch, then the
// updates of shared entries colour by colour.  65,536 bricks: 2.03 ms in eight colour launches of 64
// CTAs, 0.25 ms and 0.06 ms of updates so.
constexpr int kThThreads = 128;
constexpr int kThScr = 44;  // 36 entries of the symmetric 8 x 8, then Rt(8)
constexpr double kThP = 0.5 * (1.0 + AK<double>::rt3), kThQ = 0.5 * (1.0 - AK<double>::rt3);
__device__ __forceinline__ constexpr int th_sx(int n) { return (n == 1 || n == 2 || n == 5 || n == 6) ? 1 : 0; }
__device__ __forceinline__ constexpr int th_sy(int n) { return (n == 2 || n == 3 || n == 6 || n == 7) ? 1 : 0; }
__device__ __forceinline__ constexpr int th_sz(int n) { return n >= 4 ? 1 : 0; }
__device__ __forceinline__ constexpr int th_node(int x, int y, int z) { return 4 * z + (y ? (x ? 2 : 3) : x); }
// N_s at the point on side t, and N_s N_s' for s + s' = pair
__device__ __forceinline__ constexpr double th_n(int s, int t) { return s == t ? kThP : kThQ; }
__device__ __forceinline__ constexpr double th_c(int pair, int t) {
    return pair == 1 ? kThP * kThQ : (pair == 2 * t ? kThP * kThP : kThQ * kThQ);
}
__device__ __forceinline__ constexpr int th_sym(int a, int b) { return a * 8 - a * (a - 1) / 2 + b - a; }  // a <= b

// The columns of J at the Gauss points: column j does not vary along direction j, so four values of
// each (point sides t1, t2 of the two other directions, in order x, y, z) in F[j][2 t2 + t1][component].
struct ThJac {
    double F[3][4][3][kThThreads];
};
__device__ void th_brick_jac(const double Xl[8][3], ThJac &S) {
    const int t = threadIdx.x;
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            double d[2][2], e[2][2];  // [side of the second direction][side of the first]
#pragma unroll
            for (int v = 0; v < 2; ++v)
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int hi = j == 0 ? th_node(1, u, v) : (j == 1 ? th_node(u, 1, v) : th_node(u, v, 1));
                    const int lo = j == 0 ? th_node(0, u, v) : (j == 1 ? th_node(u, 0, v) : th_node(u, v, 0));
                    d[v][u] = Xl[hi][c] - Xl[lo][c];
                }
#pragma unroll
            for (int v = 0; v < 2; ++v)
#pragma unroll
                for (int u = 0; u < 2; ++u) e[v][u] = 0.5 * kThP * d[v][u] + 0.5 * kThQ * d[v][1 - u];
#pragma unroll
            for (int v = 0; v < 2; ++v)
#pragma unroll
                for (int u = 0; u < 2; ++u) S.F[j][2 * v + u][c][t] = kThP * e[v][u] + kThQ * e[1 - v][u];
        }
}
// J at point (x, y, z) and its determinant with the adjugate's first row
__device__ __forceinline__ double th_brick_point(const ThJac &S, int x, int y, int z, double J[3][3], double a0[3]) {
    const int t = threadIdx.x;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        J[c][0] = S.F[0][2 * z + y][c][t];
        J[c][1] = S.F[1][2 * z + x][c][t];
        J[c][2] = S.F[2][2 * y + x][c][t];
    }
    a0[0] = J[1][1] * J[2][2] - J[1][2] * J[2][1];
    a0[1] = J[1][2] * J[2][0] - J[1][0] * J[2][2];
    a0[2] = J[1][0] * J[2][1] - J[1][1] * J[2][0];
    return J[0][0] * a0[0] + J[0][1] * a0[1] + J[0][2] * a0[2];
}
// sums of a value per point against N_x N_x' N_y N_y' N_z N_z' (pairs): V[px][py][pz]
__device__ __forceinline__ void th_brick_pairs(const double d[8], double V[3][3][3]) {
    double a[3][2][2], b[3][3][2];
#pragma unroll
    for (int p = 0; p < 3; ++p)
#pragma unroll
        for (int z = 0; z < 2; ++z)
#pragma unroll
            for (int y = 0; y < 2; ++y)
                a[p][y][z] = th_c(p, 0) * d[4 * z + 2 * y] + th_c(p, 1) * d[4 * z + 2 * y + 1];
#pragma unroll
    for (int p = 0; p < 3; ++p)
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int z = 0; z < 2; ++z) b[p][r][z] = th_c(r, 0) * a[p][0][z] + th_c(r, 1) * a[p][1][z];
#pragma unroll
    for (int p = 0; p < 3; ++p)
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int m = 0; m < 3; ++m) V[p][r][m] = th_c(m, 0) * b[p][r][0] + th_c(m, 1) * b[p][r][1];
}

// r_getElRt of one brick per thread: Rt and, with buildMat, dRt/dT into the scratch
__global__ void __launch_bounds__(kThThreads) k_th_brick(ThArgs A) {
    __shared__ ThJac S;
    const int q = blockIdx.x * kThThreads + threadIdx.x;
    if (q >= A.count) return;
    const int e = A.els[q];
    double *out = A.scr + (size_t)q * kThScr;
    int rk[8];
    {
        double Xl[8][3];
        th_frame<8>(A, e, Xl, rk);
        th_brick_jac(Xl, S);
    }
    const double *pp = A.props + (size_t)kProps * e;
    double Rt[8], T[8];
#pragma unroll
    for (int a = 0; a < 8; ++a) {
        Rt[a] = 0.0;
        T[a] = A.temp ? A.temp[rk[a]] : 0.0;
    }
    if (A.dynamic) {
        // capacitance: Rt = M Tdot, and M / (gamma dt) as the start of the matrix
        double d[8], V[3][3][3], Td[8];
#pragma unroll
        for (int g = 0; g < 8; ++g) {
            double J[3][3], a0[3];
            d[g] = pp[9] * th_brick_point(S, g & 1, g >> 1 & 1, g >> 2, J, a0);
        }
        th_brick_pairs(d, V);
#pragma unroll
        for (int a = 0; a < 8; ++a) {
            const double pT = A.ptemp ? A.ptemp[rk[a]] : 0.0, pTd = A.ptdot ? A.ptdot[rk[a]] : 0.0;
            Td[a] = (1.0 / A.gamma) * ((1.0 / A.delT) * (T[a] - pT) - 1.0 * (1.0 - A.gamma) * pTd);
        }
        const double f = 1.0 / (A.gamma * A.delT);
#pragma unroll
        for (int a = 0; a < 8; ++a)
#pragma unroll
            for (int b = a; b < 8; ++b) {
                const double m = V[th_sx(a) + th_sx(b)][th_sy(a) + th_sy(b)][th_sz(a) + th_sz(b)];
                Rt[a] += m * Td[b];
                if (b != a) Rt[b] += m * Td[a];
                if (A.buildMat) out[th_sym(a, b)] = f * m;
            }
    }
    double U1[3][3], U2[3][3], U3[3][3], W12[2][2][3], W13[2][2][3], W23[2][2][3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) U1[i][j] = U2[i][j] = U3[i][j] = 0.0;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int k = 0; k < 3; ++k) W12[i][j][k] = W13[i][j][k] = W23[i][j][k] = 0.0;
    const double k11 = pp[0], k22 = pp[4], k33 = pp[8], k12 = pp[1], k13 = pp[2], k23 = pp[5];
#pragma unroll
    for (int g = 0; g < 8; ++g) {
        const int x = g & 1, y = g >> 1 & 1, z = g >> 2;
        double J[3][3], c[3][3], a0[3];
        const double det = th_brick_point(S, x, y, z, J, a0);
        // adj(J): c[j][b] = det dxi_j/dX_b
        c[0][0] = a0[0];
        c[1][0] = a0[1];
        c[2][0] = a0[2];
        c[0][1] = J[0][2] * J[2][1] - J[0][1] * J[2][2];
        c[1][1] = J[0][0] * J[2][2] - J[0][2] * J[2][0];
        c[2][1] = J[0][1] * J[2][0] - J[0][0] * J[2][1];
        c[0][2] = J[0][1] * J[1][2] - J[0][2] * J[1][1];
        c[1][2] = J[0][2] * J[1][0] - J[0][0] * J[1][2];
        c[2][2] = J[0][0] * J[1][1] - J[0][1] * J[1][0];
        const double di = 0.25 / det;
        double Q[6];  // 11 22 33 12 13 23
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const double t0 = di * (c[j][0] * k11 + c[j][1] * k12 + c[j][2] * k13);
            const double t1 = di * (c[j][0] * k12 + c[j][1] * k22 + c[j][2] * k23);
            const double t2 = di * (c[j][0] * k13 + c[j][1] * k23 + c[j][2] * k33);
            Q[j] = t0 * c[j][0] + t1 * c[j][1] + t2 * c[j][2];
            if (j < 2) Q[3 + j] = t0 * c[j + 1][0] + t1 * c[j + 1][1] + t2 * c[j + 1][2];  // 12, 23
            if (j == 0) Q[5] = t0 * c[2][0] + t1 * c[2][1] + t2 * c[2][2];                 // 13
        }
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                U1[i][j] += Q[0] * (th_c(i, y) * th_c(j, z));
                U2[i][j] += Q[1] * (th_c(i, x) * th_c(j, z));
                U3[i][j] += Q[2] * (th_c(i, x) * th_c(j, y));
            }
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    W12[i][j][k] += Q[3] * (th_n(i, x) * th_n(j, y) * th_c(k, z));
                    W23[i][j][k] += Q[4] * (th_n(i, y) * th_n(j, z) * th_c(k, x));
                    W13[i][j][k] += Q[5] * (th_n(i, x) * th_n(j, z) * th_c(k, y));
                }
    }
#pragma unroll
    for (int a = 0; a < 8; ++a)
#pragma unroll
        for (int b = a; b < 8; ++b) {
            const int xa = th_sx(a), xb = th_sx(b), ya = th_sy(a), yb = th_sy(b), za = th_sz(a), zb = th_sz(b);
            double k = xa == xb ? U1[ya + yb][za + zb] : -U1[ya + yb][za + zb];
            k = ya == yb ? k + U2[xa + xb][za + zb] : k - U2[xa + xb][za + zb];
            k = za == zb ? k + U3[xa + xb][ya + yb] : k - U3[xa + xb][ya + yb];
            k = xa == yb ? k + W12[xb][ya][za + zb] : k - W12[xb][ya][za + zb];
            k = ya == xb ? k + W12[xa][yb][za + zb] : k - W12[xa][yb][za + zb];
            k = xa == zb ? k + W13[xb][za][ya + yb] : k - W13[xb][za][ya + yb];
            k = za == xb ? k + W13[xa][zb][ya + yb] : k - W13[xa][zb][ya + yb];
            k = ya == zb ? k + W23[yb][za][xa + xb] : k - W23[yb][za][xa + xb];
            k = za == yb ? k + W23[ya][zb][xa + xb] : k - W23[ya][zb][xa + xb];
            Rt[a] += k * T[b];
            if (b != a) Rt[b] += k * T[a];
            if (A.buildMat) out[th_sym(a, b)] = A.dynamic ? out[th_sym(a, b)] + k : k;
        }
#pragma unroll
    for (int a = 0; a < 8; ++a) out[36 + a] = Rt[a];
}

// bodyHeatGen of one brick per thread: q times the integral of N into the scratch's Rt part
__global__ void __launch_bounds__(kThThreads) k_th_brick_heat(ThArgs A, double qv) {
    __shared__ ThJac S;
    const int q = blockIdx.x * kThThreads + threadIdx.x;
    if (q >= A.count) return;
    {
        double Xl[8][3];
        int rk[8];
        th_frame<8>(A, A.els[q], Xl, rk);
        th_brick_jac(Xl, S);
    }
    double d[8];
#pragma unroll
    for (int g = 0; g < 8; ++g) {
        double J[3][3], a0[3];
        d[g] = qv * th_brick_point(S, g & 1, g >> 1 & 1, g >> 2, J, a0);
    }
    // one direction after the other: point sides become node sides
#pragma unroll
    for (int m = 1; m < 8; m *= 2)
#pragma unroll
        for (int g = 0; g < 8; ++g)
            if (!(g & m)) {
                const double lo = d[g], hi = d[g | m];
                d[g] = kThP * lo + kThQ * hi;
                d[g | m] = kThQ * lo + kThP * hi;
            }
    double *out = A.scr + (size_t)q * kThScr + 36;
#pragma unroll
    for (int a = 0; a < 8; ++a) out[a] = d[th_sx(a) + 2 * th_sy(a) + 4 * th_sz(a)];
}

// One colour's bricks from the scratch: 64 threads an element for the matrix entries (buildMat), then 8
// for the load: -Rt, or with mult + mult[element] times the heat generation.  Where an element may name a
// node twice, its entries for that node are one: a thread an element then, its entries in turn.
__global__ void k_th_brick_add(ThArgs A, const double *__restrict__ mult) {
    const int per = A.buildMat ? 72 : 8;
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    auto add = [&](int q, int i) {
        const int e = A.els[q];
        const double *scr = A.scr + (size_t)q * kThScr;
        if (i < 0) {
            const int ab = i + 64, a = ab >> 3, b = ab & 7;
            A.val[A.elBlk[64 * (size_t)e + ab]] += scr[a <= b ? th_sym(a, b) : th_sym(b, a)];
        } else if (A.load) {
            const int r = A.rank[A.elist[8 * (size_t)e + i] - 1] - 1;
            A.load[r] += mult ? mult[q] * scr[36 + i] : -scr[36 + i];
        }
    };
    if (!A.repeats) {
        if (t < (long long)per * A.count) add(A.q0 + (int)(t / per), (int)(t % per) - (per - 8));
    } else if (t < A.count) {
        for (int i = 8 - per; i < 8; ++i) add(A.q0 + (int)t, i);
    }
}

// r_getElRt of one shell per thread: thermalLoad(rank) -= Rt, K_T += dRt/dT (colour order)
__global__ void k_th_elem(ThArgs A) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= A.count) return;
    const int e = A.els[q];
    constexpr int npe = 4, ngp = 4;
    double Xl[8][3];
    int rk[8];
    th_frame<4>(A, e, Xl, rk);
    const double *pp = A.props + (size_t)kProps * e;
    double tc[3][3];
    for (int i = 0; i < 9; ++i) tc[i / 3][i % 3] = pp[i];
    double T[npe], Td[npe];
    for (int a = 0; a < npe; ++a) {
        T[a] = A.temp ? A.temp[rk[a]] : 0.0;
        if (A.dynamic) {
            const double pT = A.ptemp ? A.ptemp[rk[a]] : 0.0, pTd = A.ptdot ? A.ptdot[rk[a]] : 0.0;
            Td[a] = (1.0 / A.gamma) * ((1.0 / A.delT) * (T[a] - pT) - 1.0 * (1.0 - A.gamma) * pTd);
        }
    }
    double Rt[npe], K[npe][npe], Rm[npe], M[npe][npe];
    for (int a = 0; a < npe; ++a) {
        Rt[a] = 0.0;
        Rm[a] = 0.0;
        for (int b = 0; b < npe; ++b) K[a][b] = M[a][b] = 0.0;
    }
    for (int g = 0; g < ngp; ++g) {
        double N[8], Nx[8][3], wd;
        th_point(1, Xl, g, N, Nx, wd);
        double Tx[3] = {0.0, 0.0, 0.0}, qv[3];
        for (int a = 0; a < npe; ++a)
            for (int k = 0; k < 3; ++k) Tx[k] = Tx[k] + Nx[a][k] * T[a];
        for (int i = 0; i < 3; ++i) qv[i] = wd * (tc[i][0] * Tx[0] + tc[i][1] * Tx[1] + tc[i][2] * Tx[2]);
        for (int a = 0; a < npe; ++a) Rt[a] = Rt[a] + Nx[a][0] * qv[0] + Nx[a][1] * qv[1] + Nx[a][2] * qv[2];
        if (A.buildMat) {
            double kN[npe][3];
            for (int a = 0; a < npe; ++a)
                for (int k = 0; k < 3; ++k)
                    kN[a][k] = wd * (Nx[a][0] * tc[0][k] + Nx[a][1] * tc[1][k] + Nx[a][2] * tc[2][k]);
            for (int a = 0; a < npe; ++a)
                for (int b = 0; b < npe; ++b)
                    K[a][b] = K[a][b] + Nx[a][0] * kN[b][0] + Nx[a][1] * kN[b][1] + Nx[a][2] * kN[b][2];
        }
        if (A.dynamic) {
            const double c = wd * pp[9];
            double pt = 0.0;
            for (int a = 0; a < npe; ++a) pt = pt + Td[a] * N[a];
            pt = c * pt;
            for (int a = 0; a < npe; ++a) Rm[a] = Rm[a] + pt * N[a];
            if (A.buildMat)
                for (int a = 0; a < npe; ++a)
                    for (int b = 0; b < npe; ++b) M[a][b] = M[a][b] + N[a] * (c * N[b]);
        }
    }
    if (A.dynamic) {
        const double f = 1.0 / (A.gamma * A.delT);
        for (int a = 0; a < npe; ++a) {
            Rt[a] = Rt[a] + Rm[a];
            if (A.buildMat)
                for (int b = 0; b < npe; ++b) K[a][b] = K[a][b] + f * M[a][b];
        }
    }
    if (A.load)
        for (int a = 0; a < npe; ++a) A.load[rk[a]] -= Rt[a];
    if (A.buildMat)
        for (int a = 0; a < npe; ++a)
            for (int b = 0; b < npe; ++b) A.val[A.elBlk[(size_t)npe * npe * e + npe * a + b]] += K[a][b];
}

// bodyHeatGen of shells: q * integral of N times the section thickness, listed elements of a colour (an
// element listed twice adds twice)
__global__ void k_th_heatgen(ThArgs A, double qv, const double *__restrict__ mult) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= A.count) return;
    const int e = A.els[q];
    constexpr int npe = 4, ngp = 4;
    double Xl[8][3];
    int rk[8];
    th_frame<4>(A, e, Xl, rk);
    double w[npe] = {0.0, 0.0, 0.0, 0.0};
    for (int g = 0; g < ngp; ++g) {
        double N[8], Nx[8][3], wd;
        th_point(1, Xl, g, N, Nx, wd);
        for (int a = 0; a < npe; ++a) w[a] = w[a] + qv * N[a] * wd;
    }
    const double t = A.props[(size_t)kProps * e + 10];
    for (int a = 0; a < npe; ++a) A.load[rk[a]] += mult[q] * (t * w[a]);
}

// thermal CSR export in the reference's column order
__global__ void k_th_export(int nb, const int *__restrict__ bRow, const int *__restrict__ bCol,
                            const int *__restrict__ rowStart, const int *__restrict__ pos,
                            const double *__restrict__ val, double *__restrict__ mat, int *__restrict__ cols) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nb) return;
    const int at = rowStart[bRow[k]] + pos[k];
    mat[at] = val[k];
    cols[at] = bCol[k] + 1;
}

__global__ void k_th_absmax(const double *__restrict__ v, int n, unsigned long long *out) {
    double m = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) m = fmax(m, fabs(v[i]));
    for (int o = 16; o; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(out, (unsigned long long)__double_as_longlong(m));
}

// getThermalConstraintLoad in two steps: the defect of every row, then per constrained node the terms
// of its rows in row order (the order in which the row loop adds them)
__global__ void k_th_mpc_defect(int rows, const int *__restrict__ range, const int *__restrict__ col,
                                const double *__restrict__ val, const double *__restrict__ rhs,
                                const double *__restrict__ temp, double *__restrict__ def) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= rows) return;
    double v = rhs[r];
    for (int k = range[r]; k < range[r + 1]; ++k)
        if (col[k] >= 0) v = v - val[k] * (temp ? temp[col[k]] : 0.0);
    def[r] = v;
}

__global__ void k_th_mpc_load(int targets, const int *__restrict__ gPtr, const int *__restrict__ gTerm,
                              const int *__restrict__ gRow, const int *__restrict__ termRow,
                              const double *__restrict__ val, const double *__restrict__ def,
                              double *__restrict__ load) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= targets) return;
    double s = load[gRow[g]];
    for (int q = gPtr[g]; q < gPtr[g + 1]; ++q) s = s + val[gTerm[q]] * def[termRow[gTerm[q]]];
    load[gRow[g]] = s;
}

// ---- conjugate gradients on K_T + C^T C -------------------------------------------------------
// Three launches an iteration, Ap = A p, the step, the direction, sixteen iterations to a graph.  A dot
// product is left as CTA partials by the launch that forms it and summed, in a fixed order, by every
// CTA of the next one: a last CTA's sum at the end of each launch cost more than the launch's own work.
// The matrix is copied once per solve into slot-major rows (one thread a row: FP64, at 1.7 lanes a clock
// and SM, bounds the product, 27 multiply-adds a row, and lane-split rows would add their sums to it).
// 64x32x32 block (70,785 nodes): 65 us an iteration in ten launches (the sum of the partials alone 15 us
// on one thread), 28 us with the sums in last CTAs, 16.4 us so.  Chaining the launches by programmatic
// dependent launch made the same graph slower (31.5 us).
constexpr int kCgThreads = 256, kCgMaxCtas = 304;
constexpr int kCgBatch = 16;  // iterations between two looks at the residual (even: rz alternates)

struct CgScal {
    double rz[2];  // of even and odd iterations
    double rr, bb;
    int its, stuck;  // resident: iterations done, and whether a wait was given up
};

// sum of n CTA partials, the same in every thread (warp 0 adds)
__device__ __forceinline__ double cg_total(const double *part, int n) {
    __shared__ double total;
    if (threadIdx.x < 32) {
        double s = 0.0;
        for (int q0 = threadIdx.x; q0 < n; q0 += 320) {
            double v[10];
#pragma unroll
            for (int u = 0; u < 10; ++u) v[u] = q0 + 32 * u < n ? part[q0 + 32 * u] : 0.0;
            s += ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7])) + (v[8] + v[9]);
        }
        s = astro_kry::warp_sum(s);
        if (threadIdx.x == 0) total = s;
    }
    __syncthreads();
    return total;
}

// this CTA's sum into part[blockIdx.x]
__device__ __forceinline__ void cg_part(double v, double *part) {
    __shared__ double sm[kCgThreads / 32];
    v = astro_kry::warp_sum(v);
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) part[blockIdx.x] = ((sm[0] + sm[1]) + (sm[2] + sm[3])) + ((sm[4] + sm[5]) + (sm[6] + sm[7]));
}

// CSR values (and, once, columns) -> slot-major, padding slots: the row itself with a zero
__global__ void k_cg_ell(int N, int S, int ld, const int *__restrict__ rp, const int *__restrict__ ci,
                         const double *__restrict__ v, double *__restrict__ ev, int *__restrict__ ec) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= (long long)S * ld) return;
    const int s = (int)(t / ld), r = (int)(t - (long long)s * ld);
    const int k = r < N ? rp[r] + s : 0;
    const bool has = r < N && k < rp[r + 1];
    ev[t] = has ? v[k] : 0.0;
    if (ec) ec[t] = has ? ci[k] : (r < N ? r : 0);
}

// (A x)_r; the first kCgPre slots' entries are in c and v already
constexpr int kCgPre = 9;
__device__ __forceinline__ void cg_prefetch(const CgMat &A, int r, int c[kCgPre], double v[kCgPre]) {
#pragma unroll
    for (int u = 0; u < kCgPre; ++u) {
        c[u] = u < A.S ? __ldg(A.col + (size_t)u * A.ld + r) : r;
        v[u] = u < A.S ? __ldg(A.v + (size_t)u * A.ld + r) : 0.0;
    }
}
__device__ __forceinline__ double cg_row(const CgMat &A, int r, const double *__restrict__ x, int c[kCgPre],
                                         double v[kCgPre], double *diag) {
    double s = 0.0, d = 0.0;
    for (int q = 0;;) {
        double xv[kCgPre];
#pragma unroll
        for (int u = 0; u < kCgPre; ++u) xv[u] = x[c[u]];
#pragma unroll
        for (int u = 0; u < kCgPre; ++u) s = s + v[u] * xv[u];
        if (diag)
#pragma unroll
            for (int u = 0; u < kCgPre; ++u)
                if (c[u] == r) d = d + v[u];
        if ((q += kCgPre) >= A.S) break;
#pragma unroll
        for (int u = 0; u < kCgPre; ++u) {
            const bool has = q + u < A.S;
            c[u] = has ? __ldg(A.col + (size_t)(q + u) * A.ld + r) : r;
            v[u] = has ? __ldg(A.v + (size_t)(q + u) * A.ld + r) : 0.0;
        }
    }
    if (A.pp)
        for (int k = A.pp[r]; k < A.pp[r + 1]; ++k) {
            s = s + A.pv[k] * x[A.pc[k]];
            if (diag && A.pc[k] == r) d = d + A.pv[k];
        }
    if (diag) *diag = d;
    return s;
}

// r = b - A x, z = D^-1 r, p = z; partials of r . z and b . b
__global__ void __launch_bounds__(kCgThreads) k_cg_init(CgMat A, const double *__restrict__ b,
                                                       const double *__restrict__ x, double *__restrict__ dinv,
                                                       double *__restrict__ r, double *__restrict__ p, double *pRz,
                                                       double *pBb) {
    double rz = 0.0, bb = 0.0;
    for (int i = blockIdx.x * kCgThreads + threadIdx.x; i < A.N; i += gridDim.x * kCgThreads) {
        int c[kCgPre];
        double v[kCgPre], d;
        cg_prefetch(A, i, c, v);
        const double ax = cg_row(A, i, x, c, v, &d), di = 1.0 / d, ri = b[i] - ax, zi = di * ri;
        dinv[i] = di;
        r[i] = ri;
        p[i] = zi;
        rz += ri * zi;
        bb += b[i] * b[i];
    }
    cg_part(rz, pRz);
    __syncthreads();
    cg_part(bb, pBb);
}
__global__ void __launch_bounds__(kCgThreads) k_cg_init_sum(int n, const double *pRz, const double *pBb, CgScal *sc) {
    const double rz = cg_total(pRz, n);
    __syncthreads();
    const double bb = cg_total(pBb, n);
    if (threadIdx.x == 0) {
        sc->rz[0] = rz;
        sc->bb = bb;
    }
}

// Ap = A p; partials of p . Ap
__global__ void __launch_bounds__(kCgThreads) k_cg_ap(CgMat A, const double *__restrict__ p, double *__restrict__ Ap,
                                                     double *pPap) {
    int i = blockIdx.x * kCgThreads + threadIdx.x;
    int c[kCgPre];
    double v[kCgPre], s = 0.0;
    if (i < A.N) cg_prefetch(A, i, c, v);
    while (i < A.N) {
        const double a = cg_row(A, i, p, c, v, nullptr);
        Ap[i] = a;
        s += p[i] * a;
        i += gridDim.x * kCgThreads;
        if (i < A.N) cg_prefetch(A, i, c, v);
    }
    cg_part(s, pPap);
}

// alpha = rz / (p . Ap): x += alpha p, r -= alpha Ap, z = D^-1 r; partials of r . z and, when asked,
// r . r (read by the host after the last iteration of a batch)
__global__ void __launch_bounds__(kCgThreads) k_cg_step(int n, int par, int wantRr, const CgScal *sc, const double *pPap,
                                                       double *__restrict__ x, double *__restrict__ r,
                                                       const double *__restrict__ p, const double *__restrict__ Ap,
                                                       const double *__restrict__ dinv, double *__restrict__ z,
                                                       double *pRz, double *pRr) {
    const double alpha = sc->rz[par] / cg_total(pPap, gridDim.x);
    double rz = 0.0, rr = 0.0;
    for (int i = blockIdx.x * kCgThreads + threadIdx.x; i < n; i += gridDim.x * kCgThreads) {
        const double xi = x[i], pi = p[i], r0 = r[i], ai = Ap[i], di = dinv[i];
        x[i] = xi + alpha * pi;
        const double ri = r0 - alpha * ai, zi = di * ri;
        r[i] = ri;
        z[i] = zi;
        rz += ri * zi;
        rr += ri * ri;
    }
    cg_part(rz, pRz);
    if (wantRr) {
        __syncthreads();
        cg_part(rr, pRr);
    }
}

// beta = r . z / the last one: p = z + beta p
__global__ void __launch_bounds__(kCgThreads) k_cg_dir(int n, int par, int wantRr, CgScal *sc, const double *pRz,
                                                      const double *pRr, const double *__restrict__ z,
                                                      double *__restrict__ p) {
    const double rz = cg_total(pRz, gridDim.x);
    const double beta = rz / sc->rz[par];
    if (blockIdx.x == 0 && threadIdx.x == 0) sc->rz[par ^ 1] = rz;
    for (int i = blockIdx.x * kCgThreads + threadIdx.x; i < n; i += gridDim.x * kCgThreads) p[i] = z[i] + beta * p[i];
    if (wantRr && blockIdx.x == 0) {
        __syncthreads();
        const double rr = cg_total(pRr, gridDim.x);
        if (threadIdx.x == 0) sc->rr = rr;
    }
}

// The iterations resident on the SMs, for matrices that fit their shared memory (27 entries a row: 90,000 rows):
// one cooperative launch, a CTA per SM with consecutive rows of the matrix and of all vectors, p's halo and the
// dot products exchanged as numbered words (krylov_resident.cuh).  The same iteration, three launches of which
// are 16.4 us on 70,785 nodes; here 13 us: the FP64 pipe (34 multiply-adds a row: 4.9 us) and two sums over
// all CTAs, each of which waits for the other.
struct CgRes {
    astro_kry::Op<double> op;
    double *x, *r, *p;
    const double *dinv;
    CgScal *sc;
    ulonglong2 *words;  // all 0 at launch: cg_words()
    double target;      // on |r|, looked at every kCgBatch iterations and after the last
    int iters, N, R, G, H, P;
    int polls;          // limit of a wait
};
constexpr int kCgResIters = 1024;  // iterations of a launch
struct CgResLayout {
    size_t v, col, list, halo, own, pptr, pinfo, pval, total;
};
__host__ __device__ inline CgResLayout cg_res_layout(int N, int S, int R, int H, int P) {
    const size_t rows = ((size_t)R + 3) / 4 * 4;
    CgResLayout L;
    size_t o = 0;
    auto put = [&](size_t bytes) {
        const size_t at = o;
        o += (bytes + 15) / 16 * 16;
        return at;
    };
    const size_t v = sizeof(double) * S * rows, marks = ((size_t)N + 3) / 4 * 4;
    L.v = put(v > marks ? v : marks);
    L.col = put(sizeof(unsigned short) * S * rows);
    L.list = put(sizeof(int) * (size_t)H);
    L.halo = put(sizeof(double) * (size_t)H);
    L.own = put(sizeof(double) * 8 * rows);  // p, r, x, D^-1, A p (then z), three of partial products (then products)
    L.pptr = put(P ? sizeof(int) * ((size_t)R + 1) : 0);
    L.pinfo = put(sizeof(int) * (size_t)P);
    L.pval = put(sizeof(double) * (size_t)P);
    L.total = o;
    return L;
}
// two exchanges of a vector, partials and every CTA's totals of three sums
static size_t cg_words(int N, int G) { return 2 * (size_t)N + 6 * (size_t)G; }

__global__ void __launch_bounds__(astro_kry::kResT, 1) k_cg_resident(CgRes A) {
    using namespace astro_kry;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ double red[8], sTot[3], sRz, sCoef;
    __shared__ int sStuck;
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
    const int row0 = blockIdx.x * A.R, rows = max(0, min(A.R, A.N - row0)), Rp = (A.R + 3) / 4 * 4, S = A.op.S;
    const CgResLayout L = cg_res_layout(A.N, S, A.R, A.H, A.P);
    double *sv = reinterpret_cast<double *>(smem + L.v);
    unsigned short *sCol = reinterpret_cast<unsigned short *>(smem + L.col);
    int *sList = reinterpret_cast<int *>(smem + L.list);
    double *sHalo = reinterpret_cast<double *>(smem + L.halo);
    double *sp = reinterpret_cast<double *>(smem + L.own), *sr = sp + Rp, *sx = sr + Rp, *sd = sx + Rp, *sq = sd + Rp,
           *sPart = sq + Rp;
    int *pPtr = reinterpret_cast<int *>(smem + L.pptr), *pLoc = reinterpret_cast<int *>(smem + L.pinfo);
    double *pVal = reinterpret_cast<double *>(smem + L.pval);
    const bool pen = A.op.penPtr && A.P > 0 && rows > 0;
    const int pen0 = pen ? A.op.penPtr[row0] : 0, nPen = pen ? A.op.penPtr[row0 + rows] - pen0 : 0;
    const int halo = res_list(A.op, row0, rows, A.H, reinterpret_cast<unsigned *>(smem + L.v), sList);
    if (halo > A.H || nPen > A.P) {  // (the host sizes both by the same counts)
        if (t == 0) A.sc->stuck = 1;
        return;
    }
    for (int i = t; i < S * Rp; i += kResT) {
        const int r = i % Rp;
        sCol[i] = r < rows ? (unsigned short)res_find(sList, halo, A.op.col[(size_t)(i / Rp) * A.op.ld + row0 + r]) : 0;
    }
    if (pen) {
        for (int i = t; i <= rows; i += kResT) pPtr[i] = A.op.penPtr[row0 + i] - pen0;
        for (int q = t; q < nPen; q += kResT) {
            pLoc[q] = res_find(sList, halo, A.op.penCol[pen0 + q]);
            pVal[q] = A.op.penVal[pen0 + q];
        }
    }
    __syncthreads();  // (the marks are read)
    for (int i = t; i < S * Rp; i += kResT) {
        const int r = i % Rp;
        sv[i] = r < rows ? __ldg(A.op.K + (size_t)(i / Rp) * A.op.ld + row0 + r) : 0.0;
    }
    ulonglong2 *const part = A.words + 2 * (size_t)A.N, *const total = part + 3 * (size_t)A.G;
    unsigned no = 1;  // exchanges of p
    for (int i = t; i < rows; i += kResT) {
        sp[i] = A.p[row0 + i];
        sr[i] = A.r[row0 + i];
        sx[i] = A.x[row0 + i];
        sd[i] = A.dinv[row0 + i];
        word_put(A.words + (size_t)(no & 1) * A.N + row0 + i, sp[i], no);
    }
    if (t == 0) {
        sRz = A.sc->rz[0];
        sStuck = 0;
    }
    __syncthreads();
    // a word of number e, polled
    auto until = [&](ulonglong2 w, const ulonglong2 *p, unsigned e) {  // (w: the word's first load)
        for (int it = 0; word_no(w) != e; w = word_get(p))
            if (++it > A.polls) {
                sStuck = 1;
                break;
            }
        return __longlong_as_double((long long)w.x);
    };
    auto poll = [&](const ulonglong2 *p, unsigned e) { return until(word_get(p), p, e); };
    // sums k0 .. k0 + n - 1 over all CTAs of the rows' values at v, v + Rp, numbered e, to sTot: four warps add a
    // CTA's, CTA k mod G adds sum k over the CTAs and hands it to all
    auto sums = [&](const double *v, int k0, int n, unsigned e) {
        __syncthreads();
        if (wid < 4 * n) {
            double a = 0.0;
            for (int i = 32 * (wid & 3) + lane; i < rows; i += 128) a += v[(wid >> 2) * Rp + i];
            a = warp_sum(a);
            if (lane == 0) red[wid] = a;
        }
        __syncthreads();
        if (t < n) word_put(part + (size_t)(k0 + t) * A.G + blockIdx.x, (red[4 * t] + red[4 * t + 1]) + (red[4 * t + 2] + red[4 * t + 3]), e);
        const int mine = kResT / 32 - 1 - wid;  // sum that the warp adds up, if this CTA does
        if (mine < n && (k0 + mine) % A.G == (int)blockIdx.x) {
            constexpr int CN = kResMaxCtas / 32;  // all loads in flight
            const ulonglong2 *p = part + (size_t)(k0 + mine) * A.G;
            ulonglong2 w[CN];
#pragma unroll
            for (int u = 0; u < CN; ++u)
                if (lane + 32 * u < A.G) w[u] = word_get(p + lane + 32 * u);
            double a = 0.0;
#pragma unroll
            for (int u = 0; u < CN; ++u)
                if (lane + 32 * u < A.G) a += until(w[u], p + lane + 32 * u, e);
            a = warp_sum(a);
            for (int q = lane; q < A.G; q += 32) word_put(total + 3 * (size_t)q + k0 + mine, a, e);
        }
        if (t < n) sTot[k0 + t] = poll(total + 3 * (size_t)blockIdx.x + k0 + t, e);
    };
    const int W = (Rp + 31) / 32 * 32, SG = 4 * W <= kResT ? 4 : (2 * W <= kResT ? 2 : 1), per = kResT / SG / 32 * 32;
    const int grp = t / per, tt = t % per;
    int it = 0;
    double rr = 0.0;
    for (bool done = false; it < A.iters && !done; ++it) {
        // A p
        const ulonglong2 *vec = A.words + (size_t)(no & 1) * A.N;
        for (int i0 = t; i0 < halo; i0 += 4 * kResT) {  // four words in flight
            ulonglong2 w[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (i0 + u * kResT < halo) w[u] = word_get(vec + sList[i0 + u * kResT]);
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (i0 + u * kResT < halo) sHalo[i0 + u * kResT] = until(w[u], vec + sList[i0 + u * kResT], no);
        }
        __syncthreads();
        if (sStuck) break;
        for (int i0 = 0; i0 < Rp; i0 += per) {
            const int i = i0 + tt;
            const bool in = i < rows && grp < SG;
            double a = 0.0;
            if (in) {
#pragma unroll 4
                for (int s = grp; s < S; s += SG) a = fma(sv[s * Rp + i], sHalo[sCol[s * Rp + i]], a);
                if (grp == 0 && pen)
                    for (int q = pPtr[i]; q < pPtr[i + 1]; ++q) a += pVal[q] * sHalo[pLoc[q]];
                if (grp) sPart[(grp - 1) * Rp + i] = a;
            }
            __syncthreads();
            if (in && grp == 0) {
                for (int g = 1; g < SG; ++g) a += sPart[(g - 1) * Rp + i];
                sq[i] = a;
                sPart[i] = sp[i] * a;  // (the entry's own partial product is read)
            }
            __syncthreads();
        }
        sums(sPart, 0, 1, 2 * no);
        if (t == 0) sCoef = sRz / sTot[0];
        __syncthreads();
        if (sStuck) break;
        const double alpha = sCoef;
        for (int i = t; i < rows; i += kResT) {
            sx[i] = sx[i] + alpha * sp[i];
            const double ri = sr[i] - alpha * sq[i], zi = sd[i] * ri;
            sr[i] = ri;
            sq[i] = zi;
            sPart[i] = ri * zi;
            sPart[Rp + i] = ri * ri;
        }
        sums(sPart, 1, 2, 2 * no + 1);
        if (t == 0) {
            sCoef = sTot[1] / sRz;
            sRz = sTot[1];
        }
        __syncthreads();
        if (sStuck) break;
        const double beta = sCoef;
        rr = sTot[2];
        ++no;
        for (int i = t; i < rows; i += kResT) {
            const double pi = sq[i] + beta * sp[i];
            sp[i] = pi;
            word_put(A.words + (size_t)(no & 1) * A.N + row0 + i, pi, no);
        }
        if ((it + 1) % kCgBatch == 0) done = !isfinite(rr) || sqrt(rr) <= A.target;
    }
    for (int i = t; i < rows; i += kResT) {
        A.x[row0 + i] = sx[i];
        A.r[row0 + i] = sr[i];
        A.p[row0 + i] = sp[i];
    }
    if (t == 0 && sStuck) A.sc->stuck = 1;
    if (t == 0 && blockIdx.x == 0) {
        A.sc->rz[0] = sRz;
        A.sc->rr = rr;
        A.sc->its = it;
    }
}

}  // namespace

// Rows, halo and shared memory of the resident iterations; R = 0 when a CTA's part does not fit.
static int cg_resident_plan(astro_ctx *ctx, ThermPlan *T, CgRes *A, size_t *smem) {
    const int N = A->N;
    int coop = 0, maxSm = 0, sms = 0, per = 0, rc;
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, ctx->device);
    cudaDeviceGetAttribute(&maxSm, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
    sms = std::max(1, std::min(sms, astro_kry::kResMaxCtas));
    // (a CTA per SM, but 16 rows at least: every CTA is one more term of the sums)
    const int R = std::max((N + sms - 1) / sms, 16), G = (N + R - 1) / R;
    A->R = 0;
    cudaFuncAttributes fa;
    CK(cudaFuncGetAttributes(&fa, k_cg_resident));
    const size_t room = (size_t)maxSm - fa.sharedSizeBytes;
    if (!ctx->resident || !coop || cg_res_layout(N, A->op.S, R, R, 0).total > room) return ASTRO_OK;
    int HP[2] = {0, 0};
    int *d_HP = &A->sc->its;  // counted in the iterations' place
    CK(cudaMemsetAsync(d_HP, 0, sizeof(HP), ctx->stream));
    CK(cudaFuncSetAttribute(astro_kry::k_res_halo<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)room));
    astro_kry::k_res_halo<double><<<G, astro_kry::kThreads, (size_t)(N + 3) / 4 * 4, ctx->stream>>>(A->op, R, d_HP);
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(HP, d_HP, sizeof(HP), cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    CK(cudaMemsetAsync(d_HP, 0, sizeof(HP), ctx->stream));
    *smem = cg_res_layout(N, A->op.S, R, HP[0], HP[1]).total;
    if (HP[0] > 65535 || *smem > room) return ASTRO_OK;
    CK(cudaFuncSetAttribute(k_cg_resident, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)room));
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_cg_resident, astro_kry::kResT, *smem) != cudaSuccess || per < 1) {
        cudaGetLastError();
        return ASTRO_OK;
    }
    if (!T->d_words.p && (rc = dev_alloc(ctx, T->d_words, sizeof(ulonglong2) * cg_words(N, G))))
        return rc == ASTRO_ERR_NOMEM ? ASTRO_OK : rc;
    A->words = dptr<ulonglong2>(T->d_words);
    A->R = R;
    A->G = G;
    A->H = HP[0];
    A->P = HP[1];
    A->polls = ctx->pollLimit ? ctx->pollLimit : astro_kry::kSpinLimit;
    return ASTRO_OK;
}

void thermal_release(astro_ctx *ctx) {
    ThermPlan *T = plan_of(ctx);
    if (!T) return;
    DevBuf *b[] = {&T->d_props,   &T->d_val,    &T->d_pos,    &T->d_rowStart, &T->d_elMatId, &T->d_matCond,
                   &T->d_matSH,   &T->d_layCond, &T->d_laySH, &T->d_mRange,   &T->d_mCol,    &T->d_sVal,
                   &T->d_sRhs,    &T->d_penPtr, &T->d_penCol, &T->d_penVal,   &T->d_mDef,    &T->d_gPtr,
                   &T->d_gTerm,   &T->d_gRow,   &T->d_termRow, &T->d_ell,     &T->d_ellCol, &T->d_scr,
                   &T->d_words};
    for (DevBuf *x : b) dev_free(*x);
    for (DevBuf &x : T->d_cg) dev_free(x);
    if (T->cgExec) cudaGraphExecDestroy(T->cgExec);
    delete T;
    ctx->thermal = nullptr;
}

static ThPropArgs th_prop_args(astro_ctx *ctx, ThermPlan *T) {
    ThPropArgs A = {};
    const bool dv = ctx->numDvars > 0 && ctx->d_e2dR.p;
    A.shell = ctx->hasShell;
    A.esec = dptr<int>(ctx->d_esec);
    A.elMatId = ctx->hasSolid ? dptr<int>(T->d_elMatId) : nullptr;
    A.elDen = ctx->hasSolid ? dptr<double>(ctx->d_elRho) : nullptr;
    A.matCond = dptr<double>(T->d_matCond);
    A.matSH = dptr<double>(T->d_matSH);
    A.layRange = ctx->hasShell ? dptr<int>(ctx->d_shLayRange) : nullptr;
    A.lay = ctx->hasShell ? dptr<LayerDev>(ctx->d_shLay) : nullptr;
    A.layCond = dptr<double>(T->d_layCond);
    A.laySH = dptr<double>(T->d_laySH);
    A.e2dR = dv ? dptr<int>(ctx->d_e2dR) : nullptr;
    A.e2d = dv ? dptr<int>(ctx->d_e2d) : nullptr;
    A.e2c = dv ? dptr<double>(ctx->d_e2c) : nullptr;
    A.dcat = dv ? dptr<int>(ctx->d_dCat) : nullptr;
    A.dlay = dv ? dptr<int>(ctx->d_dLayer) : nullptr;
    A.dcomp = dv ? dptr<int>(ctx->d_dComp) : nullptr;
    A.dval = dv ? dptr<double>(ctx->d_dVal) : nullptr;
    return A;
}

extern "C" int astro_thermal_setup(astro_ctx *ctx, const astro_thermal_props *p, int32_t *therm_mat_size,
                                   int32_t *therm_mpc_dim) {
    if (!ctx || !p || p->num_materials < 1 || !p->material_therm_cond || !p->material_spec_heat) return ASTRO_ERR_ARG;
    if (ctx->hasShell && ctx->hasSolid) return set_err(ctx, ASTRO_ERR_UNSUPPORTED, "thermal path on a mixed mesh");
    const AstroPrep &P = ctx->P;
    const int N = P.N, E = P.E;
    if (ctx->hasSolid)
        for (int e = 0; e < E; ++e)
            if (ctx->elMatId[e] > p->num_materials) return set_err(ctx, ASTRO_ERR_ARG, "thermal: material out of range");
    for (int m : ctx->layMat)
        if (m < 1 || m > p->num_materials) return set_err(ctx, ASTRO_ERR_ARG, "thermal: layer material out of range");
    // constraint rows (buildThermalMPC on expanded equations: duplicate columns in a row skipped)
    std::vector<int> mRange(1, 0), mCol;
    std::vector<double> mVal, mRhs;
    for (int r = 0; r < p->num_mpc; ++r) {
        const int t0 = p->mpc_range[r], t1 = p->mpc_range[r + 1];
        const int base = (int)mCol.size();
        for (int t = t0; t < t1; ++t) {
            const int nd = p->mpc_node[t];
            if (nd < 1 || nd > N) return set_err(ctx, ASTRO_ERR_ARG, "thermal: constraint node out of range");
            mCol.push_back(-1);
            mVal.push_back(0.0);
        }
        for (int t = t0; t < t1; ++t) {
            const int col = P.currentRank[p->mpc_node[t]] - 1;
            for (int s = base; s < base + (t1 - t0); ++s) {
                if (mCol[s] < 0) {
                    mCol[s] = col;
                    mVal[s] = p->mpc_coef[t];
                    break;
                }
                if (mCol[s] == col) break;
            }
        }
        mRange.push_back((int)mCol.size());
        mRhs.push_back(p->mpc_rhs[r]);
    }
    thermal_release(ctx);
    ThermPlan *T = new ThermPlan();
    ctx->thermal = T;
    T->nMat = p->num_materials;
    T->mpcDim = p->num_mpc;
    T->mRange = mRange;
    T->mCol = mCol;
    T->mVal = mVal;
    T->mRhs = mRhs;
    // thermMatRange and the reference's column order: first insertion in the element loop
    std::vector<int> pos(P.nb, -1), fillRow(N, 0);
    T->rowStart.assign(N + 1, 0);
    for (int r = 0; r < N; ++r) T->rowStart[r + 1] = T->rowStart[r] + (P.bRowPtr[r + 1] - P.bRowPtr[r]);
    std::vector<int> rowOf(P.nb);
    for (int r = 0; r < N; ++r)
        for (int k = P.bRowPtr[r]; k < P.bRowPtr[r + 1]; ++k) rowOf[k] = r;
    const int npe = P.npe;
    for (int e = 0; e < E; ++e)
        for (int a = 0; a < npe; ++a)
            for (int b = 0; b < npe; ++b) {
                const int k = P.elBlk[(size_t)npe * npe * e + npe * a + b];
                if (pos[k] < 0) pos[k] = fillRow[rowOf[k]]++;
            }
    T->matSize = T->rowStart[N];
    int rc;
    std::vector<double> layCond(6 * std::max<size_t>(ctx->layMat.size(), 1)), laySH(std::max<size_t>(ctx->layMat.size(), 1));
    for (size_t l = 0; l < ctx->layMat.size(); ++l) {
        for (int k = 0; k < 6; ++k) layCond[6 * l + k] = p->material_therm_cond[6 * (ctx->layMat[l] - 1) + k];
        laySH[l] = p->material_spec_heat[ctx->layMat[l] - 1];
    }
    std::vector<int> rowStartI(T->rowStart.begin(), T->rowStart.end());
    if ((rc = upload(ctx, T->d_pos, pos.data(), sizeof(int) * P.nb)) ||
        (rc = upload(ctx, T->d_rowStart, rowStartI.data(), sizeof(int) * (N + 1))) ||
        (rc = upload(ctx, T->d_matCond, p->material_therm_cond, sizeof(double) * 6 * p->num_materials)) ||
        (rc = upload(ctx, T->d_matSH, p->material_spec_heat, sizeof(double) * p->num_materials)) ||
        (rc = upload(ctx, T->d_layCond, layCond.data(), sizeof(double) * layCond.size())) ||
        (rc = upload(ctx, T->d_laySH, laySH.data(), sizeof(double) * laySH.size())) ||
        (rc = dev_alloc(ctx, T->d_props, sizeof(double) * kProps * (size_t)E)) ||
        (rc = dev_alloc(ctx, T->d_val, sizeof(double) * (size_t)P.nb)))
        return rc;
    if (ctx->hasSolid && (rc = upload(ctx, T->d_elMatId, ctx->elMatId.data(), sizeof(int) * E))) return rc;
    k_th_props<<<(E + 127) / 128, 128, 0, ctx->stream>>>(th_prop_args(ctx, T), E, dptr<double>(T->d_props));
    rc = cuda_check(ctx, cudaGetLastError(), "thermal properties");
    if (!rc) rc = cuda_check(ctx, cudaStreamSynchronize(ctx->stream), "thermal properties");
    if (rc) return rc;
    if (therm_mat_size) *therm_mat_size = T->matSize;
    if (therm_mpc_dim) *therm_mpc_dim = T->mpcDim;
    return ASTRO_OK;
}

static ThArgs th_args(astro_ctx *ctx, ThermPlan *T) {
    ThArgs A = {};
    A.nodes = dptr<double>(ctx->d_nodes);
    A.orient = ctx->hasSolid ? dptr<double>(ctx->d_secOrient) : nullptr;
    A.sprops = ctx->hasShell ? dptr<ShellProps>(ctx->d_secABD) : nullptr;
    A.elist = dptr<int>(ctx->d_elist);
    A.rank = dptr<int>(ctx->d_rank);
    A.elBlk = dptr<int>(ctx->d_elBlk);
    A.props = dptr<double>(T->d_props);
    A.shell = ctx->hasShell;
    A.repeats = ctx->repeats;
    return A;
}

// host vector (rank order) -> device, or null
static int up_opt(astro_ctx *ctx, DevBuf &b, const double *h, int n) {
    if (!h) return ASTRO_OK;
    return upload(ctx, b, h, sizeof(double) * n);
}

// The bricks of a colour-grouped list (device els, colour c covering ptr[c] .. ptr[c+1]): the element
// stage for a chunk of up to 256 k elements of any colours (90 MB of scratch), then the updates colour
// by colour in the order of the list.
constexpr int kThChunk = 1 << 18, kChunkMin = 256;

template <class F>
static int th_bricks(astro_ctx *ctx, ThermPlan *T, ThArgs A, const int *els, const std::vector<int> &ptr,
                     const double *mult, F stage) {
    const int total = ptr.back();
    int cap = std::min(kThChunk, total);
    if (!total) return ASTRO_OK;
    while (T->d_scr.bytes < sizeof(double) * kThScr * (size_t)cap) {
        const int rc = dev_alloc(ctx, T->d_scr, sizeof(double) * kThScr * (size_t)cap);
        if (rc && (rc != ASTRO_ERR_NOMEM || cap <= kChunkMin)) return rc;
        if (rc) cap = (cap + 1) / 2;  // smaller chunks give the same
    }
    A.scr = dptr<double>(T->d_scr);
    for (int c0 = 0; c0 < total; c0 += cap) {
        const int c1 = std::min(total, c0 + cap);
        A.els = els + c0;
        A.count = c1 - c0;
        stage(A, (unsigned)((A.count + kThThreads - 1) / kThThreads));
        for (size_t c = 0; c + 1 < ptr.size(); ++c) {
            const int b0 = std::max(ptr[c], c0), b1 = std::min(ptr[c + 1], c1);
            if (b0 >= b1) continue;
            A.q0 = b0 - c0;
            A.count = b1 - b0;
            const long long n = (long long)(A.buildMat ? 72 : 8) * A.count;
            k_th_brick_add<<<(unsigned)((n + 255) / 256), 256, 0, ctx->stream>>>(A, mult ? mult + c0 : nullptr);
        }
    }
    return cuda_check(ctx, cudaGetLastError(), "thermal bricks");
}

extern "C" int astro_thermal_soln_load(astro_ctx *ctx, int32_t build_mat, const astro_thermal_state *st,
                                       double *thermal_load, double *therm_mat, int32_t *therm_cols) {
    if (!ctx || !thermal_load) return ASTRO_ERR_ARG;
    ThermPlan *T = plan_of(ctx);
    if (!T) return set_err(ctx, ASTRO_ERR_STATE, "thermal: astro_thermal_setup not called");
    if (st && st->dynamic && !(st->nm_gamma != 0.0 && st->del_t != 0.0))
        return set_err(ctx, ASTRO_ERR_ARG, "thermal: dynamic step needs gamma and a time step");
    const AstroPrep &P = ctx->P;
    const int N = P.N;
    cudaStream_t s = ctx->stream;
    DevBuf dT, dpT, dpTd, dL;
    int rc;
    if ((rc = up_opt(ctx, dT, st ? st->node_temp : nullptr, N)) ||
        (rc = up_opt(ctx, dpT, st ? st->prev_temp : nullptr, N)) ||
        (rc = up_opt(ctx, dpTd, st ? st->prev_tdot : nullptr, N)) ||
        (rc = upload(ctx, dL, thermal_load, sizeof(double) * N))) {
        DevBuf *v[] = {&dT, &dpT, &dpTd, &dL};
        for (DevBuf *x : v) dev_free(*x);
        return rc;
    }
    ThArgs A = th_args(ctx, T);
    A.temp = dT.p ? dptr<double>(dT) : nullptr;
    A.ptemp = dpT.p ? dptr<double>(dpT) : nullptr;
    A.ptdot = dpTd.p ? dptr<double>(dpTd) : nullptr;
    A.dynamic = st ? st->dynamic : 0;
    A.gamma = st ? st->nm_gamma : 0.5;
    A.delT = st ? st->del_t : 0.0;
    A.buildMat = build_mat == 1;
    A.load = dptr<double>(dL);
    A.val = dptr<double>(T->d_val);
    if (A.buildMat) cudaMemsetAsync(T->d_val.p, 0, sizeof(double) * P.nb, s);
    if (A.shell) {
        for (int col = 0; col < P.ncolors; ++col) {
            A.els = dptr<int>(ctx->d_colorEls) + P.colorPtr[col];
            A.count = P.colorPtr[col + 1] - P.colorPtr[col];
            if (A.count) k_th_elem<<<(A.count + 127) / 128, 128, 0, s>>>(A);
        }
        rc = ASTRO_OK;
    } else {
        rc = th_bricks(ctx, T, A, dptr<int>(ctx->d_colorEls), P.colorPtr, nullptr,
                       [&](const ThArgs &B, unsigned g) { k_th_brick<<<g, kThThreads, 0, s>>>(B); });
    }
    if (!rc) rc = cuda_check(ctx, cudaGetLastError(), "thermal elements");
    if (!rc && A.buildMat) {
        T->haveMat = 1;
        T->scaled = 0;
        if (therm_mat && therm_cols) {
            DevBuf dm, dc;
            if (!(rc = dev_alloc(ctx, dm, sizeof(double) * T->matSize)) &&
                !(rc = dev_alloc(ctx, dc, sizeof(int) * T->matSize))) {
                k_th_export<<<(P.nb + 255) / 256, 256, 0, s>>>(P.nb, dptr<int>(ctx->d_bRow), dptr<int>(ctx->d_bCol),
                                                               dptr<int>(T->d_rowStart), dptr<int>(T->d_pos),
                                                               dptr<double>(T->d_val), dptr<double>(dm), dptr<int>(dc));
                cudaError_t e = cudaMemcpyAsync(therm_mat, dm.p, sizeof(double) * T->matSize, cudaMemcpyDeviceToHost, s);
                if (e == cudaSuccess)
                    e = cudaMemcpyAsync(therm_cols, dc.p, sizeof(int) * T->matSize, cudaMemcpyDeviceToHost, s);
                if (e == cudaSuccess) e = cudaStreamSynchronize(s);
                rc = cuda_check(ctx, e, "thermal export");
            }
            dev_free(dm);
            dev_free(dc);
        }
    }
    if (!rc) {
        cudaError_t e = cudaMemcpyAsync(thermal_load, dL.p, sizeof(double) * N, cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        rc = cuda_check(ctx, e, "thermal load");
    }
    DevBuf *v[] = {&dT, &dpT, &dpTd, &dL};
    for (DevBuf *x : v) dev_free(*x);
    return rc;
}

extern "C" int astro_thermal_scale_mpc(astro_ctx *ctx, double *mpc_mat, double *mpc_rhs) {
    if (!ctx) return ASTRO_ERR_ARG;
    ThermPlan *T = plan_of(ctx);
    if (!T || !T->haveMat) return set_err(ctx, ASTRO_ERR_STATE, "thermal: conductivity matrix not assembled");
    const AstroPrep &P = ctx->P;
    cudaStream_t s = ctx->stream;
    DevBuf d;
    int rc = dev_alloc(ctx, d, sizeof(unsigned long long));
    if (rc) return rc;
    unsigned long long h = 0;
    cudaMemsetAsync(d.p, 0, sizeof(unsigned long long), s);
    k_th_absmax<<<4 * 152, 256, 0, s>>>(dptr<double>(T->d_val), P.nb, dptr<unsigned long long>(d));
    cudaError_t e = cudaMemcpyAsync(&h, d.p, sizeof(h), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    dev_free(d);
    if ((rc = cuda_check(ctx, e, "thermal scale"))) return rc;
    double maxMat;
    long long bits = (long long)h;
    std::memcpy(&maxMat, &bits, sizeof(maxMat));
    // scaleThermalMPC: each row to unit length, then times 100 max|thermMat|
    T->sVal = T->mVal;
    T->sRhs = T->mRhs;
    for (int r = 0; r < T->mpcDim; ++r) {
        double mag = 0.0;
        for (int k = T->mRange[r]; k < T->mRange[r + 1]; ++k) mag = mag + T->sVal[k] * T->sVal[k];
        mag = std::sqrt(mag);
        for (int k = T->mRange[r]; k < T->mRange[r + 1]; ++k) T->sVal[k] = (1.0 / mag) * T->sVal[k];
        T->sRhs[r] = (1.0 / mag) * T->sRhs[r];
    }
    for (double &v : T->sVal) v = 100.0 * maxMat * v;
    for (double &v : T->sRhs) v = 100.0 * maxMat * v;
    // penalty C^T C by row
    std::map<std::pair<int, int>, double> pen;
    for (int r = 0; r < T->mpcDim; ++r)
        for (int a = T->mRange[r]; a < T->mRange[r + 1]; ++a)
            for (int b = T->mRange[r]; b < T->mRange[r + 1]; ++b)
                if (T->mCol[a] >= 0 && T->mCol[b] >= 0) pen[{T->mCol[a], T->mCol[b]}] += T->sVal[a] * T->sVal[b];
    std::vector<int> pp(P.N + 1, 0), pc;
    std::vector<double> pv;
    for (auto &kv : pen) pp[kv.first.first + 1]++;
    for (int r = 0; r < P.N; ++r) pp[r + 1] += pp[r];
    for (auto &kv : pen) {
        pc.push_back(kv.first.second);
        pv.push_back(kv.second);
    }
    T->penCount = (int)pc.size();
    std::vector<int> mr(T->mRange), mc(T->mCol);
    if (mc.empty()) mc.push_back(-1);
    std::vector<double> sv(T->sVal), sr(T->sRhs);
    if (sv.empty()) sv.push_back(0.0);
    if (sr.empty()) sr.push_back(0.0);
    if (pc.empty()) {
        pc.push_back(0);
        pv.push_back(0.0);
    }
    if ((rc = upload(ctx, T->d_mRange, mr.data(), sizeof(int) * mr.size())) ||
        (rc = upload(ctx, T->d_mCol, mc.data(), sizeof(int) * mc.size())) ||
        (rc = upload(ctx, T->d_sVal, sv.data(), sizeof(double) * sv.size())) ||
        (rc = upload(ctx, T->d_sRhs, sr.data(), sizeof(double) * sr.size())) ||
        (rc = upload(ctx, T->d_penPtr, pp.data(), sizeof(int) * pp.size())) ||
        (rc = upload(ctx, T->d_penCol, pc.data(), sizeof(int) * pc.size())) ||
        (rc = upload(ctx, T->d_penVal, pv.data(), sizeof(double) * pv.size())))
        return rc;
    // gather lists of the constraint load
    std::vector<int> termRow(mc.size(), 0), order;
    for (int r = 0; r < T->mpcDim; ++r)
        for (int k = T->mRange[r]; k < T->mRange[r + 1]; ++k) {
            termRow[k] = r;
            if (T->mCol[k] >= 0) order.push_back(k);
        }
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return T->mCol[a] < T->mCol[b]; });
    std::vector<int> gptr, grow;
    for (size_t q = 0; q < order.size(); ++q)
        if (q == 0 || T->mCol[order[q]] != T->mCol[order[q - 1]]) {
            gptr.push_back((int)q);
            grow.push_back(T->mCol[order[q]]);
        }
    gptr.push_back((int)order.size());
    T->targets = (int)grow.size();
    if (order.empty()) {
        order.push_back(0);  // placeholders, never read (no target)
        grow.push_back(0);
    }
    if ((rc = upload(ctx, T->d_gPtr, gptr.data(), sizeof(int) * gptr.size())) ||
        (rc = upload(ctx, T->d_gTerm, order.data(), sizeof(int) * order.size())) ||
        (rc = upload(ctx, T->d_gRow, grow.data(), sizeof(int) * grow.size())) ||
        (rc = upload(ctx, T->d_termRow, termRow.data(), sizeof(int) * termRow.size())) ||
        (rc = dev_alloc(ctx, T->d_mDef, sizeof(double) * std::max(T->mpcDim, 1))))
        return rc;
    T->scaled = 1;
    if (mpc_mat) std::copy(T->sVal.begin(), T->sVal.end(), mpc_mat);
    if (mpc_rhs) std::copy(T->sRhs.begin(), T->sRhs.end(), mpc_rhs);
    return ASTRO_OK;
}

extern "C" int astro_thermal_constraint_load(astro_ctx *ctx, const double *node_temp, double *thermal_load) {
    if (!ctx || !thermal_load) return ASTRO_ERR_ARG;
    ThermPlan *T = plan_of(ctx);
    if (!T) return set_err(ctx, ASTRO_ERR_STATE, "thermal: astro_thermal_setup not called");
    if (T->mpcDim == 0) return ASTRO_OK;
    if (!T->scaled) return set_err(ctx, ASTRO_ERR_STATE, "thermal: constraints not scaled (astro_thermal_scale_mpc)");
    const int N = ctx->P.N;
    DevBuf dT, dL;
    int rc = up_opt(ctx, dT, node_temp, N);
    if (!rc) rc = upload(ctx, dL, thermal_load, sizeof(double) * N);
    if (!rc) {
        k_th_mpc_defect<<<(T->mpcDim + 127) / 128, 128, 0, ctx->stream>>>(
            T->mpcDim, dptr<int>(T->d_mRange), dptr<int>(T->d_mCol), dptr<double>(T->d_sVal), dptr<double>(T->d_sRhs),
            dT.p ? dptr<double>(dT) : nullptr, dptr<double>(T->d_mDef));
        if (T->targets)
            k_th_mpc_load<<<(T->targets + 127) / 128, 128, 0, ctx->stream>>>(
                T->targets, dptr<int>(T->d_gPtr), dptr<int>(T->d_gTerm), dptr<int>(T->d_gRow), dptr<int>(T->d_termRow),
                dptr<double>(T->d_sVal), dptr<double>(T->d_mDef), dptr<double>(dL));
        cudaError_t e = cudaGetLastError();
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(thermal_load, dL.p, sizeof(double) * N, cudaMemcpyDeviceToHost, ctx->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
        rc = cuda_check(ctx, e, "thermal constraint load");
    }
    dev_free(dT);
    dev_free(dL);
    return rc;
}

extern "C" int astro_thermal_heat_gen(astro_ctx *ctx, double q, const int32_t *elements, int32_t count,
                                      double *thermal_load) {
    if (!ctx || !thermal_load || count < 0) return ASTRO_ERR_ARG;
    ThermPlan *T = plan_of(ctx);
    if (!T) return set_err(ctx, ASTRO_ERR_STATE, "thermal: astro_thermal_setup not called");
    const AstroPrep &P = ctx->P;
    if (elements)
        for (int k = 0; k < count; ++k)
            if (elements[k] < 1 || elements[k] > P.E) return set_err(ctx, ASTRO_ERR_ARG, "element number out of range");
    std::vector<int> on((size_t)P.E, elements ? 0 : 1);
    if (elements)
        for (int k = 0; k < count; ++k) ++on[elements[k] - 1];
    std::vector<int> list, ptr(1, 0);
    std::vector<double> mult;
    for (int col = 0; col < P.ncolors; ++col) {
        for (int k = P.colorPtr[col]; k < P.colorPtr[col + 1]; ++k)
            if (on[P.colorEls[k]]) {
                list.push_back(P.colorEls[k]);
                mult.push_back((double)on[P.colorEls[k]]);
            }
        ptr.push_back((int)list.size());
    }
    if (list.empty()) return ASTRO_OK;
    DevBuf dl, dm, dL;
    int rc = upload(ctx, dl, list.data(), sizeof(int) * list.size());
    if (!rc) rc = upload(ctx, dm, mult.data(), sizeof(double) * mult.size());
    if (!rc) rc = upload(ctx, dL, thermal_load, sizeof(double) * P.N);
    if (!rc) {
        ThArgs A = th_args(ctx, T);
        A.load = dptr<double>(dL);
        for (int col = 0; A.shell && col < P.ncolors; ++col) {
            A.count = ptr[col + 1] - ptr[col];
            if (!A.count) continue;
            A.els = dptr<int>(dl) + ptr[col];
            k_th_heatgen<<<(A.count + 127) / 128, 128, 0, ctx->stream>>>(A, q, dptr<double>(dm) + ptr[col]);
        }
        if (!A.shell)
            rc = th_bricks(ctx, T, A, dptr<int>(dl), ptr, dptr<double>(dm), [&](const ThArgs &B, unsigned g) {
                k_th_brick_heat<<<g, kThThreads, 0, ctx->stream>>>(B, q);
            });
    }
    if (!rc) {
        cudaError_t e = cudaGetLastError();
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(thermal_load, dL.p, sizeof(double) * P.N, cudaMemcpyDeviceToHost, ctx->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
        rc = cuda_check(ctx, e, "heat generation");
    }
    dev_free(dl);
    dev_free(dm);
    dev_free(dL);
    return rc;
}

// thermal -= component 1 of the traction load (the surfaceFlux branch takes the flux as the first
// traction component and subtracts the element's component-1 nodal forces)
__global__ void k_th_flux_extract(int N, int dpn, const double *__restrict__ el, double *__restrict__ load) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r < N) load[r] = load[r] - el[(size_t)r * dpn];
}

extern "C" int astro_thermal_surface_flux(astro_ctx *ctx, int32_t nfaces, const int32_t *face_el,
                                          const int32_t *face_num, double flux, double *thermal_load) {
    if (!ctx || !thermal_load || nfaces < 0 || (nfaces && (!face_el || !face_num))) return ASTRO_ERR_ARG;
    if (!plan_of(ctx)) return set_err(ctx, ASTRO_ERR_STATE, "thermal: astro_thermal_setup not called");
    const AstroPrep &P = ctx->P;
    for (int f = 0; f < nfaces; ++f) {
        const int e = face_el[f], fn = face_num[f];
        if (e < 1 || e > P.E) return set_err(ctx, ASTRO_ERR_ARG, "face element out of range");
        if (fn < 1 || fn > ((ctx->etype[e - 1] == 8 || ctx->etype[e - 1] == 81) ? 6 : 2)) return set_err(ctx, ASTRO_ERR_ARG, "face number out of range");
    }
    if (!nfaces) return ASTRO_OK;
    DevBuf dfe, dfn, del, dL;
    int rc = upload(ctx, dfe, face_el, sizeof(int) * nfaces);
    if (!rc) rc = upload(ctx, dfn, face_num, sizeof(int) * nfaces);
    if (!rc) rc = dev_alloc(ctx, del, sizeof(double) * P.n);
    if (!rc) rc = upload(ctx, dL, thermal_load, sizeof(double) * P.N);
    if (!rc) {
        cudaMemsetAsync(del.p, 0, sizeof(double) * P.n, ctx->stream);
        const double tr[3] = {flux, 0.0, 0.0};
        rc = surface_load_dev(ctx, nfaces, dptr<int>(dfe), dptr<int>(dfn), tr, 0.0, dptr<double>(del));
    }
    if (!rc) {
        k_th_flux_extract<<<(P.N + 255) / 256, 256, 0, ctx->stream>>>(P.N, P.dpn, dptr<double>(del), dptr<double>(dL));
        cudaError_t e = cudaGetLastError();
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(thermal_load, dL.p, sizeof(double) * P.N, cudaMemcpyDeviceToHost, ctx->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
        rc = cuda_check(ctx, e, "surface flux");
    }
    DevBuf *v[] = {&dfe, &dfn, &del, &dL};
    for (DevBuf *x : v) dev_free(*x);
    return rc;
}

extern "C" int astro_thermal_solve(astro_ctx *ctx, const double *rhs, double *dtemp, double rtol, int32_t max_iters,
                                   astro_solve_stats *stats) {
    if (!ctx || !rhs || !dtemp || !(rtol > 0.0) || max_iters < 1) return ASTRO_ERR_ARG;
    ThermPlan *T = plan_of(ctx);
    if (!T || !T->haveMat) return set_err(ctx, ASTRO_ERR_STATE, "thermal: conductivity matrix not assembled");
    if (T->mpcDim > 0 && !T->scaled)
        return set_err(ctx, ASTRO_ERR_STATE, "thermal: constraints not scaled (astro_thermal_scale_mpc)");
    const AstroPrep &P = ctx->P;
    const int N = P.N;
    cudaStream_t s = ctx->stream;
    const unsigned rg = std::min((N + kCgThreads - 1) / kCgThreads, kCgMaxCtas);
    DevBuf b, &x = T->d_cg[0], &r = T->d_cg[1], &z = T->d_cg[2], &p = T->d_cg[3], &Ap = T->d_cg[4], &dinv = T->d_cg[5],
              &part = T->d_cg[6], &sc = T->d_cg[7];
    int rc;
    if (!T->slots) {
        for (int i = 0; i < N; ++i) T->slots = std::max(T->slots, P.bRowPtr[i + 1] - P.bRowPtr[i]);
        T->ld = (N + 31) / 32 * 32;
    }
    const size_t ellN = (size_t)T->slots * T->ld;
    if (!sc.p) {
        if ((rc = dev_alloc(ctx, T->d_ellCol, sizeof(int) * ellN)) || (rc = dev_alloc(ctx, T->d_ell, sizeof(double) * ellN)) ||
            (rc = dev_alloc(ctx, x, sizeof(double) * N)) || (rc = dev_alloc(ctx, r, sizeof(double) * N)) ||
            (rc = dev_alloc(ctx, z, sizeof(double) * N)) || (rc = dev_alloc(ctx, p, sizeof(double) * N)) ||
            (rc = dev_alloc(ctx, Ap, sizeof(double) * N)) || (rc = dev_alloc(ctx, dinv, sizeof(double) * N)) ||
            (rc = dev_alloc(ctx, part, sizeof(double) * 3 * rg)) || (rc = dev_alloc(ctx, sc, sizeof(CgScal))))
            return rc;
    }
    if ((rc = upload(ctx, b, rhs, sizeof(double) * N)) ||
        (rc = cuda_check(ctx, cudaMemcpyAsync(x.p, dtemp, sizeof(double) * N, cudaMemcpyHostToDevice, s), "upload"))) {
        dev_free(b);
        return rc;
    }
    struct Events {
        cudaEvent_t e0 = nullptr, e1 = nullptr;
        Events() {
            cudaEventCreate(&e0);
            cudaEventCreate(&e1);
        }
        ~Events() {
            cudaEventDestroy(e0);
            cudaEventDestroy(e1);
        }
    } ev;
    CgMat A;
    std::memset(&A, 0, sizeof(A));  // compared bytewise as the graph's key
    A.N = N;
    A.S = T->slots;
    A.ld = T->ld;
    A.v = dptr<double>(T->d_ell);
    A.col = dptr<int>(T->d_ellCol);
    A.pp = T->mpcDim ? dptr<int>(T->d_penPtr) : nullptr;
    A.pc = dptr<int>(T->d_penCol);
    A.pv = dptr<double>(T->d_penVal);
    CgScal *S = dptr<CgScal>(sc);
    cudaMemsetAsync(sc.p, 0, sizeof(CgScal), s);
    cudaEventRecord(ev.e0, s);
    k_cg_ell<<<(unsigned)((ellN + 255) / 256), 256, 0, s>>>(N, T->slots, T->ld, dptr<int>(ctx->d_bRowPtr),
                                                           dptr<int>(ctx->d_bCol), dptr<double>(T->d_val),
                                                           dptr<double>(T->d_ell),
                                                           T->haveCols ? nullptr : dptr<int>(T->d_ellCol));
    if ((rc = cuda_check(ctx, cudaGetLastError(), "thermal solve"))) {
        dev_free(b);
        return rc;
    }
    T->haveCols = 1;
    double *pPap = dptr<double>(part), *pRz = pPap + rg, *pRr = pRz + rg;
    auto start = [&] {
        k_cg_init<<<rg, kCgThreads, 0, s>>>(A, dptr<double>(b), dptr<double>(x), dptr<double>(dinv), dptr<double>(r),
                                            dptr<double>(p), pRz, pRr);
        k_cg_init_sum<<<1, kCgThreads, 0, s>>>((int)rg, pRz, pRr, S);
    };
    start();
    auto iterate = [&](int it0, int count) {
        for (int k = 0; k < count; ++k) {
            const int par = (it0 + k) & 1, want = k == count - 1;
            k_cg_ap<<<rg, kCgThreads, 0, s>>>(A, dptr<double>(p), dptr<double>(Ap), pPap);
            k_cg_step<<<rg, kCgThreads, 0, s>>>(N, par, want, S, pPap, dptr<double>(x), dptr<double>(r), dptr<double>(p),
                                                dptr<double>(Ap), dptr<double>(dinv), dptr<double>(z), pRz, pRr);
            k_cg_dir<<<rg, kCgThreads, 0, s>>>(N, par, want, S, pRz, pRr, dptr<double>(z), dptr<double>(p));
        }
    };
    CgRes Q;
    size_t smem = 0;
    Q.op = {A.v, A.col, A.S, A.ld, A.pp, nullptr, A.pc, A.pv, N, 1};
    Q.x = dptr<double>(x);
    Q.r = dptr<double>(r);
    Q.p = dptr<double>(p);
    Q.dinv = dptr<double>(dinv);
    Q.sc = S;
    Q.N = N;
    if ((rc = cg_resident_plan(ctx, T, &Q, &smem))) {
        dev_free(b);
        return rc;
    }
    // a batch as a graph, kept while the matrix tables stay where they are
    auto batch = [&]() -> int {
        if (T->cgExec && std::memcmp(&T->cgMat, &A, sizeof(A)) == 0) return ASTRO_OK;
        if (T->cgExec) cudaGraphExecDestroy(T->cgExec);
        T->cgExec = nullptr;
        cudaGraph_t g = nullptr;
        cudaError_t e = cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal);
        if (e == cudaSuccess) {
            iterate(0, kCgBatch);
            e = cudaStreamEndCapture(s, &g);
        }
        if (e == cudaSuccess) e = cudaGraphInstantiate(&T->cgExec, g, 0);
        if (g) cudaGraphDestroy(g);
        const int grc = cuda_check(ctx, e, "thermal solve graph");
        if (grc) T->cgExec = nullptr;
        else std::memcpy(&T->cgMat, &A, sizeof(A));
        return grc;
    };
    if (!Q.R && (rc = batch())) {
        dev_free(b);
        return rc;
    }
    double rr = 0.0;
    CgScal hs{};
    int it = 0, status = ASTRO_ERR_MAXIT;
    cudaMemcpyAsync(&hs, S, sizeof(hs), cudaMemcpyDeviceToHost, s);
    cudaStreamSynchronize(s);
    const double bn = std::sqrt(hs.bb);
    if (bn == 0.0) status = ASTRO_OK;
    while (!rc && status == ASTRO_ERR_MAXIT && it < max_iters) {
        cudaError_t e = cudaSuccess;
        bool refused = false;
        if (Q.R) {
            Q.iters = std::min(kCgResIters, max_iters - it);
            Q.target = rtol * bn;
            void *args[] = {&Q};
            e = cudaMemsetAsync(T->d_words.p, 0, T->d_words.bytes, s);
            if (e == cudaSuccess)
                e = cudaLaunchCooperativeKernel((const void *)k_cg_resident, dim3(Q.G), dim3(astro_kry::kResT), args, smem, s);
            refused = e != cudaSuccess;
        } else {
            const int chunk = std::min(kCgBatch, max_iters - it);
            if (chunk == kCgBatch) cudaGraphLaunch(T->cgExec, s);
            else iterate(0, chunk);  // (after whole batches: even)
            it += chunk;
            e = cudaGetLastError();
        }
        if (e == cudaSuccess) e = cudaMemcpyAsync(&hs, S, sizeof(hs), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (refused || (e == cudaSuccess && hs.stuck)) {
            // the GPU does not hold the whole grid now (other work on it): on from this x in batches (the CTAs
            // may have stopped at different iterations, so r and p are formed anew)
            cudaGetLastError();
            if (!refused) it += hs.its;
            Q.R = 0;
            if ((rc = cuda_check(ctx, cudaMemsetAsync(sc.p, 0, sizeof(CgScal), s), "thermal solve")) || (rc = batch())) break;
            start();
            continue;
        }
        if ((rc = cuda_check(ctx, e, "thermal solve"))) break;
        rr = hs.rr;
        if (Q.R) it += hs.its;
        if (!std::isfinite(rr)) {
            status = ASTRO_ERR_NAN;
            break;
        }
        if (std::sqrt(rr) <= rtol * bn) status = ASTRO_OK;
    }
    cudaEventRecord(ev.e1, s);
    if (!rc) {
        cudaError_t e = cudaMemcpyAsync(dtemp, x.p, sizeof(double) * N, cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        rc = cuda_check(ctx, e, "thermal solve");
    }
    if (stats) {
        std::memset(stats, 0, sizeof(*stats));
        stats->iterations = it;
        stats->status = rc ? rc : status;
        stats->rel_residual = bn > 0.0 ? std::sqrt(rr) / bn : 0.0;
        stats->residual_kind = 64;
        float ms = 0.0f;
        cudaEventElapsedTime(&ms, ev.e0, ev.e1);
        stats->seconds = ms * 1e-3;
    }
    dev_free(b);
    if (rc) return rc;
    if (status == ASTRO_ERR_MAXIT) return set_err(ctx, ASTRO_ERR_MAXIT, "thermal solve: iteration limit");
    if (status == ASTRO_ERR_NAN) return set_err(ctx, ASTRO_ERR_NAN, "thermal solve: non-finite residual");
    return ASTRO_OK;
}

// ---- design sensitivities (getdRthermaldD, Working/AStrO_commandFunctions.f90:1016-1170) ---------
// Complex step: the elements that depend on the design variable are evaluated in complex FP64
// with d + i h, one thread per element, colour by colour (a colour's elements share no node), and
// Im / h is accumulated at their nodes.  The complex path's Gauss points are the single-precision
// 1/sqrt(3) of the reference's c_ constants.
namespace {

struct ThCsArgs {
    int dvar;
    double h;
    const double *secOrig;  // (S,9) column-major section orientation as given
    const int *n2dR, *n2d;  // node design maps (null: none)
    const double *n2c;
    const double *mult;     // per listed element: how often the load lists it (heat generation)
    double q;               // heat generation per unit volume
    double *out;            // rank-order derivative
};

// The element frame and its nodes in it, in T: nodes with + i h coef on d's nodeCoord terms
// (r_getNodeCoord, designProp :945-968; the real offsets of every nodeCoord variable are already
// in the node list), the section orientation rotated by its orientation variables
// (r_getOrientation, :187-221) and, for shells, correctAlpha.
template <class T>
__device__ void th_frame_t(const ThArgs &A, const ThPropArgs &P, const ThCsArgs &C, int e, T Xl[8][3], int rk[8]) {
    const int npe = A.shell ? 4 : 8;
    const T ih = pert_i<T>(C.h);
    T Xg[8][3];
    for (int a = 0; a < npe; ++a) {
        const int nd = A.elist[8 * (size_t)e + a];
        rk[a] = A.rank[nd - 1] - 1;
        for (int k = 0; k < 3; ++k) Xg[a][k] = T(A.nodes[3 * (size_t)(nd - 1) + k]);
        if (C.n2dR)
            for (int t = C.n2dR[nd - 1]; t < C.n2dR[nd]; ++t) {
                const int d = C.n2d[t];
                if (d == C.dvar && P.dcat[d - 1] == ASTRO_DCAT_NODE_COORD) Xg[a][P.dcomp[d - 1] - 1] += C.n2c[t] * ih;
            }
    }
    T loc[3] = {T(0.0), T(0.0), T(0.0)};
    if (P.e2dR)
        for (int q = P.e2dR[e]; q < P.e2dR[e + 1]; ++q) {
            const int d = P.e2d[q];
            if (P.dcat[d - 1] != ASTRO_DCAT_ORIENTATION) continue;
            T v = T(P.dval[d - 1]);
            if (d == C.dvar) v = v + ih;
            loc[P.dcomp[d - 1] - 1] = loc[P.dcomp[d - 1] - 1] + P.e2c[q] * v;
        }
    const int sec = P.esec[e];
    T al[3][3], gr[3], orient[3][3];
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) al[i][j] = T(C.secOrig[9 * (size_t)(sec - 1) + 3 * j + i]);
    for (int i = 0; i < 3; ++i) gr[i] = al[0][i] * loc[0] + al[1][i] * loc[1] + al[2][i] * loc[2];
    a_rotate<T>(orient, al, gr, 0, 0);
    if (A.shell) {
        T X4[4][3];
        for (int a = 0; a < 4; ++a)
            for (int k = 0; k < 3; ++k) X4[a][k] = Xg[a][k];
        shell_correct_alpha<T>(orient, X4);
    }
    for (int a = 0; a < npe; ++a)
        for (int i = 0; i < 3; ++i) Xl[a][i] = orient[i][0] * Xg[a][0] + orient[i][1] * Xg[a][1] + orient[i][2] * Xg[a][2];
}

// The complex Gauss point, called out of line.  Inlined into k_th_elem_cs, this CUDA 13.0 build
// for sm_103a returned wrong shape-function gradients for every node but the first, although
// the parametric derivatives and the inverse Jacobian inside the routine were right.  The same source
// built for the host, built with -G, or called out of line gives the right gradients.
__device__ __noinline__ void th_point_cs(int shell, const cplx Xl[8][3], int g, double N[8], cplx Nx[8][3],
                                         cplx &wdet) {
    th_point_t<cplx>(shell, Xl, AK<cplx>::rt3, g, N, Nx, wdet);
}

// element part: out[rank] += Im(Rt) / h (r_getElRtk + r_getElRtm in complex)
__global__ void k_th_elem_cs(ThArgs A, ThPropArgs P, ThCsArgs C) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= A.count) return;
    const int e = A.els[q];
    const int npe = A.shell ? 4 : 8, ngp = A.shell ? 4 : 8;
    cplx Xl[8][3];
    int rk[8];
    th_frame_t<cplx>(A, P, C, e, Xl, rk);
    cplx tc[3][3], sh, secT;
    th_props_t<cplx>(P, e, C.dvar, C.h, tc, sh, secT);
    double T[8], Td[8];
    for (int a = 0; a < npe; ++a) {
        T[a] = A.temp ? A.temp[rk[a]] : 0.0;
        Td[a] = 0.0;
        if (A.dynamic) {
            const double pT = A.ptemp ? A.ptemp[rk[a]] : 0.0, pTd = A.ptdot ? A.ptdot[rk[a]] : 0.0;
            Td[a] = (1.0 / A.gamma) * ((1.0 / A.delT) * (T[a] - pT) - 1.0 * (1.0 - A.gamma) * pTd);
        }
    }
    cplx Rt[8];
    for (int g = 0; g < ngp; ++g) {
        double N[8];
        cplx Nx[8][3], wd;
        th_point_cs(A.shell, Xl, g, N, Nx, wd);
        cplx Tx[3];
        for (int a = 0; a < npe; ++a)
            for (int k = 0; k < 3; ++k) Tx[k] = Tx[k] + Nx[a][k] * T[a];
        cplx qv[3];
        for (int i = 0; i < 3; ++i) qv[i] = wd * (tc[i][0] * Tx[0] + tc[i][1] * Tx[1] + tc[i][2] * Tx[2]);
        for (int a = 0; a < npe; ++a) Rt[a] = Rt[a] + Nx[a][0] * qv[0] + Nx[a][1] * qv[1] + Nx[a][2] * qv[2];
        if (A.dynamic) {
            double pt = 0.0;
            for (int a = 0; a < npe; ++a) pt = pt + Td[a] * N[a];
            const cplx c = (wd * sh) * pt;
            for (int a = 0; a < npe; ++a) Rt[a] = Rt[a] + c * N[a];
        }
    }
    const double hInv = 1.0 / C.h;
    for (int a = 0; a < npe; ++a) C.out[rk[a]] += hInv * Rt[a].im;
}

// bodyHeatGen branch: out[rank] -= mult Im(q integral of N (times the section thickness for
// shells)) / h
__global__ void k_th_heatgen_cs(ThArgs A, ThPropArgs P, ThCsArgs C) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= A.count) return;
    const int e = A.els[q];
    const int npe = A.shell ? 4 : 8, ngp = A.shell ? 4 : 8;
    cplx Xl[8][3];
    int rk[8];
    th_frame_t<cplx>(A, P, C, e, Xl, rk);
    cplx w[8];
    for (int g = 0; g < ngp; ++g) {
        double N[8];
        cplx Nx[8][3], wd;
        th_point_cs(A.shell, Xl, g, N, Nx, wd);
        for (int a = 0; a < npe; ++a) w[a] = w[a] + (C.q * N[a]) * wd;
    }
    cplx t = cplx(1.0);
    if (A.shell) {
        cplx tc[3][3], sh;
        th_props_t<cplx>(P, e, C.dvar, C.h, tc, sh, t);
    }
    const double hInv = 1.0 / C.h;
    for (int a = 0; a < npe; ++a) C.out[rk[a]] -= C.mult[q] * (hInv * (t * w[a]).im);
}

// surfaceFlux branch, one thread per face: the face's four nodal values Im(flux integral of
// N dA) / h, dA the true area element (as the load itself), into fv[4 f + k]
__global__ void k_th_flux_cs(int nf, const int *__restrict__ faceEl, const int *__restrict__ faceNum,
                             const int *__restrict__ etype, const int *__restrict__ elist,
                             const double *__restrict__ nodes, const int *__restrict__ n2dR,
                             const int *__restrict__ n2d, const double *__restrict__ n2c, const int *__restrict__ dcat,
                             const int *__restrict__ dcomp, int dvar, double h, double flux, double *__restrict__ fv) {
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= nf) return;
    const int hexF[6][4] = {{4, 3, 2, 1}, {5, 6, 7, 8}, {1, 2, 6, 5}, {2, 3, 7, 6}, {3, 4, 8, 7}, {4, 1, 5, 8}};
    const int shF[2][4] = {{1, 2, 3, 4}, {1, 4, 3, 2}};
    const int el = faceEl[f] - 1, fn = faceNum[f] - 1;
    const int *fl = (etype[el] == 8 || etype[el] == 81) ? hexF[fn] : shF[fn];
    cplx X[4][3];
    for (int k = 0; k < 4; ++k) {
        const int nd = elist[8 * (size_t)el + fl[k] - 1];
        for (int d = 0; d < 3; ++d) X[k][d] = cplx(nodes[3 * (size_t)(nd - 1) + d]);
        if (n2dR)
            for (int t = n2dR[nd - 1]; t < n2dR[nd]; ++t)
                if (n2d[t] == dvar && dcat[dvar - 1] == ASTRO_DCAT_NODE_COORD)
                    X[k][dcomp[dvar - 1] - 1] += cplx(0.0, n2c[t] * h);
    }
    const double g = AK<cplx>::rt3;
    cplx acc[4];
    for (int gp = 0; gp < 4; ++gp) {
        const double s = (gp & 1) ? g : -g, r = (gp & 2) ? g : -g;
        const double N_[4] = {0.25 * (1 - s) * (1 - r), 0.25 * (1 + s) * (1 - r), 0.25 * (1 + s) * (1 + r),
                              0.25 * (1 - s) * (1 + r)};
        const double Ns[4] = {-0.25 * (1 - r), 0.25 * (1 - r), 0.25 * (1 + r), -0.25 * (1 + r)};
        const double Nr[4] = {-0.25 * (1 - s), -0.25 * (1 + s), 0.25 * (1 + s), 0.25 * (1 - s)};
        cplx a[3], b[3];
        for (int k = 0; k < 4; ++k)
            for (int d = 0; d < 3; ++d) {
                a[d] = a[d] + Ns[k] * X[k][d];
                b[d] = b[d] + Nr[k] * X[k][d];
            }
        const cplx cx = a[1] * b[2] - a[2] * b[1], cy = a[2] * b[0] - a[0] * b[2], cz = a[0] * b[1] - a[1] * b[0];
        const cplx s2 = cx * cx + cy * cy + cz * cz;
        // principal square root to first order in the imaginary part (exact for the complex step)
        const double re = sqrt(s2.re);
        const cplx dA(re, s2.im / (2.0 * re));
        for (int k = 0; k < 4; ++k) acc[k] = acc[k] + (flux * N_[k]) * dA;
    }
    for (int k = 0; k < 4; ++k) fv[4 * (size_t)f + k] = acc[k].im / h;
}

// out[row[g]] += the face values of its slots, in face order (gPtr / gSlot as face_gather_kernel)
__global__ void k_th_face_gather(int ng, const int *__restrict__ gPtr, const int *__restrict__ gSlot,
                                 const int *__restrict__ gRow, const double *__restrict__ fv, double *__restrict__ out) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= ng) return;
    double s = out[gRow[g]];
    for (int q = gPtr[g]; q < gPtr[g + 1]; ++q) s = s + fv[gSlot[q]];
    out[gRow[g]] = s;
}

// 'nodeLoad' / 'thermal' variables (d_component 7) active at t (dActTime(1) < t < dActTime(2)):
// mode 0 load[rank] += coef d of every variable, mode 1 load[rank] -= coef for dvar only
__global__ void k_th_node_dload(int N, const int *__restrict__ rank, const int *__restrict__ n2dR,
                                const int *__restrict__ n2d, const double *__restrict__ n2c,
                                const int *__restrict__ dcat, const int *__restrict__ dcomp,
                                const double *__restrict__ dval, const double *__restrict__ act, double t, int mode,
                                int dvar, double *__restrict__ load) {
    const int nd = blockIdx.x * blockDim.x + threadIdx.x;
    if (nd >= N) return;
    double v = load[rank[nd] - 1];
    for (int q = n2dR[nd]; q < n2dR[nd + 1]; ++q) {
        const int d = n2d[q];
        if (dcat[d - 1] != ASTRO_DCAT_NODE_LOAD || dcomp[d - 1] != 7 || (mode == 1 && d != dvar)) continue;
        if (act && !(t > act[2 * (d - 1)] && act[2 * (d - 1) + 1] > t)) continue;
        v = v + (mode == 0 ? n2c[q] * dval[d - 1] : -n2c[q]);
    }
    load[rank[nd] - 1] = v;
}

}  // namespace

// Per element (0-based): 1 when it depends on dvar (getdToElComp, Working/AStrO_bookKeeping.f90:7-129:
// the element's own design variables, and the nodeCoord variables of its nodes).
static std::vector<char> th_dependents(const astro_ctx *ctx, int dvar) {
    const AstroPrep &P = ctx->P;
    std::vector<char> dep((size_t)P.E, 0);
    for (int e = 0; e < P.E; ++e)
        for (int q = ctx->e2dRange[e]; q < ctx->e2dRange[e + 1]; ++q)
            if (ctx->e2d[q] == dvar) dep[e] = 1;
    if (!ctx->n2dRange.empty() && ctx->dCat[dvar - 1] == ASTRO_DCAT_NODE_COORD) {
        std::vector<char> nd((size_t)P.N + 1, 0);
        for (int n = 1; n <= P.N; ++n)
            for (int q = ctx->n2dRange[n - 1]; q < ctx->n2dRange[n]; ++q)
                if (ctx->n2d[q] == dvar) nd[n] = 1;
        for (int e = 0; e < P.E; ++e)
            for (int a = 0; a < P.npe; ++a)
                if (nd[ctx->elist[8 * (size_t)e + a]]) dep[e] = 1;
    }
    return dep;
}

static int th_check_dvar(astro_ctx *ctx, int dvar, double h) {
    if (!plan_of(ctx)) return set_err(ctx, ASTRO_ERR_STATE, "thermal: astro_thermal_setup not called");
    if (dvar < 1 || dvar > ctx->numDvars)
        return set_err(ctx, ASTRO_ERR_ARG, "design variable " + std::to_string(dvar) + " out of range");
    if (!(h > 0.0)) return set_err(ctx, ASTRO_ERR_ARG, "complex step h must be positive");
    return ASTRO_OK;
}

static ThCsArgs th_cs_args(astro_ctx *ctx, int dvar, double h, double *out) {
    ThCsArgs C = {};
    C.dvar = dvar;
    C.h = h;
    C.secOrig = dptr<double>(ctx->d_secOrig);
    const bool nd = !ctx->n2dRange.empty();
    C.n2dR = nd ? dptr<int>(ctx->d_n2dR) : nullptr;
    C.n2d = nd ? dptr<int>(ctx->d_n2d) : nullptr;
    C.n2c = nd ? dptr<double>(ctx->d_n2c) : nullptr;
    C.out = out;
    return C;
}

// The listed elements (with multiplicity, or all when elements is null) that depend on dvar, by
// colour.
static void th_listed_dependents(const astro_ctx *ctx, const std::vector<char> &dep, const int32_t *elements,
                                 int count, std::vector<int> &list, std::vector<double> &mult, std::vector<int> &ptr) {
    const AstroPrep &P = ctx->P;
    std::vector<int> times((size_t)P.E, elements ? 0 : 1);
    if (elements)
        for (int k = 0; k < count; ++k) ++times[elements[k] - 1];
    list.clear();
    mult.clear();
    ptr.assign(1, 0);
    for (int col = 0; col < P.ncolors; ++col) {
        for (int k = P.colorPtr[col]; k < P.colorPtr[col + 1]; ++k) {
            const int e = P.colorEls[k];
            if (dep[e] && times[e]) {
                list.push_back(e);
                mult.push_back((double)times[e]);
            }
        }
        ptr.push_back((int)list.size());
    }
}

// Runs `launch(els, count, mult)` over the colours of the listed elements with the derivative
// vector on the device, then copies it back.
template <class F>
static int th_cs_run(astro_ctx *ctx, const std::vector<int> &list, const std::vector<double> &mult,
                     const std::vector<int> &ptr, double *drtdd, bool zero, F launch) {
    const int N = ctx->P.N;
    DevBuf dl, dm, dout;
    int rc = ASTRO_OK;
    struct Free {
        DevBuf *b[3];
        ~Free() {
            for (auto *x : b) dev_free(*x);
        }
    } fr{{&dl, &dm, &dout}};
    if (zero) {
        if ((rc = dev_alloc(ctx, dout, sizeof(double) * N))) return rc;
        CK(cudaMemsetAsync(dout.p, 0, sizeof(double) * N, ctx->stream));
    } else if ((rc = upload(ctx, dout, drtdd, sizeof(double) * N))) {
        return rc;
    }
    if (!list.empty()) {
        if ((rc = upload(ctx, dl, list.data(), sizeof(int) * list.size())) ||
            (rc = upload(ctx, dm, mult.data(), sizeof(double) * mult.size())))
            return rc;
        for (size_t col = 0; col + 1 < ptr.size(); ++col) {
            const int cnt = ptr[col + 1] - ptr[col];
            if (cnt) launch(dptr<int>(dl) + ptr[col], cnt, dptr<double>(dm) + ptr[col], dptr<double>(dout));
        }
        if ((rc = cuda_check(ctx, cudaGetLastError(), "thermal complex step"))) return rc;
    }
    CK(cudaMemcpyAsync(drtdd, dout.p, sizeof(double) * N, cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    return ASTRO_OK;
}

extern "C" int astro_thermal_drdd(astro_ctx *ctx, int32_t dvar, double h, const astro_thermal_state *st,
                                  double *drtdd) {
    if (!ctx || !drtdd) return ASTRO_ERR_ARG;
    int rc;
    if ((rc = th_check_dvar(ctx, dvar, h))) return rc;
    if (st && st->dynamic && !(st->nm_gamma != 0.0 && st->del_t != 0.0))
        return set_err(ctx, ASTRO_ERR_ARG, "thermal: dynamic step needs gamma and a time step");
    ThermPlan *T = plan_of(ctx);
    const int N = ctx->P.N;
    std::vector<int> list, ptr;
    std::vector<double> mult;
    th_listed_dependents(ctx, th_dependents(ctx, dvar), nullptr, 0, list, mult, ptr);
    DevBuf dT, dpT, dpTd;
    struct Free {
        DevBuf *b[3];
        ~Free() {
            for (auto *x : b) dev_free(*x);
        }
    } fr{{&dT, &dpT, &dpTd}};
    if ((rc = up_opt(ctx, dT, st ? st->node_temp : nullptr, N)) ||
        (rc = up_opt(ctx, dpT, st ? st->prev_temp : nullptr, N)) ||
        (rc = up_opt(ctx, dpTd, st ? st->prev_tdot : nullptr, N)))
        return rc;
    ThArgs A = th_args(ctx, T);
    A.temp = dT.p ? dptr<double>(dT) : nullptr;
    A.ptemp = dpT.p ? dptr<double>(dpT) : nullptr;
    A.ptdot = dpTd.p ? dptr<double>(dpTd) : nullptr;
    A.dynamic = st ? st->dynamic : 0;
    A.gamma = st ? st->nm_gamma : 0.5;
    A.delT = st ? st->del_t : 0.0;
    const ThPropArgs Pa = th_prop_args(ctx, T);
    return th_cs_run(ctx, list, mult, ptr, drtdd, true, [&](const int *els, int cnt, const double *, double *out) {
        ThArgs a = A;
        a.els = els;
        a.count = cnt;
        k_th_elem_cs<<<(cnt + 63) / 64, 64, 0, ctx->stream>>>(a, Pa, th_cs_args(ctx, dvar, h, out));
    });
}

extern "C" int astro_thermal_heat_gen_drdd(astro_ctx *ctx, int32_t dvar, double h, double q, const int32_t *elements,
                                           int32_t count, double *drtdd) {
    if (!ctx || !drtdd || count < 0) return ASTRO_ERR_ARG;
    int rc;
    if ((rc = th_check_dvar(ctx, dvar, h))) return rc;
    const AstroPrep &P = ctx->P;
    if (elements)
        for (int k = 0; k < count; ++k)
            if (elements[k] < 1 || elements[k] > P.E) return set_err(ctx, ASTRO_ERR_ARG, "element number out of range");
    ThermPlan *T = plan_of(ctx);
    std::vector<int> list, ptr;
    std::vector<double> mult;
    th_listed_dependents(ctx, th_dependents(ctx, dvar), elements, count, list, mult, ptr);
    if (list.empty()) return ASTRO_OK;
    const ThArgs A = th_args(ctx, T);
    const ThPropArgs Pa = th_prop_args(ctx, T);
    return th_cs_run(ctx, list, mult, ptr, drtdd, false, [&](const int *els, int cnt, const double *m, double *out) {
        ThArgs a = A;
        a.els = els;
        a.count = cnt;
        ThCsArgs C = th_cs_args(ctx, dvar, h, out);
        C.mult = m;
        C.q = q;
        k_th_heatgen_cs<<<(cnt + 63) / 64, 64, 0, ctx->stream>>>(a, Pa, C);
    });
}

extern "C" int astro_thermal_surface_flux_drdd(astro_ctx *ctx, int32_t dvar, double h, int32_t nfaces,
                                               const int32_t *face_el, const int32_t *face_num, double flux,
                                               double *drtdd) {
    if (!ctx || !drtdd || nfaces < 0 || (nfaces && (!face_el || !face_num))) return ASTRO_ERR_ARG;
    int rc;
    if ((rc = th_check_dvar(ctx, dvar, h))) return rc;
    const AstroPrep &P = ctx->P;
    for (int f = 0; f < nfaces; ++f) {
        const int e = face_el[f], fn = face_num[f];
        if (e < 1 || e > P.E) return set_err(ctx, ASTRO_ERR_ARG, "face element out of range");
        if (fn < 1 || fn > ((ctx->etype[e - 1] == 8 || ctx->etype[e - 1] == 81) ? 6 : 2))
            return set_err(ctx, ASTRO_ERR_ARG, "face number out of range");
    }
    // the faces whose element depends on dvar, and the gather lists of their corner values
    static const int hexF[6][4] = {{4, 3, 2, 1}, {5, 6, 7, 8}, {1, 2, 6, 5}, {2, 3, 7, 6}, {3, 4, 8, 7}, {4, 1, 5, 8}};
    static const int shF[2][4] = {{1, 2, 3, 4}, {1, 4, 3, 2}};
    const std::vector<char> dep = th_dependents(ctx, dvar);
    std::vector<int> fe, fnum, slotRow;
    for (int f = 0; f < nfaces; ++f) {
        const int e = face_el[f] - 1;
        if (!dep[e]) continue;
        fe.push_back(face_el[f]);
        fnum.push_back(face_num[f]);
        const int *fl = (ctx->etype[e] == 8 || ctx->etype[e] == 81) ? hexF[face_num[f] - 1] : shF[face_num[f] - 1];
        for (int k = 0; k < 4; ++k) slotRow.push_back(P.currentRank[ctx->elist[8 * (size_t)e + fl[k] - 1]] - 1);
    }
    if (fe.empty()) return ASTRO_OK;
    std::vector<int> order(slotRow.size());
    for (size_t k = 0; k < order.size(); ++k) order[k] = (int)k;
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return slotRow[a] < slotRow[b]; });
    std::vector<int> gPtr(1, 0), gRow;
    for (size_t k = 0; k < order.size(); ++k) {
        if (k == 0 || slotRow[order[k]] != slotRow[order[k - 1]]) {
            if (k) gPtr.push_back((int)k);
            gRow.push_back(slotRow[order[k]]);
        }
    }
    gPtr.push_back((int)order.size());
    const int nf = (int)fe.size(), ng = (int)gRow.size(), N = P.N;
    DevBuf dfe, dfn, dfv, dgp, dgs, dgr, dout;
    struct Free {
        DevBuf *b[7];
        ~Free() {
            for (auto *x : b) dev_free(*x);
        }
    } fr{{&dfe, &dfn, &dfv, &dgp, &dgs, &dgr, &dout}};
    if ((rc = upload(ctx, dfe, fe.data(), sizeof(int) * nf)) || (rc = upload(ctx, dfn, fnum.data(), sizeof(int) * nf)) ||
        (rc = dev_alloc(ctx, dfv, sizeof(double) * 4 * (size_t)nf)) ||
        (rc = upload(ctx, dgp, gPtr.data(), sizeof(int) * gPtr.size())) ||
        (rc = upload(ctx, dgs, order.data(), sizeof(int) * order.size())) ||
        (rc = upload(ctx, dgr, gRow.data(), sizeof(int) * ng)) || (rc = upload(ctx, dout, drtdd, sizeof(double) * N)))
        return rc;
    const bool nd = !ctx->n2dRange.empty();
    k_th_flux_cs<<<(nf + 127) / 128, 128, 0, ctx->stream>>>(
        nf, dptr<int>(dfe), dptr<int>(dfn), dptr<int>(ctx->d_etype), dptr<int>(ctx->d_elist), dptr<double>(ctx->d_nodes),
        nd ? dptr<int>(ctx->d_n2dR) : nullptr, nd ? dptr<int>(ctx->d_n2d) : nullptr,
        nd ? dptr<double>(ctx->d_n2c) : nullptr, dptr<int>(ctx->d_dCat), dptr<int>(ctx->d_dComp), dvar, h, flux,
        dptr<double>(dfv));
    k_th_face_gather<<<(ng + 127) / 128, 128, 0, ctx->stream>>>(ng, dptr<int>(dgp), dptr<int>(dgs), dptr<int>(dgr),
                                                                 dptr<double>(dfv), dptr<double>(dout));
    if ((rc = cuda_check(ctx, cudaGetLastError(), "surface flux derivative"))) return rc;
    CK(cudaMemcpyAsync(drtdd, dout.p, sizeof(double) * N, cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    return ASTRO_OK;
}

static int th_node_dload(astro_ctx *ctx, double t, int mode, int dvar, double *vec) {
    const AstroPrep &P = ctx->P;
    if (ctx->n2dRange.empty()) return ASTRO_OK;
    DevBuf dv, act;
    int rc;
    struct Free {
        DevBuf *b[2];
        ~Free() {
            for (auto *x : b) dev_free(*x);
        }
    } fr{{&dv, &act}};
    if ((rc = upload(ctx, dv, vec, sizeof(double) * P.N))) return rc;
    if (!ctx->dActTime.empty() && (rc = upload(ctx, act, ctx->dActTime.data(), sizeof(double) * ctx->dActTime.size())))
        return rc;
    k_th_node_dload<<<(P.N + 127) / 128, 128, 0, ctx->stream>>>(
        P.N, dptr<int>(ctx->d_rank), dptr<int>(ctx->d_n2dR), dptr<int>(ctx->d_n2d), dptr<double>(ctx->d_n2c),
        dptr<int>(ctx->d_dCat), dptr<int>(ctx->d_dComp), dptr<double>(ctx->d_dVal), act.p ? dptr<double>(act) : nullptr,
        t, mode, dvar, dptr<double>(dv));
    if ((rc = cuda_check(ctx, cudaGetLastError(), "thermal nodal design load"))) return rc;
    CK(cudaMemcpyAsync(vec, dv.p, sizeof(double) * P.N, cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    return ASTRO_OK;
}

extern "C" int astro_thermal_design_node_load(astro_ctx *ctx, double time, double *thermal_load) {
    if (!ctx || !thermal_load) return ASTRO_ERR_ARG;
    return th_node_dload(ctx, time, 0, 0, thermal_load);
}

extern "C" int astro_thermal_node_load_drdd(astro_ctx *ctx, int32_t dvar, double time, double *drtdd) {
    if (!ctx || !drtdd) return ASTRO_ERR_ARG;
    if (dvar < 1 || dvar > ctx->numDvars)
        return set_err(ctx, ASTRO_ERR_ARG, "design variable " + std::to_string(dvar) + " out of range");
    return th_node_dload(ctx, time, 1, dvar, drtdd);
}
