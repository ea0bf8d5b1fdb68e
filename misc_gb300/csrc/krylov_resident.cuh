// A restart cycle of GMRES as one cooperative launch, for operators that fit the SMs' shared memory.
//
// The graph of krylov.cu spends 4 launches on an Arnoldi step and one on every hop of the polynomial
// preconditioner, and on models of up to 100,000 DOF or so each of them is a chain of latencies (launch,
// loads of the operator from L2, a last CTA that adds partial sums): 41 us a step in FP64 on 14,112
// rows, 8 us a hop on 91,875.  Here one CTA per SM owns R consecutive block rows for the whole cycle:
//   * their part of the operator (FP64 or FP32 values, or the FP16 planes of the hops), and in FP64
//     where it fits also of the Krylov basis, stays in shared memory;
//   * what a product needs of other CTAs' rows, the halo, is gathered from global memory (L2) into
//     shared memory once per product, and the columns are kept as 16-bit positions in it;
//   * a step needs a grid barrier per exchange: one per hop, one for the dot products, one for the norm
//     together with the next product's input.  The partial sums are then added by every CTA for
//     itself, in the same fixed order, so that all of them take the same decisions.
// 4,704 nodes in FP64: a step 38 us in the graph, 20 us here; 30,625 nodes: a hop 8.0 us there, 5.6 us here.
//
// The arithmetic is that of the graph's kernels (same precisions, classical Gram-Schmidt with the second
// pass on the Kahan-Parlett test, Givens rotations), the order of the sums differs.
//
// The grid barrier is a counter in global memory that only ever grows within a launch; the launch is
// cooperative, so all CTAs are resident.  Its wait is bounded: past the limit the CTA sets ctl->stuck and
// returns, as the others then do.
#pragma once
#include "krylov_ops.cuh"

namespace astro_kry {

constexpr int kResT = 1024, kResW = kResT / 32;
constexpr int kSpinLimit = 1 << 21;  // polls of the barrier (more than a second)
constexpr int kResMaxRows = 256;     // rows of a CTA: four lanes each in the hops

template <class TM, class TV> struct ResArgs {
    Op<TM> op;
    OpH hop;              // polynomial preconditioner (its values), or unused
    int deg;              // hops, 0 = Jacobi
    float theta, delta;   // the map of the recurrence
    const float *W;       // hop weights, (deg + 1) x dpn x dpn, already divided by lambda
    const float *amod;    // per-node hop scales, or null
    const TV *y0s;        // scales a residual into the preconditioner's input
    TV *x;
    const double *b;
    TV *V;                // Krylov basis, vector-major (used when it does not fit shared memory)
    size_t ld;
    TV *z[2];             // exchanged vectors (n each)
    GmresCtl *ctl;
    const double *target;
    double *part;         // 3 (kMaxM + 2) partial sums per CTA
    unsigned *bar;
    int *penLoc;          // per penalty entry of the row lists: its column's position in the owner's halo
    int m, n, N, R, G, H; // H: capacity of the halo
    int vShared;
};

struct ResLayout {
    size_t k, kr, col, list, halo, own, hes, v, total;
};
// Byte offsets of the CTA's arrays in dynamic shared memory.  poly: the hops' FP16 planes instead of the
// values of op.
template <class TM, class TV, int DPN>
__host__ __device__ inline ResLayout res_layout(int N, int S, int R, int H, int m, int poly, int vShared) {
    const size_t rows = ((size_t)R + 3) / 4 * 4;
    ResLayout L;
    size_t o = 0;
    auto put = [&](size_t bytes) {
        const size_t at = o;
        o += (bytes + 15) / 16 * 16;
        return at;
    };
    const size_t k = poly ? sizeof(uint4) * BvShape<DPN>::NV * S * rows : sizeof(TM) * (size_t)(DPN * DPN) * S * rows;
    const size_t bitmap = ((size_t)N + 31) / 32 * 4;  // of the halo, before the values are loaded
    L.k = put(k > bitmap ? k : bitmap);
    L.kr = put(poly ? sizeof(unsigned short) * BvShape<DPN>::REM * S * rows : 0);
    L.col = put(sizeof(unsigned short) * S * rows);
    L.list = put(sizeof(int) * (size_t)H);
    L.halo = put(sizeof(TV) * (size_t)H * DPN);
    L.own = put(sizeof(TV) * 5 * rows * DPN);  // w, products, three partial products
    L.hes = put(sizeof(double) * (size_t)(m + 1) * m);
    L.v = put(vShared ? sizeof(TV) * (size_t)(m + 1) * R * DPN : 0);
    L.total = o;
    return L;
}

// Marks the block columns of a CTA's rows (and of their penalty entries) in a bitmap of N bits; the halo
// size in *count.  Used by the count kernel and by the cycle itself.
template <class TM>
__device__ void res_mark(const Op<TM> &op, int row0, int rows, unsigned *bits, int words) {
    for (int i = threadIdx.x; i < words; i += blockDim.x) bits[i] = 0u;
    __syncthreads();
    for (int i = threadIdx.x; i < rows * op.S; i += blockDim.x) {
        const int c = op.col[(size_t)(i / rows) * op.ld + row0 + i % rows];
        atomicOr(bits + (c >> 5), 1u << (c & 31));
    }
    if (op.penPtr)
        for (int t = op.penPtr[row0] + threadIdx.x; t < op.penPtr[row0 + rows]; t += blockDim.x) {
            const int c = op.penCol[t] / op.dpn;
            atomicOr(bits + (c >> 5), 1u << (c & 31));
        }
    __syncthreads();
}

template <class TM> __global__ void k_res_halo(Op<TM> op, int R, int *maxHalo) {
    extern __shared__ unsigned bits[];
    const int row0 = blockIdx.x * R, rows = min(R, op.N - row0), words = (op.N + 31) / 32;
    if (rows <= 0) return;
    res_mark(op, row0, rows, bits, words);
    int c = 0;
    for (int i = threadIdx.x; i < words; i += blockDim.x) c += __popc(bits[i]);
    for (int o = 16; o; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    __shared__ int total;
    if (threadIdx.x == 0) total = 0;
    __syncthreads();
    if ((threadIdx.x & 31) == 0) atomicAdd(&total, c);
    __syncthreads();
    if (threadIdx.x == 0) atomicMax(maxHalo, total);
}

// Grid barrier number `phase` (1, 2, ...) in two halves, so that a warp can work between them; the wait
// is false when it was given up.
__device__ __forceinline__ void res_arrive(unsigned *bar) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
    }
}
__device__ __forceinline__ bool res_wait(unsigned *bar, unsigned phase, GmresCtl *ctl) {
    __shared__ int ok;
    if (threadIdx.x == 0) {
        const unsigned want = phase * gridDim.x;
        unsigned v = 0;
        int it = 0;
        for (; it < kSpinLimit; ++it) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
            if (v >= want) break;
        }
        ok = it < kSpinLimit;
        if (!ok) ctl->stuck = 1;
    }
    __syncthreads();
    return ok != 0;
}

template <class TM, class TV, int DPN, bool POLY>
__global__ void __launch_bounds__(kResT, 1) k_gmres_resident(ResArgs<TM, TV> A) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int DD = DPN * DPN;
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
    const int row0 = blockIdx.x * A.R, rows = max(0, min(A.R, A.N - row0)), nown = rows * DPN;
    const int Rp = (A.R + 3) / 4 * 4, S = A.op.S, m = A.m;
    const ResLayout L = res_layout<TM, TV, DPN>(A.N, S, A.R, A.H, m, POLY, A.vShared);
    TM *sK = reinterpret_cast<TM *>(smem + L.k);
    uint4 *sKv = reinterpret_cast<uint4 *>(smem + L.k);
    unsigned short *sKr = reinterpret_cast<unsigned short *>(smem + L.kr);
    unsigned short *sCol = reinterpret_cast<unsigned short *>(smem + L.col);
    int *sList = reinterpret_cast<int *>(smem + L.list);
    TV *sHalo = reinterpret_cast<TV *>(smem + L.halo);
    TV *sw = reinterpret_cast<TV *>(smem + L.own), *sy = sw + Rp * DPN;
    double *Hs = reinterpret_cast<double *>(smem + L.hes);  // column j at Hs + j (m + 1)
    TV *V = A.vShared ? reinterpret_cast<TV *>(smem + L.v) : A.V + (size_t)row0 * DPN;
    const size_t vld = A.vShared ? (size_t)A.R * DPN : A.ld;
    __shared__ double sh[kMaxM + 2], scs[kMaxM], ssn[kMaxM], sg[kMaxM + 1], sky[kMaxM], red[kResW];
    __shared__ double sInv, sHrot;
    __shared__ int sDone, sReorth, sHaloN, sBreak, sBad;
    unsigned phase = 0;
#define RES_BARRIER()  \
    res_arrive(A.bar); \
    if (!res_wait(A.bar, ++phase, A.ctl)) return

    // ---- the CTA's rows into shared memory: halo list, local columns, operator -----------------------
    {
        // bitmap of the halo in the (still unused) operator area
        unsigned *bits = reinterpret_cast<unsigned *>(smem + L.k);
        const int words = (A.N + 31) / 32;
        if (rows > 0) res_mark(A.op, row0, rows, bits, words);
        __shared__ int cnt[kResT + 1];
        const int per = (words + kResT - 1) / kResT, w0 = min(words, t * per), w1 = min(words, w0 + per);
        int c = 0;
        if (rows > 0)
            for (int i = w0; i < w1; ++i) c += __popc(bits[i]);
        cnt[t + 1] = c;
        if (t == 0) cnt[0] = 0;
        __syncthreads();
        for (int o = 1; o < kResT; o *= 2) {  // inclusive scan of cnt[1 ..]
            const int v = t + 1 > o ? cnt[t + 1 - o] : 0;
            __syncthreads();
            cnt[t + 1] += v;
            __syncthreads();
        }
        if (t == 0) sHaloN = cnt[kResT];
        if (cnt[kResT] > A.H) {  // (the host sizes H by the same count)
            if (t == 0) A.ctl->stuck = 1;
            return;
        }
        if (rows > 0) {
            int at = cnt[t];
            for (int i = w0; i < w1; ++i)
                for (unsigned b = bits[i]; b; b &= b - 1) sList[at++] = 32 * i + __ffs(b) - 1;
        }
        __syncthreads();
        auto find = [&](int c) {  // position of block column c in the (ascending) list
            int lo = 0, hi = sHaloN - 1;
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (sList[mid] < c) lo = mid + 1;
                else hi = mid;
            }
            return lo;
        };
        for (int i = t; i < S * Rp; i += kResT) {
            const int r = i % Rp;
            sCol[i] = r < rows ? (unsigned short)find(A.op.col[(size_t)(i / Rp) * A.op.ld + row0 + r]) : 0;
        }
        if (A.op.penPtr && rows > 0)
            for (int q = A.op.penPtr[row0] + t; q < A.op.penPtr[row0 + rows]; q += kResT)
                A.penLoc[q] = DPN * find(A.op.penCol[q] / DPN) + A.op.penCol[q] % DPN;
        __syncthreads();
        if constexpr (POLY) {
            for (int i = t; i < S * BvShape<DPN>::NV * Rp; i += kResT) {
                const int r = i % Rp, sp = i / Rp;
                sKv[i] = r < rows ? __ldg(A.hop.Kv + (size_t)sp * A.op.ld + row0 + r) : make_uint4(0, 0, 0, 0);
            }
            using RT_ = typename BvRem<BvShape<DPN>::REM>::T;
            const RT_ *kr = static_cast<const RT_ *>(A.hop.Kr);
            for (int i = t; i < S * Rp; i += kResT) {
                const int r = i % Rp;
                RT_ v = RT_();
                if (r < rows) v = __ldg(kr + (size_t)(i / Rp) * A.op.ld + row0 + r);
                reinterpret_cast<RT_ *>(sKr)[i] = v;
            }
        } else {
            for (int i = t; i < S * DD * Rp; i += kResT) {
                const int r = i % Rp;
                sK[i] = r < rows ? __ldg(A.op.K + (size_t)(i / Rp) * A.op.ld + row0 + r) : TM(0);
            }
        }
        __syncthreads();
    }
    const int halo = sHaloN;

    // the halo of a vector written by all CTAs before the last barrier
    auto gather = [&](const TV *v) {
        for (int i = t; i < halo * DPN; i += kResT) sHalo[i] = __ldcg(v + (size_t)sList[i / DPN] * DPN + i % DPN);
        __syncthreads();
    };
    // sy = (A halo)_own in the precision of the basis; the values from shared memory or, beside the
    // hops' planes, from L2.  SG (1, 2 or 4) threads per (row, component), the penalty by the first; one
    // thread adds in the order of the residual kernel.
    const int W = (Rp * DPN + 31) / 32 * 32, stepSG = 4 * W <= kResT ? 4 : (2 * W <= kResT ? 2 : 1);
    auto product = [&](const int SG) {
        const int per = kResT / SG, grp = t / per, tt = t % per;
        for (int i0 = 0; i0 < Rp * DPN; i0 += per) {
            const int i = i0 + tt, r = i % Rp, c = i / Rp;
            TV a = TV(0);
            const bool in = i < Rp * DPN && r < rows;
            if (in) {
#pragma unroll 4
                for (int s = grp; s < S; s += SG) {
                    const TV *xv = sHalo + DPN * sCol[s * Rp + r];
#pragma unroll
                    for (int jj = 0; jj < DPN; ++jj) {
                        TM k;
                        if constexpr (POLY) k = __ldg(A.op.K + (size_t)(s * DD + c * DPN + jj) * A.op.ld + row0 + r);
                        else k = sK[(size_t)(s * DD + c * DPN + jj) * Rp + r];
                        a += (TV)k * xv[jj];
                    }
                }
                if (grp == 0 && A.op.penPtr)
                    for (int q = A.op.penPtr[row0 + r]; q < A.op.penPtr[row0 + r + 1]; ++q)
                        if (A.op.penRow[q] == c) a += (TV)(A.op.penVal[q] * (double)sHalo[A.penLoc[q]]);
                sy[(size_t)grp * Rp * DPN + r * DPN + c] = a;
            }
            __syncthreads();
            if (in && grp == 0 && SG > 1) {
                for (int g = 1; g < SG; ++g) a += sy[(size_t)g * Rp * DPN + r * DPN + c];
                sy[r * DPN + c] = a;
            }
        }
        __syncthreads();
    };
    // CTA sum of a double per thread (every thread gets it)
    auto cta_sum = [&](double v) {
        v = warp_sum(v);
        if (lane == 0) red[wid] = v;
        __syncthreads();
        double a = 0.0;
        if (wid == 0) {
            a = warp_sum(red[lane]);
            if (lane == 0) red[0] = a;
        }
        __syncthreads();
        a = red[0];
        __syncthreads();
        return a;
    };
    double *partH = A.part, *partH2 = partH + (size_t)(kMaxM + 2) * A.G, *partN = partH2 + (size_t)(kMaxM + 2) * A.G;
    // sum over the CTAs of one partial each, by a warp
    auto total_norm = [&]() {
        double a = 0.0;
        for (int q0 = lane; q0 < A.G; q0 += 256) {
            double v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = q0 + 32 * u < A.G ? __ldcg(partN + q0 + 32 * u) : 0.0;
            a += ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
        }
        return warp_sum(a);
    };
    // partial dots of sw with V[0 .. j] (and, self, with itself as number j + 1).  LPV lanes a vector: the
    // FP64 pipe pays for every addition of a lane tree, FP32 rather wants the loads spread
    constexpr int LPV = sizeof(TV) == 8 ? 8 : 32, VPW = 32 / LPV;
    auto dots = [&](int j, bool self, double *part) {
        const int nv = j + 1 + (self ? 1 : 0), l = lane % LPV;
        for (int k0 = VPW * wid; k0 < nv; k0 += VPW * kResW) {
            const int k = k0 + lane / LPV;
            TV a = TV(0);
            if (k < nv) {
                const TV *v = k <= j ? V + (size_t)k * vld : sw;
                int i = l;
                for (; i + 3 * LPV < nown; i += 4 * LPV) {
                    const TV v0 = v[i], v1 = v[i + LPV], v2 = v[i + 2 * LPV], v3 = v[i + 3 * LPV];
                    a = fma(v0, sw[i], a);
                    a = fma(v1, sw[i + LPV], a);
                    a = fma(v2, sw[i + 2 * LPV], a);
                    a = fma(v3, sw[i + 3 * LPV], a);
                }
                for (; i < nown; i += LPV) a = fma(v[i], sw[i], a);
            }
#pragma unroll
            for (int o = LPV / 2; o; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
            if (l == 0 && k < nv) part[(size_t)k * A.G + blockIdx.x] = (double)a;
        }
    };
    // sh[0 .. nv-1] = sums over the CTAs
    auto totals = [&](int nv, const double *part) {
        const int l8 = lane & 7;
        for (int k0 = 4 * wid; k0 < nv; k0 += 4 * kResW) {
            const int k = k0 + lane / 8;
            double a = 0.0, c = 0.0;
            if (k < nv)
                for (int q0 = l8; q0 < A.G; q0 += 80) {
                    double v[10];
#pragma unroll
                    for (int u = 0; u < 10; ++u) v[u] = q0 + 8 * u < A.G ? __ldcg(part + (size_t)k * A.G + q0 + 8 * u) : 0.0;
#pragma unroll
                    for (int u = 0; u < 10; u += 2) {
                        a += v[u];
                        c += v[u + 1];
                    }
                }
            a += c;
#pragma unroll
            for (int o = 4; o; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
            if (l8 == 0 && k < nv) sh[k] = a;
        }
        __syncthreads();
    };
    // The hops of the preconditioner on y0 = zin (in z[0] behind a barrier); leaves P v in z[zi] behind a
    // barrier and returns zi (-1: given up).  A row's four lanes are the same in every hop, so lane 0 keeps
    // the row's recurrence in registers.
    auto hops = [&]() -> int {
        const int sub = wid % 4, r = (wid / 4) * 32 + lane, g = row0 + r;
        const bool own = r < rows, fin = own && sub == 0;
        TV yc[DPN], yp[DPN], sc[DPN], za[DPN];
#pragma unroll
        for (int q = 0; q < DPN; ++q) {
            yc[q] = fin ? __ldcg(A.z[0] + (size_t)g * DPN + q) : TV(0);
            sc[q] = fin ? A.y0s[(size_t)g * DPN + q] : TV(0);
            yp[q] = za[q] = TV(0);
        }
        const TV dinvC = TV(1) / (TV)A.delta;
        TV *sp = sy;  // [3][Rp][DPN]: the partial products of lanes 1 .. 3
        for (int k = 0; k < A.deg; ++k) {
            gather(A.z[k & 1]);
            TV a[DPN];
#pragma unroll
            for (int q = 0; q < DPN; ++q) a[q] = TV(0);
            if (own) {
                for (int s = sub; s < S; s += 4) {
                    float kv[DD];
#pragma unroll
                    for (int p = 0; p < BvShape<DPN>::NV; ++p) {
                        const uint4 u = sKv[(size_t)(s * BvShape<DPN>::NV + p) * Rp + r];
                        const unsigned w4[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&w4[e]));
                            kv[8 * p + 2 * e] = f.x;
                            kv[8 * p + 2 * e + 1] = f.y;
                        }
                    }
                    if constexpr (BvShape<DPN>::REM == 1) {
                        kv[8 * BvShape<DPN>::NV] = h2f_bits(sKr[s * Rp + r]);
                    } else {
                        const uint2 u = reinterpret_cast<const uint2 *>(sKr)[s * Rp + r];
                        const float2 f0 = __half22float2(*reinterpret_cast<const __half2 *>(&u.x)),
                                     f1 = __half22float2(*reinterpret_cast<const __half2 *>(&u.y));
                        kv[8 * BvShape<DPN>::NV] = f0.x;
                        kv[8 * BvShape<DPN>::NV + 1] = f0.y;
                        kv[8 * BvShape<DPN>::NV + 2] = f1.x;
                        kv[8 * BvShape<DPN>::NV + 3] = f1.y;
                    }
                    const TV *xv = sHalo + DPN * sCol[s * Rp + r];
#pragma unroll
                    for (int i = 0; i < DPN; ++i)
#pragma unroll
                        for (int jj = 0; jj < DPN; ++jj) a[i] += (TV)kv[i * DPN + jj] * xv[jj];
                }
                if (sub == 0 && A.hop.penPtr)
                    for (int q = A.hop.penPtr[g]; q < A.hop.penPtr[g + 1]; ++q) {
                        const TV pv = (TV)(A.hop.penVal[q] * (double)sHalo[A.penLoc[q]]);
#pragma unroll
                        for (int i = 0; i < DPN; ++i) a[i] += i == A.hop.penRow[q] ? pv : TV(0);
                    }
            }
            if (own && sub)
#pragma unroll
                for (int q = 0; q < DPN; ++q) sp[((size_t)(sub - 1) * Rp + r) * DPN + q] = a[q];
            __syncthreads();
            const bool last = k + 1 == A.deg;
            if (fin) {
#pragma unroll
                for (int u = 0; u < 3; ++u)
#pragma unroll
                    for (int q = 0; q < DPN; ++q) a[q] += sp[((size_t)u * Rp + r) * DPN + q];
                const TV c = (k == 0 ? TV(1) : TV(2)) * dinvC;
                TV yn[DPN];
#pragma unroll
                for (int q = 0; q < DPN; ++q) {
                    yn[q] = c * (a[q] - (TV)A.theta * yc[q]);
                    if (k) yn[q] -= yp[q];
                }
                if (k == 0) {
                    const TV a0 = A.amod ? (TV)A.amod[g] : TV(1);
#pragma unroll
                    for (int q = 0; q < DPN; ++q) {
                        TV z0 = TV(0);
#pragma unroll
                        for (int jj = 0; jj < DPN; ++jj) z0 += (TV)__ldg(A.W + q * DPN + jj) * (sc[jj] * yc[jj]);
                        za[q] = a0 * z0;
                    }
                }
                const TV a1 = A.amod ? (TV)A.amod[(size_t)(k + 1) * A.N + g] : TV(1);
                const float *Wk = A.W + (size_t)(k + 1) * DD;
#pragma unroll
                for (int q = 0; q < DPN; ++q) {
                    TV z1 = TV(0);
#pragma unroll
                    for (int jj = 0; jj < DPN; ++jj) z1 += (TV)__ldg(Wk + q * DPN + jj) * (sc[jj] * yn[jj]);
                    za[q] += a1 * z1;
                    yp[q] = yc[q];
                    yc[q] = yn[q];
                    A.z[(k + 1) & 1][(size_t)g * DPN + q] = last ? za[q] : yn[q];
                }
            }
            res_arrive(A.bar);
            if (!res_wait(A.bar, ++phase, A.ctl)) return -1;
        }
        return A.deg & 1;
    };

    // ---- r = b - A x (products in FP64, every row's sum in the order of the residual kernel: a cycle that
    // starts below the target by its own rounding, but not by the solver's check, would never move x), beta
    {
        double rr = 0.0;
        if constexpr (sizeof(TV) == 8) {
            gather(A.x);
            product(1);
            for (int i = t; i < nown; i += kResT) {
                const size_t g = (size_t)row0 * DPN + i;
                const double v = A.b[g] - sy[i];
                sw[i] = v;
                A.z[0][g] = A.y0s[g] * v;
                rr += v * v;
            }
        } else {
            for (int i = t; i < nown; i += kResT) {
                const int r = i % rows, c = i / rows, g = row0 + r;
                double a = 0.0;
                for (int s = 0; s < S; ++s) {
                    const TV *xv = A.x + (size_t)A.op.col[(size_t)s * A.op.ld + g] * DPN;
#pragma unroll
                    for (int jj = 0; jj < DPN; ++jj)
                        a += (double)__ldg(A.op.K + (size_t)(s * DD + c * DPN + jj) * A.op.ld + g) * (double)__ldcg(xv + jj);
                }
                if (A.op.penPtr)
                    for (int q = A.op.penPtr[g]; q < A.op.penPtr[g + 1]; ++q)
                        if (A.op.penRow[q] == c) a += A.op.penVal[q] * (double)__ldcg(A.x + A.op.penCol[q]);
                const double v = A.b[(size_t)g * DPN + c] - a;
                const TV rv = (TV)v;
                sw[r * DPN + c] = rv;
                A.z[0][(size_t)g * DPN + c] = A.y0s[(size_t)g * DPN + c] * rv;
                rr += v * v;
            }
        }
        rr = cta_sum(rr);
        if (t == 0) partN[blockIdx.x] = rr;
        RES_BARRIER();
        if (wid == 0) {
            const double beta = sqrt(total_norm());
            if (lane == 0) {
                sDone = beta <= *A.target || beta == 0.0 || !isfinite(beta);
                sBad = !isfinite(beta);
                sBreak = 0;
                sInv = beta > 0.0 ? 1.0 / beta : 0.0;
                sg[0] = beta;
            }
        }
        __syncthreads();
    }
    int j = 0, reorths = 0;
    for (;;) {
        // w = A (P or D^-1) v_j, v_j = sw * inv; the product's input is in z[0].  Without hops the control
        // of the step before runs beside the gather
        if constexpr (POLY) {
            if (sDone) break;
            const int zi = hops();
            if (zi < 0) return;
            gather(A.z[zi]);
        } else {
            gather(A.z[0]);
            if (sDone) break;
        }
        product(stepSG);
        {
            const TV inv = (TV)sInv;
            for (int i = t; i < nown; i += kResT) {
                V[(size_t)j * vld + i] = sw[i] * inv;
                sw[i] = sy[i] * inv;
            }
        }
        __syncthreads();
        dots(j, true, partH);
        RES_BARRIER();
        totals(j + 2, partH);
        double *Hc = Hs + (size_t)j * (m + 1);
        if (wid == 0) {
            double hh = 0.0;
            for (int k = lane; k <= j; k += 32) {
                hh += sh[k] * sh[k];
                Hc[k] = sh[k];
            }
            hh = warp_sum(hh);
            if (lane == 0) sReorth = sh[j + 1] - hh < 0.5 * sh[j + 1];
        }
        __syncthreads();
        auto subtract = [&]() {
            for (int i = t; i < nown; i += kResT) {
                TV a = sw[i];
                int k = 0;
                for (; k + 8 <= j + 1; k += 8) {
                    TV v[8];
#pragma unroll
                    for (int u = 0; u < 8; ++u) v[u] = V[(size_t)(k + u) * vld + i];
#pragma unroll
                    for (int u = 0; u < 8; ++u) a -= (TV)sh[k + u] * v[u];
                }
                for (; k <= j; ++k) a -= (TV)sh[k] * V[(size_t)k * vld + i];
                sw[i] = a;
            }
        };
        subtract();
        if (sReorth) {
            ++reorths;
            __syncthreads();
            dots(j, false, partH2);
            RES_BARRIER();
            totals(j + 1, partH2);
            for (int k = t; k <= j; k += kResT) Hc[k] += sh[k];
            subtract();
        }
        // ||w||^2 and the next product's input (each thread's own entries of sw)
        double nn = 0.0;
        for (int i = t; i < nown; i += kResT) {
            const TV a = sw[i];
            nn += (double)a * (double)a;
            A.z[0][(size_t)row0 * DPN + i] = A.y0s[(size_t)row0 * DPN + i] * a;
        }
        nn = cta_sum(nn);
        if (t == 0) partN[blockIdx.x] = nn;
        res_arrive(A.bar);
        // the earlier rotations of the column beside the wait: sequential in the carried entry alone
        if (wid == kResW - 1) {
            double s2[2], c2[2], h2[2], t2[2], ak[2] = {0.0, 0.0}, a = Hc[0];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int k = lane + 32 * u;
                s2[u] = k < j ? ssn[k] : 0.0;
                c2[u] = k < j ? scs[k] : 0.0;
                h2[u] = k < j ? Hc[k + 1] : 0.0;
                t2[u] = c2[u] * h2[u];
            }
            __syncwarp();
#pragma unroll
            for (int u = 0; u < 2; ++u)
                for (int k = 0; k < 32 && k + 32 * u < j; ++k) {
                    if (lane == k) ak[u] = a;
                    a = fma(-__shfl_sync(0xffffffffu, s2[u], k), a, __shfl_sync(0xffffffffu, t2[u], k));
                }
#pragma unroll
            for (int u = 0; u < 2; ++u)
                if (lane + 32 * u < j) Hc[lane + 32 * u] = c2[u] * ak[u] + s2[u] * h2[u];
            if (lane == 0) sHrot = a;
        }
        if (!res_wait(A.bar, ++phase, A.ctl)) return;
        if (wid == kResW - 1) {
            const double nrm = sqrt(total_norm());
            if (lane == 0) {
                const double a = sHrot, rr = hypot(a, nrm);
                double c = 1.0, sn = 0.0;
                if (rr > 0.0) {
                    c = a / rr;
                    sn = nrm / rr;
                }
                scs[j] = c;
                ssn[j] = sn;
                Hc[j] = rr;
                const double gj = sg[j];
                sg[j] = c * gj;
                sg[j + 1] = -sn * gj;
                int done = fabs(sg[j + 1]) <= *A.target || j + 1 >= m;
                if (!isfinite(nrm) || !isfinite(rr)) {
                    sBad = 1;
                    done = 1;
                } else if (!(nrm > 1e-300)) {
                    sBreak = 1;
                    done = 1;
                }
                sDone = done;
            }
        } else if (wid == kResW - 2) {
            const double s2 = total_norm();
            if (lane == 0) sInv = s2 > 0.0 ? 1.0 / sqrt(s2) : 0.0;
        }
        ++j;
        if constexpr (POLY) __syncthreads();
    }
    // ---- least squares and the update of x --------------------------------------------------------------
    if (wid == 0) {
        double g[2], d[2], rc[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int i = lane + 32 * u;
            g[u] = i < j ? sg[i] : 0.0;
            d[u] = i < j ? Hs[(size_t)i * (m + 1) + i] : 1.0;
            rc[u] = 1.0 / d[u];
        }
#pragma unroll
        for (int v = 1; v >= 0; --v)
            for (int k = min(31, j - 1 - 32 * v); k >= 0; --k) {
                const int col = 32 * v + k;
                const double q0 = g[v] * rc[v], y = __shfl_sync(0xffffffffu, fma(fma(-d[v], q0, g[v]), rc[v], q0), k);
                if (lane == k) sky[col] = y;
#pragma unroll
                for (int u = 0; u < 2; ++u)
                    if (u <= v && lane + 32 * u < col) g[u] = fma(-Hs[(size_t)col * (m + 1) + lane + 32 * u], y, g[u]);
            }
    }
    __syncthreads();
    for (int i = t; i < nown; i += kResT) {
        TV a = TV(0);
        int k = 0;
        for (; k + 8 <= j; k += 8) {
            TV v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = V[(size_t)(k + u) * vld + i];
#pragma unroll
            for (int u = 0; u < 8; ++u) a += (TV)sky[k + u] * v[u];
        }
        for (; k < j; ++k) a += (TV)sky[k] * V[(size_t)k * vld + i];
        const size_t g = (size_t)row0 * DPN + i;
        a *= A.y0s[g];
        if constexpr (POLY) A.z[0][g] = a;
        else A.x[g] += a;
    }
    if constexpr (POLY) {
        if (j > 0) {
            RES_BARRIER();
            const int zi = hops();
            if (zi < 0) return;
            for (int i = t; i < nown; i += kResT) {
                const size_t g = (size_t)row0 * DPN + i;
                A.x[g] += __ldcg(A.z[zi] + g);
            }
        }
    }
    if (blockIdx.x == 0 && t == 0) {
        A.ctl->resest = fabs(sg[j]);
        A.ctl->j = j;
        A.ctl->done = sDone;
        A.ctl->breakdown = sBreak;
        A.ctl->nonfinite = sBad;
        A.ctl->reorths = reorths;
    }
#undef RES_BARRIER
}

}  // namespace astro_kry
