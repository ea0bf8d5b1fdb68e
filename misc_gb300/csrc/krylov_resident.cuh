// A restart cycle of GMRES as one cooperative launch, for operators that fit the SMs' shared memory.
//
// The graph of krylov.cu spends 4 launches on an Arnoldi step and one on every hop of the polynomial
// preconditioner, and on models of up to 100,000 DOF or so each of them is a chain of latencies (launch,
// loads of the operator from L2, a last CTA that adds partial sums): 38 us a step in FP64 on 14,112
// rows, 8 us a hop on 91,875.  Here one CTA per SM owns R consecutive block rows for the whole cycle:
//   * their part of the operator (FP64 or FP32 values, or the FP16 planes of the hops), and in FP64
//     where it fits also of the Krylov basis, stays in shared memory;
//   * what a product needs of other CTAs' rows, the halo, is gathered from global memory (L2) into
//     shared memory once per product, and the columns are kept as 16-bit positions in it;
//   * CTAs exchange 16-byte words of values and a number that says which exchange they belong to, stored and
//     loaded whole: a reader polls the words that it needs, so that there is no barrier, no fence and no
//     separate flag (hops behind a flag per CTA: 9,200 clocks, 3,300 of them the flag's; behind a grid
//     barrier 11,000);
//   * a dot product's partial sums go to one CTA, which adds them in a fixed order and hands the total to
//     all (each CTA adding the 152 partials of 26 vectors by itself took the FP64 pipe 1.6 us a pass).
// The arithmetic is that of the graph's kernels (same precisions, classical Gram-Schmidt, Givens
// rotations) but for the order of the sums and one point: the second Gram-Schmidt pass always runs (the
// graph's test asks for it in 49 steps of 50), and its dot products include ||w||^2, so that the norm
// behind it is ||w||^2 - ||h||^2 with little to cancel and needs no exchange of its own.  Where more than
// half cancels, w was numerically in the space: the cycle ends with that column.
// What bounds it: in FP64 the pipe (1.66 lanes a clock and SM: products 2.4 us, Gram-Schmidt 3.2 us a step
// at 31 rows a CTA), then the exchanges (0.7 us each); in the hops shared-memory loads and the exchange.
// 4,704 nodes in FP64: a step 38 us in the graph, 12.8 us here; 30,625 nodes: a hop 8.0 us there, 2.7 here.
//
// An exchange's words may be overwritten by the one after the next: a CTA writes exchange x + 1 when it
// has read x from the owners of its halo, who wrote x after they had read x - 1.  The owners of a CTA's halo
// are also those who read its rows: the pattern is symmetric.  The launch is cooperative, so all CTAs are
// resident, and every poll is bounded: past the limit the CTA sets ctl->stuck and returns, as the others
// then do; the host takes the solve on in the graph's form (x is then a part of the way, which a cycle may start from).
#pragma once
#include "krylov_ops.cuh"

namespace astro_kry {

constexpr int kResT = 1024, kResW = kResT / 32;
constexpr int kSpinLimit = 1 << 21;  // polls of a word (more than a second), unless ASTRO_OPT_POLL_LIMIT says else
constexpr int kResMaxRows = 256;     // rows of a CTA in the hops: a warp takes eight, four lanes each
constexpr int kResMaxCtas = 160;

template <class TM, class TV> struct ResArgs {
    Op<TM> op;
    OpH hop;              // polynomial preconditioner (its values), or unused
    int deg;              // hops, 0 = Jacobi
    float theta, delta;   // the map of the recurrence
    int power;            // power iterations of the hops' operator instead of a cycle; the norm to ctl->y[0]
    const float *W;       // hop weights, (deg + 1) x dpn x dpn, already divided by lambda
    const float *amod;    // per-node hop scales, or null
    const TV *y0s;        // scales a residual into the preconditioner's input
    TV *x;
    const double *b;
    TV *V;                // Krylov basis, vector-major (used when it does not fit shared memory)
    size_t ld;
    ulonglong2 *words;    // exchanged words, all 0 at launch: res_words()
    GmresCtl *ctl;
    const double *target;
    int m, N, R, G, H, P; // H, P: capacity of the halo and of a CTA's penalty entries
    int vShared;
    int polls;            // limit of a wait
};

struct ResLayout {
    size_t k, kr, col, list, halo, own, hes, w, pptr, pinfo, pval, v, total;
};
// Row stride of a CTA's operator.  In the hops a warp reads eight rows of four slots: 8 mod 16, so that the
// four do not share banks.
__host__ __device__ constexpr int res_rows(int R, int deg) { return deg ? (R + 7) / 16 * 16 + 8 : (R + 3) / 4 * 4; }
// Words of a node in an exchange: three floats and the number, or one double and the number.
template <class TV, int DPN> __host__ __device__ constexpr int res_node_words() { return sizeof(TV) == 8 ? DPN : DPN / 3; }
// Words in all: two exchanges of a vector, the partial sums of two passes and every CTA's copy of the totals.
template <class TV, int DPN> __host__ __device__ constexpr size_t res_words(int N, int G) {
    return 2 * (size_t)N * res_node_words<TV, DPN>() + 4 * (size_t)(kMaxM + 2) * G;
}
// Components of a node in the halo: a float4 for three floats (one 16-byte load instead of three).
template <class TV, int DPN> __host__ __device__ constexpr int res_hs() { return sizeof(TV) == 4 && DPN == 3 ? 4 : DPN; }
// Byte offsets of the CTA's arrays in dynamic shared memory.  deg > 0: the hops' FP16 planes instead of the
// values of op.
template <class TM, class TV, int DPN>
__host__ __device__ inline ResLayout res_layout(int N, int S, int R, int H, int P, int m, int deg, int vShared) {
    const size_t rows = res_rows(R, deg);
    ResLayout L;
    size_t o = 0;
    auto put = [&](size_t bytes) {
        const size_t at = o;
        o += (bytes + 15) / 16 * 16;
        return at;
    };
    const size_t k = deg ? sizeof(uint4) * BvShape<DPN>::NV * S * rows : sizeof(TM) * (size_t)(DPN * DPN) * S * rows;
    const size_t marks = ((size_t)N + 3) / 4 * 4;  // of the halo, before the values are loaded
    L.k = put(k > marks ? k : marks);
    // hops, 3 DOF: the block's ninth value beside the column in one word; 6 DOF: the last four values
    L.kr = put(deg && DPN != 3 ? sizeof(uint2) * S * rows : 0);
    L.col = put((deg && DPN == 3 ? sizeof(unsigned) : sizeof(unsigned short)) * S * rows);
    L.list = put(sizeof(int) * (size_t)H);
    L.halo = put(sizeof(TV) * (size_t)H * res_hs<TV, DPN>());
    L.own = put(sizeof(TV) * 5 * rows * DPN);  // w and the products of up to four threads an entry
    L.hes = put(sizeof(double) * (size_t)(m + 1) * m);
    L.w = put(sizeof(float) * (size_t)(deg + 1) * DPN * DPN);
    L.pptr = put(P ? sizeof(int) * ((size_t)R + 1) : 0);
    L.pinfo = put(sizeof(int) * (size_t)P);
    L.pval = put(sizeof(double) * (size_t)(deg ? 2 * P : P));  // hops: the matrix' own behind the scaled
    L.v = put(vShared ? sizeof(TV) * (size_t)(m + 1) * R * DPN : 0);
    L.total = o;
    return L;
}

// Marks the block columns of a CTA's rows (and of their penalty entries) in a byte each of `words` words.
// Used by the count kernel and by the cycle itself.  (Bits set by atomics: neighbouring rows' columns share
// words, and marking alone took 50,000 clocks of a cycle.)
template <class TM>
__device__ void res_mark(const Op<TM> &op, int row0, int rows, unsigned *marks, int words) {
    unsigned char *mk = reinterpret_cast<unsigned char *>(marks);
    for (int i = threadIdx.x; i < words; i += blockDim.x) marks[i] = 0u;
    __syncthreads();
    for (int i = threadIdx.x; i < rows * op.S; i += blockDim.x) mk[op.col[(size_t)(i / rows) * op.ld + row0 + i % rows]] = 1;
    if (op.penPtr)
        for (int t = op.penPtr[row0] + threadIdx.x; t < op.penPtr[row0 + rows]; t += blockDim.x) mk[op.penCol[t] / op.dpn] = 1;
    __syncthreads();
}

// The block columns of a CTA's rows, ascending, into list (kResT threads; marks: a byte per column of scratch);
// their number, at most H of which are written.
template <class TM>
__device__ int res_list(const Op<TM> &op, int row0, int rows, int H, unsigned *marks, int *list) {
    __shared__ int cnt[kResT + 1];
    const int t = threadIdx.x, words = (op.N + 3) / 4;
    if (rows > 0) res_mark(op, row0, rows, marks, words);
    const int per = (words + kResT - 1) / kResT, w0 = min(words, t * per), w1 = min(words, w0 + per);
    int c = 0;
    if (rows > 0)
        for (int i = w0; i < w1; ++i) c += __popc(marks[i]);
    cnt[t + 1] = c;
    if (t == 0) cnt[0] = 0;
    __syncthreads();
    for (int o = 1; o < kResT; o *= 2) {  // inclusive scan of cnt[1 ..]
        const int v = t + 1 > o ? cnt[t + 1 - o] : 0;
        __syncthreads();
        cnt[t + 1] += v;
        __syncthreads();
    }
    if (rows > 0 && cnt[kResT] <= H) {
        int at = cnt[t];
        for (int i = w0; i < w1; ++i)
            for (unsigned b = marks[i]; b; b &= b - 1) list[at++] = 4 * i + (__ffs(b) - 1) / 8;
    }
    __syncthreads();
    return cnt[kResT];
}
// Position of column c in the list.
__device__ __forceinline__ int res_find(const int *list, int n, int c) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (list[mid] < c) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// Largest halo (most[0]) and number of penalty entries (most[1]) of a CTA.
template <class TM> __global__ void k_res_halo(Op<TM> op, int R, int *most) {
    extern __shared__ unsigned marks[];
    const int row0 = blockIdx.x * R, rows = min(R, op.N - row0), words = (op.N + 3) / 4;
    if (rows <= 0) return;
    res_mark(op, row0, rows, marks, words);
    int c = 0;
    for (int i = threadIdx.x; i < words; i += blockDim.x) c += __popc(marks[i]);
    for (int o = 16; o; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    __shared__ int total;
    if (threadIdx.x == 0) total = 0;
    __syncthreads();
    if ((threadIdx.x & 31) == 0) atomicAdd(&total, c);
    __syncthreads();
    if (threadIdx.x == 0) {
        atomicMax(most, total);
        if (op.penPtr) atomicMax(most + 1, op.penPtr[row0 + rows] - op.penPtr[row0]);
    }
}

__device__ __forceinline__ void word_put(ulonglong2 *p, unsigned long long a, unsigned long long b) {
    asm volatile("{\n\t.reg .b128 w;\n\tmov.b128 w, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], w;\n\t}" ::"l"(p), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ ulonglong2 word_get(const ulonglong2 *p) {
    ulonglong2 v;
    asm volatile("{\n\t.reg .b128 w;\n\tld.relaxed.gpu.global.b128 w, [%2];\n\tmov.b128 {%0, %1}, w;\n\t}" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
    return v;
}
// One double, or three floats, and the exchange's number.
__device__ __forceinline__ void word_put(ulonglong2 *p, double v, unsigned no) {
    word_put(p, (unsigned long long)__double_as_longlong(v), (unsigned long long)no << 32);
}
__device__ __forceinline__ void word_put(ulonglong2 *p, float a, float b, float c, unsigned no) {
    word_put(p, (unsigned long long)__float_as_uint(b) << 32 | __float_as_uint(a), (unsigned long long)no << 32 | __float_as_uint(c));
}
__device__ __forceinline__ unsigned word_no(const ulonglong2 &v) { return (unsigned)(v.y >> 32); }

// A float as a double by integer instructions.  The conversion instruction runs at the rate of the FP64 pipe,
// of which the residual's two a product took two thirds.  Subnormals are shifted to a leading one, the
// exponent 255 becomes 2047.
__device__ __forceinline__ double widen(double v) { return v; }
__device__ __forceinline__ double widen(float v) {
    const unsigned u = __float_as_uint(v), m = u & 0x7fffffffu;
    const unsigned s = m < 0x800000u ? __clz((int)m) - 8 : 0, mm = m << s, e = (m >= 0x7f800000u ? 1792u : 896u) - s;
    return __hiloint2double((int)((u & 0x80000000u) | (m ? (mm >> 3) + (e << 20) : 0u)), (int)(mm << 29));
}

template <class TM, class TV, int DPN, bool POLY>
__global__ void __launch_bounds__(kResT, 1) k_gmres_resident(ResArgs<TM, TV> A) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int DD = DPN * DPN, HS = res_hs<TV, DPN>();
    // Without hops the last warp only does the control of the steps (rotations, residual estimate), which is
    // as long as the products: the others, the workers, meet at a barrier of their own.
    constexpr int kWT = POLY ? kResT : kResT - 32, kWW = kWT / 32;
    auto wsync = [] {
        if constexpr (POLY) __syncthreads();
        else asm volatile("bar.sync 1, %0;" ::"n"(kWT) : "memory");
    };
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
    const int row0 = blockIdx.x * A.R, rows = max(0, min(A.R, A.N - row0)), nown = rows * DPN;
    const int Rp = res_rows(A.R, POLY), S = A.op.S, m = A.m;
    const ResLayout L = res_layout<TM, TV, DPN>(A.N, S, A.R, A.H, A.P, m, POLY ? A.deg : 0, A.vShared);
    TM *sK = reinterpret_cast<TM *>(smem + L.k);
    uint4 *sKv = reinterpret_cast<uint4 *>(smem + L.k);
    uint2 *sKr = reinterpret_cast<uint2 *>(smem + L.kr);
    unsigned short *sCol = reinterpret_cast<unsigned short *>(smem + L.col);
    unsigned *sColH = reinterpret_cast<unsigned *>(smem + L.col);
    int *sList = reinterpret_cast<int *>(smem + L.list);
    TV *sHalo = reinterpret_cast<TV *>(smem + L.halo);
    TV *sw = reinterpret_cast<TV *>(smem + L.own), *sy = sw + Rp * DPN;
    double *Hs = reinterpret_cast<double *>(smem + L.hes);  // column j at Hs + j (m + 1)
    float *sW = reinterpret_cast<float *>(smem + L.w);
    // penalty entries by row: place of the column's value in the halo | component << 24, and values
    int *pPtr = reinterpret_cast<int *>(smem + L.pptr), *pInfo = reinterpret_cast<int *>(smem + L.pinfo);
    double *pVal = reinterpret_cast<double *>(smem + L.pval);
    const bool pen = A.op.penPtr && A.P > 0;
    const int pen0 = pen && rows > 0 ? A.op.penPtr[row0] : 0, nPen = pen && rows > 0 ? A.op.penPtr[row0 + rows] - pen0 : 0;
    TV *V = A.vShared ? reinterpret_cast<TV *>(smem + L.v) : A.V + (size_t)row0 * DPN;
    const size_t vld = A.vShared ? (size_t)A.R * DPN : A.ld;
    __shared__ double sh1[kMaxM + 2], sh2[kMaxM + 2], scs[kMaxM], ssn[kMaxM], sg[kMaxM + 1], red[kResW];
    __shared__ TV shT[kMaxM + 2], sInv;  // (conversions from FP64 run at its rate: once, not per thread)
    __shared__ int sDone, sHaloN, sBreak, sBad, sStuck;
    unsigned no = 0;  // vector exchanges so far: number no is in the words of vec(no)
    constexpr int NW = res_node_words<TV, DPN>();
    auto vec = [&](unsigned e) { return A.words + (size_t)(e & 1) * A.N * NW; };
    ulonglong2 *const part = A.words + 2 * (size_t)A.N * NW, *const total = part + 2 * (size_t)(kMaxM + 2) * A.G;

    // ---- the CTA's rows into shared memory: halo list, local columns, operator -----------------------
    {
        // marks of the halo in the (still unused) operator area
        const int n = res_list(A.op, row0, rows, A.H, reinterpret_cast<unsigned *>(smem + L.k), sList);
        if (t == 0) {
            sHaloN = n;
            sStuck = 0;
        }
        if (n > A.H || nPen > A.P) {  // (the host sizes both by the same counts)
            if (t == 0) A.ctl->stuck = 1;
            return;
        }
        __syncthreads();
        auto find = [&](int c) { return res_find(sList, sHaloN, c); };
        for (int i = t; i < S * Rp; i += kResT) {
            const int r = i % Rp, c = r < rows ? find(A.op.col[(size_t)(i / Rp) * A.op.ld + row0 + r]) : 0;
            if constexpr (POLY && DPN == 3) {
                const unsigned short *kr = static_cast<const unsigned short *>(A.hop.Kr);
                sColH[i] = c | (r < rows ? (unsigned)__ldg(kr + (size_t)(i / Rp) * A.op.ld + row0 + r) << 16 : 0u);
            } else {
                sCol[i] = (unsigned short)c;
            }
        }
        if (pen) {
            for (int i = t; i <= rows; i += kResT) pPtr[i] = A.op.penPtr[row0 + i] - pen0;
            for (int q = t; q < nPen; q += kResT) {
                const int c = A.op.penCol[pen0 + q];
                pInfo[q] = (HS * find(c / DPN) + c % DPN) | A.op.penRow[pen0 + q] << 24;
                // hops: as two floats, whose products with a float are added with one rounding to speak of (the
                // FP64 product rounded to a float in all but one of 60 million random pairs)
                const double v = POLY ? A.hop.penVal[pen0 + q] : A.op.penVal[pen0 + q];
                if constexpr (POLY) {
                    reinterpret_cast<float2 *>(pVal)[q] = make_float2((float)v, (float)(v - (double)(float)v));
                    pVal[A.P + q] = A.op.penVal[pen0 + q];
                }
                else pVal[q] = v;
            }
        }
        __syncthreads();
        if constexpr (POLY) {
            for (int i = t; i < S * BvShape<DPN>::NV * Rp; i += kResT) {
                const int r = i % Rp, sp = i / Rp;
                sKv[i] = r < rows ? __ldg(A.hop.Kv + (size_t)sp * A.op.ld + row0 + r) : make_uint4(0, 0, 0, 0);
            }
            if constexpr (DPN != 3) {
                const uint2 *kr = static_cast<const uint2 *>(A.hop.Kr);
                for (int i = t; i < S * Rp; i += kResT) {
                    const int r = i % Rp;
                    sKr[i] = r < rows ? __ldg(kr + (size_t)(i / Rp) * A.op.ld + row0 + r) : make_uint2(0, 0);
                }
            }
            for (int i = t; i < (A.deg + 1) * DD; i += kResT) sW[i] = A.W[i];
        } else {
            for (int i = t; i < S * DD * Rp; i += kResT) {
                const int r = i % Rp;
                sK[i] = r < rows ? __ldg(A.op.K + (size_t)(i / Rp) * A.op.ld + row0 + r) : TM(0);
            }
        }
        __syncthreads();
    }
    const int halo = sHaloN;

    // gives up: the control warp, waiting at the CTA's barrier, sees sStuck behind it
    auto give_up = [&] {
        if (t == 0) A.ctl->stuck = 1;
        if constexpr (!POLY) __syncthreads();
    };
    // entry i of the CTA's rows, or node row r, into exchange e (FP32: whole nodes)
    auto put_node = [&](unsigned e, int r, const TV *v) {
#pragma unroll
        for (int w = 0; w < NW; ++w) {
            ulonglong2 *p = vec(e) + (size_t)(row0 + r) * NW + w;
            if constexpr (sizeof(TV) == 8) word_put(p, v[w], e);
            else word_put(p, v[3 * w], v[3 * w + 1], v[3 * w + 2], e);
        }
    };
    // the halo of exchange e, polled word by word; false when one was given up
    auto gather = [&](unsigned e) {
        const ulonglong2 *v = vec(e);
        for (int i0 = t; i0 < halo * NW; i0 += 2 * kWT) {  // two words in flight
            ulonglong2 w[2];
            const ulonglong2 *p[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int i = min(i0 + u * kWT, halo * NW - 1);
                p[u] = v + (size_t)sList[i / NW] * NW + i % NW;
                w[u] = word_get(p[u]);
            }
            for (int it = 0; word_no(w[0]) != e || word_no(w[1]) != e;) {
                if (++it > A.polls) {
                    sStuck = 1;
                    break;
                }
                w[0] = word_get(p[0]);
                w[1] = word_get(p[1]);
            }
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int i = i0 + u * kWT;
                if (i >= halo * NW) break;
                if constexpr (sizeof(TV) == 8) {
                    sHalo[i] = __longlong_as_double((long long)w[u].x);
                } else {
                    TV *h = sHalo + (i / NW) * HS + 3 * (i % NW);
                    h[0] = __uint_as_float((unsigned)w[u].x);
                    h[1] = __uint_as_float((unsigned)(w[u].x >> 32));
                    h[2] = __uint_as_float((unsigned)w[u].y);
                }
            }
        }
        wsync();
        return sStuck == 0;
    };
    // Totals of nv partial sums, pass 0 or 1, tagged e: the partials of sum k go to CTA k mod G, one warp of
    // which adds them in a fixed order and writes the total to every CTA's own words (all polling the same
    // ones made their L2 slice the bottleneck); every CTA takes the totals to sh.
    auto put_part = [&](int pass, int k, double v, unsigned e) {
        word_put(part + ((size_t)pass * (kMaxM + 2) + k) * A.G + blockIdx.x, v, e);
    };
    auto totals = [&](int pass, int nv, unsigned e, double *sh) {
        // (the last warps: the first are busy with the dot products)
        for (int q = kWW - 1 - wid, k; (k = blockIdx.x + q * A.G) < nv; q += kWW) {
            constexpr int CN = kResMaxCtas / 32;
            const ulonglong2 *p = part + ((size_t)pass * (kMaxM + 2) + k) * A.G;
            ulonglong2 w[CN];
            bool all = false;
            for (int it = 0; !all && it < A.polls; ++it) {
                all = true;
#pragma unroll
                for (int u = 0; u < CN; ++u) w[u] = lane + 32 * u < A.G ? word_get(p + lane + 32 * u) : make_ulonglong2(0, (unsigned long long)e << 32);
#pragma unroll
                for (int u = 0; u < CN; ++u) all = all && word_no(w[u]) == e;
            }
            if (!all) sStuck = 1;
            double a = 0.0;
#pragma unroll
            for (int u = 0; u < CN; ++u) a += __longlong_as_double((long long)w[u].x);
            a = warp_sum(a);
#pragma unroll
            for (int u = 0; u < CN; ++u)
                if (lane + 32 * u < A.G) word_put(total + ((size_t)pass * A.G + lane + 32 * u) * (kMaxM + 2) + k, a, e);
        }
        for (int k = t; k < nv; k += kWT) {
            const ulonglong2 *p = total + ((size_t)pass * A.G + blockIdx.x) * (kMaxM + 2) + k;
            ulonglong2 w = word_get(p);
            for (int it = 0; word_no(w) != e; w = word_get(p))
                if (++it > A.polls) {
                    sStuck = 1;
                    break;
                }
            sh[k] = __longlong_as_double((long long)w.x);
            shT[k] = (TV)sh[k];
        }
    };
    // The products of the halo with the CTA's rows, added in TA: fin(i, a) with entry i = row DPN + component.
    // The values from shared memory or, beside the hops' planes, from L2.  SG (1, 2 or 4) threads per entry,
    // the penalty by the first; one thread adds in the order of the residual kernel.
    const int wEnt = (Rp * DPN + 31) / 32 * 32, stepSG = 4 * wEnt <= kWT ? 4 : (2 * wEnt <= kWT ? 2 : 1);
    auto product = [&](const int SG, auto zero, auto fin) {
        using TA = decltype(zero);
        const int per = kWT / SG / 32 * 32, grp = t / per, tt = t % per;  // whole warps
        for (int i0 = 0; i0 < Rp * DPN; i0 += per) {
            const int i = i0 + tt, r = i % Rp, c = i / Rp;
            TA a = zero;
            const bool in = i < Rp * DPN && r < rows && grp < SG;
            if (in) {
#pragma unroll(POLY ? 9 : 4)
                for (int s = grp; s < S; s += SG) {
                    int col;
                    if constexpr (POLY && DPN == 3) col = sColH[s * Rp + r] & 0xffff;
                    else col = sCol[s * Rp + r];
                    const TV *xv = sHalo + HS * col;
#pragma unroll
                    for (int jj = 0; jj < DPN; ++jj) {
                        TM k;
                        if constexpr (POLY) k = __ldg(A.op.K + (size_t)(s * DD + c * DPN + jj) * A.op.ld + row0 + r);
                        else k = sK[(s * DD + c * DPN + jj) * Rp + r];
                        if constexpr (sizeof(TA) == 8) a += widen(k) * widen(xv[jj]);
                        else a += (TA)k * (TA)xv[jj];
                    }
                }
                if (grp == 0 && pen)
                    for (int q = pPtr[r]; q < pPtr[r + 1]; ++q)
                        if (pInfo[q] >> 24 == c)
                            a += (TA)(pVal[POLY ? A.P + q : q] * (double)sHalo[pInfo[q] & 0xffffff]);
            }
            if (SG > 1) {
                if (in && grp) sy[(grp * Rp + r) * DPN + c] = (TV)a;
                wsync();
                if (in && !grp)
                    for (int g = 1; g < SG; ++g) a += (TA)sy[(g * Rp + r) * DPN + c];
            }
            if (in && !grp) fin(r * DPN + c, a);
            if (SG > 1 && i0 + per < Rp * DPN) wsync();
        }
    };
    // partial dots of sw with V[0 .. j] (and in pass 1 with itself as number j + 1), tagged j + 2.  LPV lanes a vector: the
    // FP64 pipe pays for every addition of a lane tree, FP32 rather wants the loads spread
    constexpr int LPV = sizeof(TV) == 8 ? 8 : 32, VPW = 32 / LPV;
    auto dots = [&](int j, int pass) {
        const int nv = j + 1 + pass, l = lane % LPV;
        for (int k0 = VPW * wid; k0 < nv; k0 += VPW * kWW) {
            const int k = k0 + lane / LPV;
            TV a = TV(0);
            if (k < nv) {
                const TV *v = k <= j ? V + (size_t)k * vld : sw;
                int i = l;
                for (; i + 3 * LPV < nown; i += 4 * LPV) {
                    TV b[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) b[u] = v[i + u * LPV];
#pragma unroll
                    for (int u = 0; u < 4; ++u) a = fma(b[u], sw[i + u * LPV], a);
                }
                if (i < nown) {
                    TV b[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) b[u] = i + u * LPV < nown ? v[i + u * LPV] : TV(0);
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (i + u * LPV < nown) a = fma(b[u], sw[i + u * LPV], a);
                }
            }
#pragma unroll
            for (int o = LPV / 2; o; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
            if (l == 0 && k < nv) put_part(pass, k, (double)a, j + 2);
        }
    };
    // w -= V h with the last totals
    auto subtract = [&](int j) {
        for (int i = t; i < nown; i += kWT) {
            TV a = sw[i];
            int k = 0;
            for (; k + 8 <= j + 1; k += 8) {
                TV v[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) v[u] = V[(size_t)(k + u) * vld + i];
#pragma unroll
                for (int u = 0; u < 8; ++u) a -= shT[k + u] * v[u];
            }
            TV v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = k + u <= j ? V[(size_t)(k + u) * vld + i] : TV(0);
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (k + u <= j) a -= shT[k + u] * v[u];
            sw[i] = a;
        }
    };
    // Control of step j by one warp: the column of H is h1 + h2, its earlier rotations (sequential in the
    // carried entry alone), the new one, the residual estimate and the stopping tests.
    auto control = [&](int j) {
        double *Hc = Hs + (size_t)j * (m + 1);
        double s2[2], c2[2], h2[2], t2[2], ak[2] = {0.0, 0.0}, hh = 0.0;
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int k = lane + 32 * u;
            const double g = k <= j ? sh2[k] : 0.0;
            hh = fma(g, g, hh);
            s2[u] = k < j ? ssn[k] : 0.0;
            c2[u] = k < j ? scs[k] : 0.0;
            h2[u] = k < j ? sh1[k + 1] + sh2[k + 1] : 0.0;
            t2[u] = c2[u] * h2[u];
        }
        double a = sh1[0] + sh2[0];
        const double ww = sh2[j + 1], nn = ww - warp_sum(hh), inv = nn > 0.0 ? rsqrt(nn) : 0.0;
        const double nrm = nn > 0.0 ? nn * inv : (nn <= 0.0 ? 0.0 : nn);
        if (lane == 0) sInv = (TV)inv;
#pragma unroll
        for (int u = 0; u < 2; ++u)
            for (int k = 0; k < 32 && k + 32 * u < j; ++k) {
                if (lane == k) ak[u] = a;
                a = fma(-__shfl_sync(0xffffffffu, s2[u], k), a, __shfl_sync(0xffffffffu, t2[u], k));
            }
#pragma unroll
        for (int u = 0; u < 2; ++u)
            if (lane + 32 * u < j) Hc[lane + 32 * u] = c2[u] * ak[u] + s2[u] * h2[u];
        if (lane == 0) {
            // (a division is 550 clocks, as is rsqrt)
            const double q = fma(a, a, fmax(nn, 0.0));
            double rr, c = 1.0, sn = 0.0;
            if (q > 1e-290 && q < 1e290) {
                const double r = rsqrt(q);
                rr = q * r;
                c = a * r;
                sn = nrm * r;
            } else {
                rr = hypot(a, nrm);
                if (rr > 0.0) {
                    c = a / rr;
                    sn = nrm / rr;
                }
            }
            scs[j] = c;
            ssn[j] = sn;
            Hc[j] = rr;
            const double gj = sg[j];
            sg[j] = c * gj;
            sg[j + 1] = -sn * gj;
            int done = fabs(sg[j + 1]) <= *A.target || j + 1 >= m || !(nn >= 0.5 * ww);
            if (!isfinite(nrm) || !isfinite(rr)) {
                sBad = 1;
                done = 1;
            } else if (!(nrm > 1e-300)) {
                sBreak = 1;
                done = 1;
            }
            sDone = done;
        }
        __syncwarp();
    };
    // The product of the hops' operator with the gathered halo: eight rows a warp, four lanes a row (the lane's
    // bits 3 and 4), each of which gets the row.
    auto hopProduct = [&](TV (&a)[DPN]) {
        constexpr int NL = 4;
        const int sub = lane >> 3, r = wid * 8 + (lane & 7);
        const bool own = r < rows;
        const int p0 = pen && own ? pPtr[r] + NL - 1 - sub : 0, p1 = pen && own ? pPtr[r + 1] : 0;
#pragma unroll
        for (int q = 0; q < DPN; ++q) a[q] = TV(0);
        if (own) {
#pragma unroll 2
            for (int s = sub; s < S; s += NL) {
                const int at = s * Rp + r;
                float kv[DD];
#pragma unroll
                for (int p = 0; p < BvShape<DPN>::NV; ++p) {
                    const uint4 u = sKv[(s * BvShape<DPN>::NV + p) * Rp + r];
                    const unsigned w4[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&w4[e]));
                        kv[8 * p + 2 * e] = f.x;
                        kv[8 * p + 2 * e + 1] = f.y;
                    }
                }
                TV xv[DPN];
                if constexpr (DPN == 3) {
                    const unsigned ch = sColH[at];
                    kv[8] = h2f_bits((unsigned short)(ch >> 16));
                    const float4 f = *reinterpret_cast<const float4 *>(sHalo + HS * (ch & 0xffff));
                    xv[0] = f.x;
                    xv[1] = f.y;
                    xv[2] = f.z;
                } else {
                    const uint2 u = sKr[at];
                    const float2 f0 = __half22float2(*reinterpret_cast<const __half2 *>(&u.x)),
                                 f1 = __half22float2(*reinterpret_cast<const __half2 *>(&u.y));
                    kv[DD - 4] = f0.x;
                    kv[DD - 3] = f0.y;
                    kv[DD - 2] = f1.x;
                    kv[DD - 1] = f1.y;
#pragma unroll
                    for (int jj = 0; jj < DPN; ++jj) xv[jj] = sHalo[HS * sCol[at] + jj];
                }
#pragma unroll
                for (int i = 0; i < DPN; ++i)
#pragma unroll
                    for (int jj = 0; jj < DPN; ++jj) a[i] += (TV)kv[i * DPN + jj] * xv[jj];
            }
            for (int q = p0; q < p1; q += NL) {  // (from the last lane: 27 slots are one fewer there)
                const float2 v = reinterpret_cast<const float2 *>(pVal)[q];
                const float x = (float)sHalo[pInfo[q] & 0xffffff];
                const TV pv = fmaf(v.x, x, v.y * x);
#pragma unroll
                for (int i = 0; i < DPN; ++i) a[i] += i == pInfo[q] >> 24 ? pv : TV(0);
            }
        }
#pragma unroll
        for (int o = 8; o < 32; o *= 2)
#pragma unroll
            for (int q = 0; q < DPN; ++q) a[q] += __shfl_xor_sync(0xffffffffu, a[q], o);
    };
    // The hops of the preconditioner on y0 = S sw (exchange no); P v goes into the next exchange or, upd, is
    // added to x.  False when a wait was given up.  The four lanes of a row each
    // have its recurrence; lane q < 3 of them collects components q, q + 3 of P v.
    auto hops = [&](const bool upd) -> bool {
        constexpr int NZ = DPN / 3;
        const int sub = lane >> 3, r = wid * 8 + (lane & 7), g = row0 + r;
        const bool own = r < rows;
        TV yc[DPN], yp[DPN], sc[DPN], za[NZ];
#pragma unroll
        for (int q = 0; q < DPN; ++q) {
            sc[q] = own ? A.y0s[(size_t)g * DPN + q] : TV(0);
            yc[q] = own ? sc[q] * sw[r * DPN + q] : TV(0);
            yp[q] = TV(0);
        }
#pragma unroll
        for (int z = 0; z < NZ; ++z) za[z] = TV(0);
        const TV dinvC = TV(1) / (TV)A.delta, theta = (TV)A.theta;
        // za += a_k W_k (s y)
        auto collect = [&](int k, const TV *y) {
            if (!own || sub > 2) return;
            const TV ak = A.amod ? (TV)A.amod[(size_t)k * A.N + g] : TV(1);
#pragma unroll
            for (int z = 0; z < NZ; ++z) {
                TV a = TV(0);
#pragma unroll
                for (int jj = 0; jj < DPN; ++jj) a += (TV)sW[k * DD + (sub + 3 * z) * DPN + jj] * (sc[jj] * y[jj]);
                za[z] += ak * a;
            }
        };
        for (int k = 0; k < A.deg; ++k) {
            if (!gather(no)) return false;
            TV a[DPN];
            hopProduct(a);
            const bool last = k + 1 == A.deg;
            const TV c = (k == 0 ? TV(1) : TV(2)) * dinvC;
#pragma unroll
            for (int q = 0; q < DPN; ++q) {  // (yp is 0 in the first hop)
                const TV yn = c * (a[q] - theta * yc[q]) - yp[q];
                yp[q] = yc[q];
                yc[q] = yn;
            }
            ++no;
            if (!last && own && sub == 0) put_node(no, r, yc);
            // (what the hop adds to P v, while its words travel)
            if (k == 0) collect(0, yp);
            collect(k + 1, yc);
            if (last && upd) {
                if (own && sub < 3)
#pragma unroll
                    for (int z = 0; z < NZ; ++z) A.x[(size_t)g * DPN + sub + 3 * z] += za[z];
            } else if (last) {
                TV v[DPN];
#pragma unroll
                for (int q = 0; q < DPN; ++q) v[q] = __shfl_sync(0xffffffffu, za[q / 3], (lane & 7) + 8 * (q % 3));
                if (own && sub == 0) put_node(no, r, v);
            }
            wsync();  // the halo is read
        }
        return true;
    };

    // Power iterations y <- A^ y / ||y|| from a fixed pseudo-random vector (k_power_init's).  The norm of a vector
    // is waited for behind the next product, which it scales.
    if constexpr (POLY) {
        if (A.power) {
            const int sub = lane >> 3, r = wid * 8 + (lane & 7);
            const bool own = r < rows;
            auto start = [](unsigned i) {
                unsigned h = i * 2654435761u + 0x9e3779b9u;
                h ^= h >> 16;
                h *= 0x85ebca6bu;
                h ^= h >> 13;
                h *= 0xc2b2ae35u;
                h ^= h >> 16;
                return (TV)((double)(h >> 8) * (2.0 / 16777216.0) - 1.0);
            };
            TV y[DPN];
            ++no;
            if (own && sub == 0) {
#pragma unroll
                for (int q = 0; q < DPN; ++q) y[q] = start((unsigned)((row0 + r) * DPN + q));
                put_node(no, r, y);
            }
            for (int it = 0; it <= A.power; ++it) {
                TV a[DPN];
                const bool more = it < A.power;
                if (more) {
                    if (!gather(no)) break;
                    hopProduct(a);
                }
                if (it) {  // the norm of the last vector
                    totals(0, 1, it, sh1);
                    if (t == 0) sInv = (TV)(sh1[0] > 0.0 ? rsqrt(sh1[0]) : 0.0);  // (of every thread: 20,000 clocks)
                    wsync();
                    if (sStuck) break;
                }
                if (!more) break;
                const TV s = it ? sInv : TV(1);
                ++no;
                double yy = 0.0;
#pragma unroll
                for (int q = 0; q < DPN; ++q) {
                    y[q] = s * a[q];
                    if (own && q % 4 == sub) yy = fma(widen(y[q]), widen(y[q]), yy);
                }
                if (own && sub == 0) put_node(no, r, y);
                yy = warp_sum(yy);
                if (lane == 0) red[wid] = yy;
                wsync();
                if (wid == 0) {
                    const double v = warp_sum(red[lane]);
                    if (lane == 0) put_part(0, 0, v, it + 1);
                }
            }
            if (t == 0 && sStuck) A.ctl->stuck = 1;
            if (t == 0 && blockIdx.x == 0 && !sStuck) A.ctl->y[0] = sqrt(sh1[0]);
            return;
        }
    }

    int j = 0;
    // The workers' part: r = b - A x (products in FP64, every row's sum in the order of the residual kernel: a
    // cycle that starts below the target by its own rounding, but not by the solver's check, would never move
    // x), beta, then the steps.  False when a wait was given up.
    auto work = [&]() -> bool {
        // sw, scaled, as the next exchange
        auto send = [&] {
            ++no;
            if constexpr (sizeof(TV) == 8) {
                for (int i = t; i < nown; i += kWT) word_put(vec(no) + (size_t)row0 * DPN + i, A.y0s[(size_t)row0 * DPN + i] * sw[i], no);
            } else {
                for (int r = t; r < rows; r += kWT) {
                    TV v[DPN];
#pragma unroll
                    for (int q = 0; q < DPN; ++q) v[q] = A.y0s[(size_t)(row0 + r) * DPN + q] * sw[r * DPN + q];
                    put_node(no, r, v);
                }
            }
        };
        double rr = 0.0;
        for (int i = t; i < halo * DPN; i += kWT) sHalo[i / DPN * HS + i % DPN] = __ldcg(A.x + (size_t)sList[i / DPN] * DPN + i % DPN);
        wsync();
        product(1, 0.0, [&](int i, double a) {
            const double v = A.b[(size_t)row0 * DPN + i] - a;
            sw[i] = (TV)v;
            rr = fma(v, v, rr);
        });
        rr = warp_sum(rr);
        if (lane == 0) red[wid] = rr;
        wsync();
        if (wid == 0) {
            const double a = warp_sum(lane < kWW ? red[lane] : 0.0);
            if (lane == 0) put_part(0, 0, a, 1);
        }
        send();
        totals(0, 1, 1, sh1);
        wsync();
        if (sStuck) return false;
        if (t == 0) {
            const double beta = sqrt(sh1[0]);
            sDone = beta <= *A.target || beta == 0.0 || !isfinite(beta);
            sBad = !isfinite(beta);
            sBreak = 0;
            sInv = (TV)(beta > 0.0 ? 1.0 / beta : 0.0);
            sg[0] = beta;
        }
        wsync();
        for (;; ++j) {
            // w = A (P or D^-1) v_j, v_j = sw * inv; the product's input is exchange no.  Without hops the control
            // of the step before runs beside gather and product
            if constexpr (POLY) {
                if (sDone) return true;
                if (!hops(false)) return false;
            }
            if (!gather(no)) return false;
            product(stepSG, TV(0), [&](int i, TV a) { sy[i] = a; });
            __syncthreads();
            if (sDone) return true;
            const TV inv = sInv;
            for (int i = t; i < nown; i += kWT) {
                V[(size_t)j * vld + i] = sw[i] * inv;
                sw[i] = sy[i] * inv;
            }
            wsync();
            dots(j, 0);
            totals(0, j + 1, j + 2, sh1);
            wsync();
            if (sStuck) return false;
            subtract(j);
            wsync();
            dots(j, 1);
            totals(1, j + 2, j + 2, sh2);
            wsync();
            if (sStuck) return false;
            if constexpr (!POLY) __syncthreads();
            if (POLY && wid == kResW - 1) control(j);
            subtract(j);
            if constexpr (sizeof(TV) != 8 || POLY) wsync();  // (FP64: a thread sends the entries that it has)
            send();
            if constexpr (POLY) __syncthreads();
        }
    };
    if (POLY || wid < kWW) {
        if (!work()) {
            give_up();
            return;
        }
    } else {
        // one barrier with the workers behind the sums of a step, one behind the products of the next
        for (;; ++j) {
            __syncthreads();
            if (sStuck || sDone) break;
            __syncthreads();
            if (sStuck) break;
            control(j);
        }
        if (sStuck) return;  // (the workers met this barrier on their way out)
    }
    // ---- least squares (as k_lsq) and the update of x ---------------------------------------------------
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
                if (lane == k) shT[col] = (TV)y;
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
            for (int u = 0; u < 8; ++u) a += shT[k + u] * v[u];
        }
        for (; k < j; ++k) a += shT[k] * V[(size_t)k * vld + i];
        if constexpr (POLY) sw[i] = a;
        else A.x[(size_t)row0 * DPN + i] += A.y0s[(size_t)row0 * DPN + i] * a;
    }
    if constexpr (POLY) {
        if (j > 0) {
            __syncthreads();
            ++no;
            for (int r = t; r < rows; r += kWT) {
                TV v[DPN];
#pragma unroll
                for (int q = 0; q < DPN; ++q) v[q] = A.y0s[(size_t)(row0 + r) * DPN + q] * sw[r * DPN + q];
                put_node(no, r, v);
            }
            if (!hops(true)) {
                give_up();
                return;
            }
        }
    }
    if (blockIdx.x == 0 && t == 0) {
        A.ctl->resest = fabs(sg[j]);
        A.ctl->j = j;
        A.ctl->done = sDone;
        A.ctl->breakdown = sBreak;
        A.ctl->nonfinite = sBad;
    }
}

}  // namespace astro_kry
