// Operator apply (the `mul` kernel of the backend API):
//     out[m, n] = alpha * sum_k A[m, k] * B[k, n] + beta * out[m, n]
// A is a small constant operator matrix, B and out are row-major with
// leading dimensions ldb/ldc and `ncol` active columns (nvars * padded
// neles for the AoSoA fields).  This replaces the GiMMiK and cuBLASLt
// providers of the reference (pyfr/backends/cuda/gimmik.py:23-121,
// pyfr/backends/cuda/cublaslt.py:169-280) with one sparsity-aware kernel.
//
// Each CTA stages a k x 64 column tile of B into shared memory with
// asynchronous 16-byte copies (cp.async: every copy of the tile is in
// flight at once, so staging costs one memory latency rather than one per
// row; with large K the tile limits residency to a few CTAs per SM, which
// then cannot hide a row-by-row staging behind each other's FMAs), or with
// coalesced loads when B is not 16-byte aligned; every warp then produces
// whole rows of the output tile,
// walking the nonzeros of A (CSR, read through the read-only cache and
// broadcast across the warp).  Structural zeros of A cost nothing, so the
// sparse tensor-product operators run at their nonzero count.
#include <algorithm>
#include <map>
#include <math.h>
#include <stdlib.h>
#include <string.h>
#include <type_traits>
#include <utility>
#include <vector>

#include "common.cuh"
#include "fixedpoint.cuh"
#include "../../include/pyfrb200.h"

namespace {

constexpr int MUL_NCOL = 64;     // columns per CTA
constexpr int MUL_WARPS = 8;     // warps per CTA

struct MulHandle {
    int m, k, nnz;
    void *block;     // device memory of all that follows
    int *rowptr;     // device, m + 1
    int *colidx;     // device, nnz
    double *val64;   // device, nnz
    float *val32;    // device, nnz
    // The fixed-point form of the operator (FP64 applies; null when the
    // operator does not fit it): per row (first entry, end, scale s,
    // threshold), per entry (column, high part, low part, |high part|); and, for
    // dense rows, the magnitudes in 8 bits: per row (first word, end, threshold,
    // 0), per word (column/4, four entries)
    int4 *fxrow, *mgrow;     // device, m
    int4 *fxval;             // device, nnz
    int2 *mgval;             // device
    // The same by groups of up to four rows of one support (null when the
    // rows do not fall into such groups): per group gn columns and four rows
    // (-1: none), and (high, low part) and the value of every entry; one scale
    int gn, ngrp, gs;
    int *gcol, *grow;    // device, ngrp x gn and ngrp x 4
    int2 *gval;          // device, ngrp x 4 x gn
    double *gdbl;        // device, the same as doubles
};

template <typename T>
__device__ __forceinline__ const T *vals(const MulHandle &h);
template <>
__device__ __forceinline__ const double *vals<double>(const MulHandle &h) { return h.val64; }
template <>
__device__ __forceinline__ const float *vals<float>(const MulHandle &h) { return h.val32; }

// Epilogue modes: FP64 arithmetic is the scarce resource on this GPU, so
// the common cases alpha = 1 with beta = 0 or beta = 1 issue no FP64 work
// beyond the FMAs of the product (beta = 1 accumulates onto the loaded C).
enum { EPI_SET = 0, EPI_ADD = 1, EPI_GENERAL = 2, EPI_SCALE = 3 };

// 16-byte global -> shared copy; bytes < 16 reads that many and zero-fills
// the rest
__device__ __forceinline__ void cp_async16(void *dst, const void *src, int bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;"
                 :: "r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes)
                 : "memory");
}

// Stage the columns col0.. of B into bs [k][NC] (zero-filled beyond ncol); the
// caller synchronises the block
template <typename T, int NC>
__device__ __forceinline__ void stage_tile(T *bs, const T *b, int64_t ldb, int k, int64_t col0,
                                           int64_t ncol, int vec) {
    if (vec) {
        constexpr int VEC = 16 / sizeof(T), NV = NC / VEC;
        for (int idx = threadIdx.x; idx < k * NV; idx += blockDim.x) {
            const int r = idx / NV, cv = (idx % NV) * VEC;
            const int64_t col = col0 + cv;
            const int64_t rem = ncol - col;
            const int bytes = rem >= VEC ? 16 : (rem > 0 ? (int)rem * (int)sizeof(T) : 0);
            // (with nothing to read the source is any valid address)
            cp_async16(bs + r * NC + cv, bytes ? b + r * ldb + col : b, bytes);
        }
        asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
    } else {
        for (int idx = threadIdx.x; idx < k * NC; idx += blockDim.x) {
            int r = idx / NC, cc = idx % NC;
            int64_t col = col0 + cc;
            bs[idx] = (col < ncol) ? b[r * ldb + col] : T(0);
        }
    }
}

template <typename T, int EPI>
__global__ void __launch_bounds__(MUL_WARPS * 32)
mul_csr_kernel(MulHandle h, const T *__restrict__ b, int64_t ldb, T *__restrict__ c,
               int64_t ldc, int64_t ncol, T alpha, T beta, int vec) {
    b200::dependent_entry(b, c);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T *bs = reinterpret_cast<T *>(smem_raw);   // [k][MUL_NCOL]

    const int64_t col0 = (int64_t)blockIdx.x * MUL_NCOL;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;

    stage_tile<T, MUL_NCOL>(bs, b, ldb, h.k, col0, ncol, vec);
    __syncthreads();

    const T *__restrict__ av = vals<T>(h);
    const int64_t ca = col0 + lane, cb = col0 + lane + 32;
    const bool oka = ca < ncol, okb = cb < ncol;

    for (int row = warp; row < h.m; row += MUL_WARPS) {
        T *crow = c + row * ldc;
        T acc0 = T(0), acc1 = T(0);
        if (EPI == EPI_ADD) {
            if (oka) acc0 = crow[ca];
            if (okb) acc1 = crow[cb];
        }
        const int p0 = __ldg(h.rowptr + row), p1 = __ldg(h.rowptr + row + 1);
        for (int p = p0; p < p1; p++) {
            const T a = __ldg(av + p);
            const int kk = __ldg(h.colidx + p);
            acc0 = fma(a, bs[kk * MUL_NCOL + lane], acc0);
            acc1 = fma(a, bs[kk * MUL_NCOL + lane + 32], acc1);
        }

        if (EPI == EPI_GENERAL) {
            if (oka) acc0 = alpha * acc0 + beta * crow[ca];
            if (okb) acc1 = alpha * acc1 + beta * crow[cb];
        } else if (EPI == EPI_SCALE) {
            acc0 *= alpha;
            acc1 *= alpha;
        }
        if (oka) crow[ca] = acc0;
        if (okb) crow[cb] = acc1;
    }
}

// ---- FP64 applies in fixed point ---------------------------------------
//
// The FP64 unit issues 2 FMAs per clock per SM here; the 32-bit integer
// multiply-add with a 64-bit sum (IMAD.WIDE) issues about 56, on another
// pipe (a probe's rates at 1.92 GHz; both run side by side undisturbed).  A
// dot product of doubles over a common exponent is a dot product of
// integers, so a row of the operator times a column of B is formed as
//
//     B[k, n] = (bh 2^31 + bl) 2^-sb,  |bh| <= 2^28, |bl| <= 2^30
//     A[m, k] = (ah 2^29 + al) 2^-(s + 29),  sum_k |ah| ~ 2^30, |al| <= 2^28
//     hh = sum ah bh,  u = sum ah bl,  v = sum al bh    (64-bit, exact)
//     A B = (hh + u/2^31 + v/2^29 + ...) 2^(31 - s - sb)
//
// three IMAD.WIDE per nonzero, and the sum is rounded to FP64 once.  sb is
// the column's own (its largest exponent), s the row's.  In units of hh the
// result is within n/2 + 3/2 for n nonzeros, whatever their values: 1/4 of a
// unit each for A's rounding and for the product al bl that is left out, 1/2
// for B's truncation and 1/2 each for the roundings of u and v.  An FP64 dot
// product is within n 2^-53 of the terms' absolute sum, so the fixed-point form
// is as good as long as
//     sum |ah bh| >= 2^53 (1/2 + 3/(2n)),
// 1/13 to 1/53 of (row sum)(column maximum) for n = 15: not where large entries
// of the row meet zeros, or where the row's support is small against the
// column.  That is tested per output; outputs below it, and those of columns
// with infinities, NaNs or exponents near the ends of the range, are formed
// again with FP64 FMAs from global memory by the whole warp.  The test costs a
// multiply-add a nonzero more (IMAD.HI), or, in wide applies of dense rows,
// one for four, on a lower bound of the sum from the leading 8 bits of every
// value (IDP4A, in a loop of its own, which narrow applies, one chain of
// latencies each, are the slower for), and columns of values within a factor
// of four of each other need none.
//
// Bounds: hh <= 2^58 and u <= 2^60 by the row sums; v <= nnz 2^56, nnz <= 64
// (FX_MAXNNZ), so no sum overflows.

constexpr int FX_MAXNNZ = 64, FX_TILE = 113 * 1024;
constexpr int FX_BBITS = 59, FX_ALBITS = 29;
// The forms of the test
constexpr int FX_NONE = 0, FX_EACH = 1, FX_PACKED = 2;

// Bytes of a tile: 8 a value and, packed, 1 of its magnitude (rows of four)
inline size_t fx_smem(int k, int cpl, bool packed) {
    return (size_t)(k * 8 + (packed ? (k + 3) / 4 * 4 : 0)) * 32 * cpl;
}

// Columns per lane: 2 (64 columns a CTA, 16-byte accesses) or 1
template <int CPL>
struct FxPair;
template <>
struct FxPair<1> { using I = int2; };
template <>
struct FxPair<2> { using I = int4; };

// The exponent field of the largest value; whether anything but zero is
// there (hi the absolute high word, or 1 for a subnormal below it)
__device__ __forceinline__ int fx_mag(double x) {
    const int hi = __double2hiint(x) & 0x7fffffff;
    return hi | (__double2loint(x) != 0);
}

// (bh, bl) of x for a column whose largest exponent field is emax
__device__ __forceinline__ int2 fx_split(double x, int emax) {
    const int hi = __double2hiint(x);
    const int e = (hi >> 20) & 0x7ff;
    const int d = min(emax - e, 63);
    // 53-bit mantissa over zero bits, shifted down by the exponent difference
    // (values below 2^-59 of the largest become zero; a zero or subnormal
    // value always does)
    unsigned long long q =
        ((unsigned long long)((hi & 0xfffff) | 0x100000) << 32) | (unsigned)__double2loint(x);
    q = (q << (FX_BBITS - 53)) >> d;
    long long b = hi < 0 ? -(long long)q : (long long)q;
    b += 1ll << 30;
    int2 r;
    r.x = (int)(b >> 31);
    r.y = (int)((unsigned)b & 0x7fffffffu) - (1 << 30);
    return r;
}

template <int EPI, int CPL, int TEST>
__global__ void __launch_bounds__(MUL_WARPS * 32)
mul_fx_kernel(MulHandle h, const double *__restrict__ b, int64_t ldb, double *__restrict__ c,
              int64_t ldc, int64_t ncol, double alpha, double beta, int vec) {
    b200::dependent_entry(b, c);
    using I = typename FxPair<CPL>::I;
    constexpr int NC = 32 * CPL;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    I *bs = reinterpret_cast<I *>(smem_raw);             // [k][32]
    unsigned *mg = reinterpret_cast<unsigned *>(bs + h.k * 32);     // [(k + 3)/4][NC]
    __shared__ int cmax[NC], cmin[NC];
    if (threadIdx.x < NC) {
        cmax[threadIdx.x] = 0;
        cmin[threadIdx.x] = 0x7fffffff;
    }

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t col = (int64_t)blockIdx.x * NC + lane * CPL;
    bool ok[CPL];
#pragma unroll
    for (int j = 0; j < CPL; j++) ok[j] = col + j < ncol;
    const bool full = ok[CPL - 1];

    // Load the tile, every warp its rows, eight rows in flight per thread;
    // the largest and smallest magnitude of each column over the warp's rows
    int mag[CPL], low[CPL];
#pragma unroll
    for (int j = 0; j < CPL; j++) {
        mag[j] = 0;
        low[j] = 0x7fffffff;
    }
    constexpr int UNR = 8;
    for (int r0 = warp; r0 < h.k; r0 += UNR * MUL_WARPS) {
        double x[UNR][CPL];
#pragma unroll
        for (int q = 0; q < UNR; q++) {
            const int r = r0 + q * MUL_WARPS;
            const double *src = b + r * ldb + col;
#pragma unroll
            for (int j = 0; j < CPL; j++) x[q][j] = 0.0;
            if (r < h.k) {
                if (CPL == 2 && vec && full) {
                    const double2 t = *reinterpret_cast<const double2 *>(src);
                    x[q][0] = t.x;
                    x[q][CPL - 1] = t.y;
                } else {
#pragma unroll
                    for (int j = 0; j < CPL; j++)
                        if (ok[j]) x[q][j] = src[j];
                }
            }
        }
#pragma unroll
        for (int q = 0; q < UNR; q++) {
            const int r = r0 + q * MUL_WARPS;
            if (r < h.k) {
                double *dst = reinterpret_cast<double *>(bs + r * 32 + lane);
#pragma unroll
                for (int j = 0; j < CPL; j++) {
                    dst[j] = x[q][j];
                    const int t = fx_mag(x[q][j]);
                    mag[j] = max(mag[j], t);
                    low[j] = min(low[j], t);
                }
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < CPL; j++) {
        atomicMax(&cmax[lane * CPL + j], mag[j]);
        atomicMin(&cmin[lane * CPL + j], low[j]);
    }
    __syncthreads();

    // Column exponents; columns of which every output (wild) or none (zero) is
    // formed by FP64; whether a column needs the test: not where its smallest
    // value is at least a quarter of its largest, which makes sum |ah bh| at
    // least 2^54, the threshold of one nonzero.  (The columns of a tile are
    // mostly one variable's: those of density and energy pass.)
    int emax[CPL];
    bool wild[CPL], zero[CPL];
    bool need = false;
#pragma unroll
    for (int j = 0; j < CPL; j++) {
        const int mx = cmax[lane * CPL + j], mn = cmin[lane * CPL + j];
        // (at least 64 for the splits: then zeros have an exponent
        // difference that makes them zero)
        emax[j] = max(mx >> 20, 64);
        zero[j] = mx == 0;
        wild[j] = !zero[j] && (emax[j] < 128 || emax[j] > 1900);
        need = need || wild[j] || (!zero[j] && mn < mx - (2 << 20));
    }

    // Split in place (each thread the values that it stored)
    for (int r = warp; r < h.k; r += MUL_WARPS) {
        double *src = reinterpret_cast<double *>(bs + r * 32 + lane);
        int2 *dst = reinterpret_cast<int2 *>(src);
        int2 t[CPL];
#pragma unroll
        for (int j = 0; j < CPL; j++) t[j] = fx_split(src[j], emax[j]);
#pragma unroll
        for (int j = 0; j < CPL; j++) {
            dst[j] = t[j];
            // (rounded down: at most 255 2^20 of 2^28)
            if (TEST == FX_PACKED)
                reinterpret_cast<unsigned char *>(mg + (r / 4) * NC + lane * CPL + j)[r % 4] =
                    (unsigned char)min(abs(t[j].x) >> 20, 255);
        }
    }
    __syncthreads();

    const auto form = [&](int row, auto test) {
        double *crow = c + row * ldc + col;
        const int4 ri = __ldg(h.fxrow + row);
        double cin[CPL];
        if (EPI == EPI_ADD || EPI == EPI_GENERAL) {
#pragma unroll
            for (int j = 0; j < CPL; j++) cin[j] = ok[j] ? crow[j] : 0.0;
        }
        // (u and v start at half a unit of hh: the final shifts round)
        long long hh[CPL], u[CPL], v[CPL];
        unsigned m[CPL], thr = (unsigned)ri.w;      // the test's sums
#pragma unroll
        for (int j = 0; j < CPL; j++) {
            hh[j] = 0;
            u[j] = 1ll << 30;
            v[j] = 1ll << (FX_ALBITS - 1);
            m[j] = zero[j] ? 1u << 30 : 0u;
        }
#pragma unroll 4
        for (int p = ri.x; p < ri.y; p++) {
            const int4 a = __ldg(h.fxval + p);
            const I t = bs[a.x * 32 + lane];
            const int *tb = reinterpret_cast<const int *>(&t);
#pragma unroll
            for (int j = 0; j < CPL; j++) {
                const int bh = tb[2 * j], bl = tb[2 * j + 1];
                hh[j] += (long long)a.y * bh;
                u[j] += (long long)a.y * bl;
                v[j] += (long long)a.z * bh;
                if (test() == FX_EACH) m[j] += __umulhi((unsigned)a.w, (unsigned)abs(bh));
            }
        }

        if (test() == FX_PACKED) {
            const int4 mi = __ldg(h.mgrow + row);
            thr = (unsigned)mi.z;
#pragma unroll 4
            for (int p = mi.x; p < mi.y; p++) {
                const int2 g = __ldg(h.mgval + p);
#pragma unroll
                for (int j = 0; j < CPL; j++)
                    m[j] = __dp4a((unsigned)g.y, mg[g.x * NC + lane * CPL + j], m[j]);
            }
        }

        double r[CPL];
        bool small = false;
#pragma unroll
        for (int j = 0; j < CPL; j++) {
            const long long t = hh[j] + (u[j] >> 31) + (v[j] >> FX_ALBITS);
            r[j] = (double)t;
            // times 2^(31 - s - sb), sb = 1022 + FX_BBITS - emax: an exponent
            // sum, in the normal range by the limits on emax and s
            if (t != 0)
                r[j] = __hiloint2double(__double2hiint(r[j]) +
                                            (emax[j] - (991 + FX_BBITS) - ri.z) * (1 << 20),
                                        __double2loint(r[j]));
            small |= wild[j] || m[j] < thr;
        }
        if (test() != FX_NONE && __any_sync(0xffffffffu, small)) {
            const int p0 = __ldg(h.rowptr + row), p1 = __ldg(h.rowptr + row + 1);
            double acc[CPL];
#pragma unroll
            for (int j = 0; j < CPL; j++) acc[j] = 0.0;
            for (int p = p0; p < p1; p++) {
                const double a = __ldg(h.val64 + p);
                const double *src = b + __ldg(h.colidx + p) * ldb + col;
#pragma unroll
                for (int j = 0; j < CPL; j++)
                    if (ok[j]) acc[j] = fma(a, src[j], acc[j]);
            }
#pragma unroll
            for (int j = 0; j < CPL; j++)
                if (wild[j] || m[j] < thr) r[j] = acc[j];
        }
#pragma unroll
        for (int j = 0; j < CPL; j++) {
            if (EPI == EPI_GENERAL) r[j] = alpha * r[j] + beta * cin[j];
            if (EPI == EPI_ADD) r[j] += cin[j];
            if (EPI == EPI_SCALE) r[j] *= alpha;
        }
        if (CPL == 2 && vec && full) {
            *reinterpret_cast<double2 *>(crow) = make_double2(r[0], r[CPL - 1]);
        } else {
#pragma unroll
            for (int j = 0; j < CPL; j++)
                if (ok[j]) crow[j] = r[j];
        }
    };
    if (__any_sync(0xffffffffu, need))
        for (int row = warp; row < h.m; row += MUL_WARPS)
            form(row, std::integral_constant<int, TEST>());
    else
        for (int row = warp; row < h.m; row += MUL_WARPS)
            form(row, std::integral_constant<int, FX_NONE>());
}

template <int CPL, int TEST>
void launch_fx(const MulHandle &h, const double *b, int64_t ldb, double *c, int64_t ldc,
               int64_t ncol, double alpha, double beta, int vec, cudaStream_t s) {
    const unsigned grid = b200::ceil_div(ncol, 32 * CPL);
    const size_t smem = fx_smem(h.k, CPL, TEST == FX_PACKED);
    auto go = [&](auto epi) {
        b200::launch(mul_fx_kernel<epi(), CPL, TEST>, grid, MUL_WARPS * 32, smem, s, h, b, ldb, c, ldc, ncol, alpha, beta, vec);
    };
    if (alpha == 1.0 && beta == 0.0)
        go(std::integral_constant<int, EPI_SET>());
    else if (alpha == 1.0 && beta == 1.0)
        go(std::integral_constant<int, EPI_ADD>());
    else if (beta == 0.0)
        go(std::integral_constant<int, EPI_SCALE>());
    else
        go(std::integral_constant<int, EPI_GENERAL>());
}

// ---- the same by groups of rows of one support ---------------------------
//
// The rows of tensor-product operators come in lines: four derivatives from the
// same four values, two face values from one line.  A group's operands are
// loaded and split once for its rows (by the splits of fixedpoint.cuh), over
// their own largest exponent, so that there is no pass over the column, no test
// and no second form of an output (but for exponents out of range).  Sums: with
// sum |ah| ~ 2^30, |al| <= 2^30 and 60 bits of B, |w| is below
// 2^61 + N 2^59 < 2^63 for the N <= 6 taken.
//
// What bounds it is issue slots (the integer pipes at 53%, the FP64 unit's
// conversions at 21%) and, in large applies, DRAM beside them: 192 x 64 gradient
// operator of p = 3 hexahedra, 35005 columns, 25.4 us by columns (above; a
// quarter of its rows formed twice where the values pass through zero), 22.0 us
// by groups, its DRAM time 10.5 us; at 320 columns 21.2 -> 11.3 us, where the
// chain of one tile is all there is.  Every other row is converted on the FP64
// unit, the rest on the integer pipes: all on the former would take its 2 a clock
// and SM 11.5 us of the kernel, all on the latter a third more instructions.
//
// Groups of pairs of values (192 x 96 and 375 x 150 lifts) are left to the FP64
// form, which is 15-50% faster there: two products do not pay for a split.

constexpr int FXG_ROWS = 4, FXG_MIN = 3, FXG_MAX = 6;

template <int EPI, int CPL, int N>
__global__ void __launch_bounds__(MUL_WARPS * 32)
mul_fxg_kernel(MulHandle h, const double *__restrict__ b, int64_t ldb, double *__restrict__ c,
               int64_t ldc, int64_t ncol, double alpha, double beta, int vec, int vecc) {
    b200::dependent_entry(b, c);
    constexpr int NC = 32 * CPL;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double *bs = reinterpret_cast<double *>(smem_raw);   // [k][NC]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t col0 = (int64_t)blockIdx.x * NC, col = col0 + lane * CPL;
    stage_tile<double, NC>(bs, b, ldb, h.k, col0, ncol, vec);
    __syncthreads();

    bool ok[CPL];
#pragma unroll
    for (int j = 0; j < CPL; j++) ok[j] = col + j < ncol;
    const bool pair = CPL == 2 && vecc && ok[CPL - 1];

    for (int g = warp; g < h.ngrp; g += MUL_WARPS) {
        double x[N][CPL];
#pragma unroll
        for (int i = 0; i < N; i++) {
            const double *src = bs + __ldg(h.gcol + g * N + i) * NC + lane * CPL;
            if (CPL == 2) {
                const double2 t = *reinterpret_cast<const double2 *>(src);
                x[i][0] = t.x;
                x[i][CPL - 1] = t.y;
            } else {
                x[i][0] = src[0];
            }
        }
        int emax[CPL];
        bool wild[CPL];
        int2 y[N][CPL];
#pragma unroll
        for (int j = 0; j < CPL; j++) {
            // (1 for a subnormal without a high word: out of range)
            int mx = 0;
#pragma unroll
            for (int i = 0; i < N; i++)
                mx = max(mx, b200::hi_abs(x[i][j]) | (__double2loint(x[i][j]) != 0));
            wild[j] = b200::out_of_range(mx);
            emax[j] = max(mx >> 20, 64);
#pragma unroll
            for (int i = 0; i < N; i++) y[i][j] = b200::split<60>(x[i][j], emax[j]);
        }
        const bool any = __any_sync(0xffffffffu, wild[0] || wild[CPL - 1]);
        const int4 rows = __ldg(reinterpret_cast<const int4 *>(h.grow) + g);
        const int rr[FXG_ROWS] = {rows.x, rows.y, rows.z, rows.w};
#pragma unroll
        for (int q = 0; q < FXG_ROWS; q++) {
            if (rr[q] < 0) break;
            double *crow = c + rr[q] * ldc + col, r[CPL];
            const int2 *av = h.gval + (g * FXG_ROWS + q) * N;
            b200::Fx s[CPL];
#pragma unroll
            for (int j = 0; j < CPL; j++) s[j].clear();
#pragma unroll
            for (int i = 0; i < N; i++) {
                const int2 a = __ldg(av + i);
#pragma unroll
                for (int j = 0; j < CPL; j++) s[j].mad(a, y[i][j]);
            }
#pragma unroll
            for (int j = 0; j < CPL; j++) {
                const int sc = emax[j] - h.gs - 1051;
                r[j] = q % 2 ? s[j].value(sc) : s[j].value_cvt(sc);
                // (a branch of the warp with a loop in it: as selected values
                // these FMAs would run for every output)
                if (any) {
                    double f = 0.0;
                    const double *ad = h.gdbl + (g * FXG_ROWS + q) * N;
#pragma unroll 1
                    for (int i = 0; i < N; i++)
                        // (a filled-up support's zero stays out of infinities)
                        if (const double av = __ldg(ad + i); av != 0.0)
                            f = fma(av, bs[__ldg(h.gcol + g * N + i) * NC + lane * CPL + j], f);
                    if (wild[j]) r[j] = f;
                }
                const double old = EPI == EPI_ADD || EPI == EPI_GENERAL
                                       ? (ok[j] ? crow[j] : 0.0) : 0.0;
                if (EPI == EPI_GENERAL) r[j] = alpha * r[j] + beta * old;
                if (EPI == EPI_ADD) r[j] += old;
                if (EPI == EPI_SCALE) r[j] *= alpha;
            }
            if (pair) {
                *reinterpret_cast<double2 *>(crow) = make_double2(r[0], r[CPL - 1]);
            } else {
#pragma unroll
                for (int j = 0; j < CPL; j++)
                    if (ok[j]) crow[j] = r[j];
            }
        }
    }
}

// fn(integral constants: columns per lane, group size, epilogue)
template <typename F>
bool with_fxg(int cpl, int n, int epi, F &&fn) {
    auto by_epi = [&](auto c, auto g) {
        switch (epi) {
        case EPI_SET: fn(c, g, std::integral_constant<int, EPI_SET>()); break;
        case EPI_ADD: fn(c, g, std::integral_constant<int, EPI_ADD>()); break;
        case EPI_GENERAL: fn(c, g, std::integral_constant<int, EPI_GENERAL>()); break;
        default: fn(c, g, std::integral_constant<int, EPI_SCALE>());
        }
    };
    auto by_n = [&](auto c) {
        switch (n) {
        case 3: by_epi(c, std::integral_constant<int, 3>()); return true;
        case 4: by_epi(c, std::integral_constant<int, 4>()); return true;
        case 5: by_epi(c, std::integral_constant<int, 5>()); return true;
        case 6: by_epi(c, std::integral_constant<int, 6>()); return true;
        default: return false;
        }
    };
    return cpl == 1 ? by_n(std::integral_constant<int, 1>())
                    : by_n(std::integral_constant<int, 2>());
}

// The operator's rows in groups of one support, or false where they are not: of
// two rows a group on average, of support sizes within one of each other, from
// FXG_MIN to FXG_MAX (a smaller one is filled up with a zero entry on a column
// that it has: the derivatives at p = 4, where the middle point's own is zero;
// 24.5 us at 320 columns, 41 by FMAs; 117 us at 35005, by columns 114 to 172, the
// more the smaller a line's values are against its column's), and with no entry
// below 1/16 of the largest row's mean.  A group's sums are within (1 + N/2 + N/8)
// 2^-57 of (largest row sum)(largest value of the support), which for such entries
// is below 5 times the classical bound of FP64 sums, N 2^-53 of the terms' absolute
// sum, whatever the values are (below 1 for the derivatives of p = 3 hexahedra,
// 3.4 for the interpolation at p = 5); an entry far below the others would lose
// the bits that it has alone where theirs meet zeros.
struct Groups {
    int n = 0, s = 0;
    std::vector<int> col, row;
    std::vector<int2> val;
    std::vector<double> dbl;
};

bool fx_groups(const double *a, int m, int k, Groups &g) {
    std::map<std::vector<int>, std::vector<int>> by;
    double top = 0.0, low = INFINITY, least = INFINITY;
    int fewest = FXG_MAX;
    for (int i = 0; i < m; i++) {
        std::vector<int> sup;
        double l1 = 0.0;
        for (int j = 0; j < k; j++) {
            const double x = fabs(a[(size_t)i * k + j]);
            if (x == 0.0) continue;
            sup.push_back(j);
            l1 += x;
            least = fmin(least, x);
        }
        const int n = (int)sup.size();
        if (n < FXG_MIN || n > FXG_MAX || !(l1 <= ldexp(1.0, 60))) return false;
        g.n = std::max(g.n, n);
        fewest = std::min(fewest, n);
        top = fmax(top, l1);
        low = fmin(low, l1);
        by[sup].push_back(i);
    }
    if (g.n - fewest > 1) return false;
    // (one scale: the smallest row keeps 57 of its bits)
    if (!(low >= ldexp(1.0, -60)) || low < top / 16 || 16 * g.n * least < top) return false;
    int e;
    frexp(top, &e);
    g.s = 30 - e;
    // (in the order of the first row, so that neighbouring groups write
    // neighbouring rows)
    std::vector<std::pair<int, const std::vector<int> *>> order;
    for (auto &kv : by) order.push_back({kv.second[0], &kv.first});
    std::sort(order.begin(), order.end());
    for (auto &o : order) {
        const std::vector<int> &rows = by[*o.second];
        for (size_t r0 = 0; r0 < rows.size(); r0 += FXG_ROWS) {
            std::vector<int> cols = *o.second;
            const int n = (int)cols.size();
            cols.resize(g.n, cols[0]);
            g.col.insert(g.col.end(), cols.begin(), cols.end());
            for (int q = 0; q < FXG_ROWS; q++) {
                const int r = r0 + q < rows.size() ? rows[r0 + q] : -1;
                g.row.push_back(r);
                for (int i = 0; i < g.n; i++) {
                    const double x = r < 0 || i >= n ? 0.0 : a[(size_t)r * k + cols[i]];
                    const long long z = llrint(ldexp(x, g.s + 31));
                    const long long ah = (z + (1ll << 30)) >> 31;
                    g.val.push_back(make_int2((int)ah, (int)(z - ah * (1ll << 31))));
                    g.dbl.push_back(x);
                }
            }
        }
    }
    return (size_t)m >= 2 * (g.row.size() / FXG_ROWS);
}

// An operator's arrays in one block of device memory: an allocation and a copy
// each took most of mul_create's time
struct Block {
    std::vector<unsigned char> bytes;
    std::vector<std::pair<void **, size_t>> ptrs;
    template <typename V>
    void add(V **dst, const std::vector<V> &src) {
        bytes.resize((bytes.size() + 15) / 16 * 16);
        ptrs.push_back({(void **)dst, bytes.size()});
        const unsigned char *p = (const unsigned char *)src.data();
        bytes.insert(bytes.end(), p, p + sizeof(V) * src.size());
    }
    int upload(void **block) {
        int rc = b200::check_cuda(cudaMalloc(block, bytes.size()), "mul_create");
        if (!rc)
            rc = b200::check_cuda(cudaMemcpy(*block, bytes.data(), bytes.size(),
                                             cudaMemcpyHostToDevice), "mul_create");
        for (auto &p : ptrs) *p.first = (unsigned char *)*block + p.second;
        return rc;
    }
};

// The operator's fixed-point form (rows, entries), or false where it does
// not fit: a row of more than FX_MAXNNZ entries, or of an absolute sum
// outside [2^-60, 2^60] (or not finite)
bool fx_operator(const double *a, int m, int k, std::vector<int4> &rows,
                 std::vector<int4> &vals, std::vector<int4> &mgrows, std::vector<int2> &mgs) {
    for (int i = 0; i < m; i++) {
        const double *ar = a + (size_t)i * k;
        double l1 = 0.0;
        int nnz = 0;
        for (int j = 0; j < k; j++) {
            l1 += fabs(ar[j]);
            nnz += ar[j] != 0.0;
        }
        if (nnz > FX_MAXNNZ || (nnz && !(l1 >= ldexp(1.0, -60) && l1 <= ldexp(1.0, 60))))
            return false;
        // sum |A| 2^s in [2^29, 2^30): with the rounding of every |ah| up
        // by at most 1 the sum of |ah| stays below 2^30 + FX_MAXNNZ
        int e = 0;
        if (nnz) frexp(l1, &e);
        const int s = 30 - e;
        const int p0 = (int)vals.size();
        for (int j = 0; j < k; j++) {
            if (ar[j] == 0.0) continue;
            const long long q = llrint(ldexp(ar[j], s + FX_ALBITS));
            const long long ah = (q + (1ll << (FX_ALBITS - 1))) >> FX_ALBITS,
                            al = q - ah * (1ll << FX_ALBITS);
            vals.push_back(make_int4(j, (int)ah, (int)al, abs((int)ah)));
        }
        // (in units of 2^32: the high words of the products)
        const double least = nnz ? 0.5 + 1.5 / nnz : 0.0;
        rows.push_back(make_int4(p0, (int)vals.size(), s, (int)ceil(ldexp(least, 53 - 32))));
        // Magnitudes |ah|/unit rounded down, the row's largest about 255; with
        // B's, |bh| 2^-20 rounded down, the sum of the products is below
        // sum |ah bh| 2^-20/unit, and so has to be at least
        int top = 0;
        for (int p = p0; p < (int)vals.size(); p++) top = std::max(top, abs(vals[p].y));
        const int unit = top / 255 + 1, q0 = (int)mgs.size();
        for (int p = p0; p < (int)vals.size(); p++) {
            const int j = vals[p].x;
            if ((int)mgs.size() == q0 || mgs.back().x != j / 4) mgs.push_back(make_int2(j / 4, 0));
            mgs.back().y |= (int)((unsigned)(abs(vals[p].y) / unit) << (8 * (j % 4)));
        }
        mgrows.push_back(
            make_int4(q0, (int)mgs.size(), (int)ceil(ldexp(least, 53 - 20) / unit), 0));
    }
    return true;
}

template <typename T>
int launch_mul(const MulHandle *h, const T *b, int64_t ldb, T *c, int64_t ldc, int64_t ncol,
               T alpha, T beta, cudaStream_t s) {
    if (!h) return b200::set_error(B200_ERR_ARG, "mul: null handle");
    if (ncol <= 0) return B200_OK;
    if (ldb < ncol || ldc < ncol)
        return b200::set_error(B200_ERR_ARG, "mul: leading dimension smaller than ncol");
    size_t smem = (size_t)h->k * MUL_NCOL * sizeof(T);
    if (smem > 227 * 1024)
        return b200::set_error(B200_ERR_UNSUPPORTED, "mul: k=%d too large for the tile", h->k);
    unsigned grid = b200::ceil_div(ncol, MUL_NCOL);
    // 16-byte copies need a 16-byte aligned base and row stride
    const int vec = !((uintptr_t)b & 15) && !((ldb * (int64_t)sizeof(T)) & 15);
    if constexpr (sizeof(T) == 8) {
        if (h->gval) {
            // Groups of rows of one support, at every width: against the faster
            // of the other two forms 21.2 -> 11.3 us at 320 columns and
            // 74.4 -> 67.6 us at 87880 for the 192 x 64 gradient, 17.8 -> 12.4
            // and 106 -> 88 us for the 150 x 125 interpolation at p = 4, and
            // from 10.9 -> 7.7 to 44.4 -> 46.5 us for the 96 x 64 one.  Two
            // columns a lane where every SM has a tile and room for two
            const int cpl = ncol > 64 * b200::SM_COUNT && smem <= 113 * 1024 ? 2 : 1;
            const int vecc = !((uintptr_t)c & 15) && !(ldc & 1);
            const int epi = alpha == 1.0 ? (beta == 0.0 ? EPI_SET : beta == 1.0 ? EPI_ADD : EPI_GENERAL)
                                         : (beta == 0.0 ? EPI_SCALE : EPI_GENERAL);
            with_fxg(cpl, h->gn, epi, [&](auto cp, auto gn, auto ep) {
                b200::launch(mul_fxg_kernel<ep(), cp(), gn()>, b200::ceil_div(ncol, 32 * cp()),
                             MUL_WARPS * 32, (size_t)h->k * 32 * cp() * sizeof(double), s, *h, b, ldb,
                             c, ldc, ncol, alpha, beta, vec, vecc);
            });
            B200_CHECK_LAUNCH("mul_fxg_kernel");
            return B200_OK;
        }
        // (the FP64 FMAs of small outputs read B again, so C must not be B)
        const bool apart = c + (int64_t)(h->m - 1) * ldc + ncol <= b ||
                           b + (int64_t)(h->k - 1) * ldb + ncol <= c;
        // Where the FMAs bound: rows of ten entries and more at every width
        // (tetrahedra's 20 x 40 lift at 20480 columns 38.5 -> 17.4 us, before
        // the test of the terms' sum), rows of four and more once every SM has
        // a tile (hexahedra's 375 x 125 gradient at p = 4, by columns, 93 -> 59
        // us at 20480 columns; below 9728 columns of rows of four the FP64
        // form's shorter chain is up to 10% faster, and for rows of two,
        // 192 x 96, it is 15-25% faster at every width).  The tile has to leave an SM room
        // for two CTAs (the 125 x 375 divergence at p = 4: 359 us against
        // 370).
        const bool many = h->nnz >= 10 * (int64_t)h->m ||
                          (h->nnz >= 4 * (int64_t)h->m && ncol > 64 * b200::SM_COUNT);
        if (h->fxval && apart && many && smem <= FX_TILE) {
            const int vec2 = vec && !((uintptr_t)c & 15) && !(ldc & 1);
            // One column per lane where two would leave SMs without a tile; the
            // packed test of dense rows from two tiles an SM on (20 x 60
            // divergence of p = 3 tetrahedra, columns that need the test: 17.1
            // us by products and 17.6 packed at 9729 columns, 28.9 and 24.7
            // at 35005, where columns that need none take 22.5)
            if (ncol <= 64 * b200::SM_COUNT)
                launch_fx<1, FX_EACH>(*h, b, ldb, c, ldc, ncol, alpha, beta, vec2, s);
            else if (h->mgval && ncol > 2 * 64 * b200::SM_COUNT && fx_smem(h->k, 2, true) <= FX_TILE)
                launch_fx<2, FX_PACKED>(*h, b, ldb, c, ldc, ncol, alpha, beta, vec2, s);
            else
                launch_fx<2, FX_EACH>(*h, b, ldb, c, ldc, ncol, alpha, beta, vec2, s);
            B200_CHECK_LAUNCH("mul_fx_kernel");
            return B200_OK;
        }
    }
    if (alpha == T(1) && beta == T(0))
        b200::launch(mul_csr_kernel<T, EPI_SET>, grid, MUL_WARPS * 32, smem, s, *h, b, ldb, c, ldc, ncol, alpha, beta, vec);
    else if (alpha == T(1) && beta == T(1))
        b200::launch(mul_csr_kernel<T, EPI_ADD>, grid, MUL_WARPS * 32, smem, s, *h, b, ldb, c, ldc, ncol, alpha, beta, vec);
    else if (beta == T(0))
        b200::launch(mul_csr_kernel<T, EPI_SCALE>, grid, MUL_WARPS * 32, smem, s, *h, b, ldb, c, ldc, ncol, alpha, beta, vec);
    else
        b200::launch(mul_csr_kernel<T, EPI_GENERAL>, grid, MUL_WARPS * 32, smem, s, *h, b, ldb, c, ldc, ncol, alpha, beta, vec);
    B200_CHECK_LAUNCH("mul_csr_kernel");
    return B200_OK;
}

// Opt every instantiation in to the largest tile.  Called from
// b200_mul_create, which never runs inside a stream capture: changing a
// function attribute while a capture is open invalidates the capture.
template <int CPL, int TEST>
int opt_in_smem_fx() {
    void (*fns[4])(MulHandle, const double *, int64_t, double *, int64_t, int64_t, double,
                   double, int) = {
        mul_fx_kernel<EPI_SET, CPL, TEST>, mul_fx_kernel<EPI_ADD, CPL, TEST>,
        mul_fx_kernel<EPI_GENERAL, CPL, TEST>, mul_fx_kernel<EPI_SCALE, CPL, TEST>};
    for (auto fn : fns) {
        cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             FX_TILE);
        if (e != cudaSuccess) return b200::check_cuda(e, "mul: smem attribute");
    }
    return B200_OK;
}

template <typename T>
int opt_in_smem() {
    void (*fns[4])(MulHandle, const T *, int64_t, T *, int64_t, int64_t, T, T, int) = {
        mul_csr_kernel<T, EPI_SET>, mul_csr_kernel<T, EPI_ADD>,
        mul_csr_kernel<T, EPI_GENERAL>, mul_csr_kernel<T, EPI_SCALE>};
    for (auto fn : fns) {
        cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             227 * 1024);
        if (e != cudaSuccess) return b200::check_cuda(e, "mul: smem attribute");
    }
    return B200_OK;
}

void free_handle(MulHandle *h) {
    cudaFree(h->block);
    free(h);
}

}  // namespace

extern "C" {

int b200_mul_create(const double *a, int m, int k, void **handle) {
    if (!a || !handle || m <= 0 || k <= 0)
        return b200::set_error(B200_ERR_ARG, "mul_create: bad arguments");
    int orc = opt_in_smem<double>();
    if (!orc) orc = opt_in_smem<float>();
    if (!orc) orc = opt_in_smem_fx<1, FX_EACH>();
    if (!orc) orc = opt_in_smem_fx<2, FX_EACH>();
    if (!orc) orc = opt_in_smem_fx<2, FX_PACKED>();
    if (orc) return orc;

    std::vector<int> rowptr(m + 1, 0), colidx;
    std::vector<double> v64;
    std::vector<float> v32;
    for (int i = 0; i < m; i++) {
        for (int j = 0; j < k; j++) {
            double x = a[(size_t)i * k + j];
            if (x != 0.0) {
                colidx.push_back(j);
                v64.push_back(x);
                v32.push_back((float)x);
            }
        }
        rowptr[i + 1] = (int)colidx.size();
    }

    MulHandle *h = (MulHandle *)calloc(1, sizeof(MulHandle));
    if (!h) return b200::set_error(B200_ERR_STATE, "mul_create: out of host memory");
    h->m = m;
    h->k = k;
    h->nnz = (int)colidx.size();
    int rc = B200_OK;
    Block block;
    block.add(&h->rowptr, rowptr);
    block.add(&h->colidx, colidx);
    block.add(&h->val64, v64);
    block.add(&h->val32, v32);
    std::vector<int4> fxrow, fxval, mgrow;
    std::vector<int2> mgval;
    Groups gr;
    if (h->nnz && fx_groups(a, m, k, gr)) {
        h->gn = gr.n;
        h->ngrp = (int)gr.row.size() / FXG_ROWS;
        h->gs = gr.s;
        block.add(&h->gcol, gr.col);
        block.add(&h->grow, gr.row);
        block.add(&h->gdbl, gr.dbl);
        block.add(&h->gval, gr.val);
        // (opted in to the largest tile here, where no capture is open)
        for (int cpl = 1; cpl <= 2; cpl++)
            for (int epi : {EPI_SET, EPI_ADD, EPI_GENERAL, EPI_SCALE})
                with_fxg(cpl, h->gn, epi, [&](auto cp, auto gn, auto ep) {
                    if (!rc)
                        rc = b200::check_cuda(
                            cudaFuncSetAttribute(mul_fxg_kernel<ep(), cp(), gn()>,
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 227 * 1024), "mul: smem attribute");
                });
    } else if (h->nnz && fx_operator(a, m, k, fxrow, fxval, mgrow, mgval)) {
        block.add(&h->fxrow, fxrow);
        block.add(&h->fxval, fxval);
        // (dense: three entries a word or more)
        if (3 * mgval.size() <= fxval.size()) {
            block.add(&h->mgrow, mgrow);
            block.add(&h->mgval, mgval);
        }
    }
    if (!rc) rc = block.upload(&h->block);
    if (rc) {
        free_handle(h);
        return rc;
    }
    *handle = h;
    return B200_OK;
}

int b200_mul_nnz(void *handle, int *nnz) {
    if (!handle || !nnz) return b200::set_error(B200_ERR_ARG, "mul_nnz: bad arguments");
    *nnz = ((MulHandle *)handle)->nnz;
    return B200_OK;
}

int b200_mul_destroy(void *handle) {
    if (!handle) return B200_OK;
    free_handle((MulHandle *)handle);
    return B200_OK;
}

int b200_mul_f64(void *handle, const double *b, int64_t ldb, double *c, int64_t ldc,
                 int64_t ncol, double alpha, double beta, void *stream) {
    return launch_mul<double>((const MulHandle *)handle, b, ldb, c, ldc, ncol, alpha, beta,
                              (cudaStream_t)stream);
}

int b200_mul_f32(void *handle, const float *b, int64_t ldb, float *c, int64_t ldc,
                 int64_t ncol, float alpha, float beta, void *stream) {
    return launch_mul<float>((const MulHandle *)handle, b, ldb, c, ldc, ncol, alpha, beta,
                             (cudaStream_t)stream);
}

}  // extern "C"
