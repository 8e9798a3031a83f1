// Element kernels of tensor-product elements (quadrilaterals and hexahedra
// with Gauss-Legendre points), whose operators are one-dimensional matrices
// applied along the lines of points of each direction:
//
//   te_interp     the solution at the flux points (M0)
//   te_gradflux   Navier-Stokes: the corrected gradient (M4 - M6 M0 and M6),
//                 its transform, the flux at the solution points, the
//                 gradient at the flux points (M0) and the divergence of the
//                 flux less its own lift (M1 - M3 M2), one element's data
//                 staying in shared memory from the first to the last
//   te_lift       R = -(1/|J|) (R + M3 Fc)
//   te_euler      Euler: the flux, its divergence, the lift of the common
//                 flux and the scaling: R from u and Fc
//
// They take the place of the operator applies and pointwise kernels that the
// systems otherwise run one by one
// (pyfr/solvers/baseadvec/elements.py:91-120,
// pyfr/solvers/baseadvecdiff/elements.py:47-116), where the gradient was
// written once and read three times and the flux written and read.
//
// Along a line every operand is used by all of its outputs from registers and
// the matrices are constants of the launch, where the general sparse apply
// loads an index, a coefficient and an operand per product.
//
// FP64: the products along a line run on the integer pipe, in fixed point over
// the line's own largest exponent (the arithmetic of the general apply,
// csrc/mul.cu: IMAD.WIDE issues 56 a clock and SM where the FP64 unit issues
// 2 FMAs; its support test is not needed, since a line is its support).
// With B of 60 bits and A of 60 or 61 below the largest row sum the result is
// within 6 2^-56 of (largest row sum)(largest value of the line), below the
// rounding of one FP64 FMA.  The divergence at a point is the sum of a line of
// each direction, every line over its own exponent, and the integer sums are
// shifted to the largest of them before the one rounding to FP64: an output
// keeps its bits however large the fluxes elsewhere in the element are, or the
// middle point of an odd line, which its own derivative leaves out.
// The FP64 unit is left to the flux, beside which the integer work of the
// other warps runs.
#include <math.h>
#include <stdlib.h>
#include <string.h>

#include "common.cuh"
#include "elemgeom.cuh"
#include "fixedpoint.cuh"
#include "physics.cuh"
#include "../../include/pyfrb200.h"

using b200::ElemGeom;
using b200::Fx;
using b200::hi_abs;
using b200::out_of_range;
using b200::split;
using b200::Gas;
using b200::soa_off;

namespace {

// ---- matrices of the lines --------------------------------------------------

// The derivative matrices are antisymmetric about the line's middle: with an
// odd number of points the middle point does not enter its own derivative, and
// is left out (so that an infinity there has the reach that it has in the
// general apply, which skips zeros).  te_create checks that the entry is zero.
template <int NO, int NI>
__device__ constexpr bool absent(int i, int j) {
    return NI == NO + 2 && (NO & 1) && i == NO / 2 && j == NO / 2;
}

template <typename T, int NO, int NI>
struct Mat;

template <int NO, int NI>
struct Mat<float, NO, NI> {
    float d[NO][NI];
};

// a = (ah, al): A = (ah 2^31 + al) 2^-(s + 31), |al| <= 2^30, every row's sum of
// |ah| below 2^30 + NI, or below 2^29 + NI (wide: rows of ND directions are
// summed).  With B of BITS = 60 bits (58 where ND lines make one sum), |bh| <
// 2^(BITS - 31), |bl| < 2^31, the cross sum of Fx stays below 2^63: 2^61 + 7 2^59
// for one line of 7 entries, 2 2^60 + 14 2^57 for two, and the high sum below
// 2^60, of which three still make less than the 2^61 that Fx::value takes.
template <int NO, int NI>
struct Mat<double, NO, NI> {
    double d[NO][NI];
    int2 a[NO][NI];
    int s;
};

template <int NO, int NI>
void set_mat(Mat<float, NO, NI> &m, const double *a, bool = false) {
    for (int i = 0; i < NO; i++)
        for (int j = 0; j < NI; j++) m.d[i][j] = (float)a[i * NI + j];
}

template <int NO, int NI>
void set_mat(Mat<double, NO, NI> &m, const double *a, bool wide = false) {
    double l1 = 0.0;
    for (int i = 0; i < NO; i++) {
        double r = 0.0;
        for (int j = 0; j < NI; j++) r += fabs(a[i * NI + j]);
        l1 = fmax(l1, r);
    }
    int e = 0;
    if (l1 > 0.0) frexp(l1, &e);
    m.s = (wide ? 29 : 30) - e;
    for (int i = 0; i < NO; i++)
        for (int j = 0; j < NI; j++) {
            const double x = a[i * NI + j];
            const long long q = llrint(ldexp(x, m.s + 31));
            const long long ah = (q + (1ll << 30)) >> 31;
            m.d[i][j] = x;
            m.a[i][j] = make_int2((int)ah, (int)(q - ah * (1ll << 31)));
        }
}

// The middle point of an odd line is no operand of its own derivative, which has
// the bits of the others alone: where that point is more than four times as
// large as they are (whether zeros or not), the line is formed by FMAs.  mx and
// mo: the largest magnitudes of the line and of its other points.
constexpr int middle(int q) { return q & 1 ? q / 2 : -1; }
__device__ __forceinline__ bool lone_middle(int mx, int mo) {
    return mo != 0 && mo < mx - (2 << 20);
}

// The operands of a line, as the products take them; MID: a point that is absent
// from its own output
template <typename T, int NI, int MID = -1>
struct Operands;

template <int NI, int MID>
struct Operands<float, NI, MID> {
    float x[NI];
    __device__ __forceinline__ explicit Operands(const float (&v)[NI]) {
#pragma unroll
        for (int j = 0; j < NI; j++) x[j] = v[j];
    }
    template <bool CVT = false, int NO>
    __device__ __forceinline__ float row(const Mat<float, NO, NI> &m, int i) const {
        float acc = m.d[i][0] * x[0];
#pragma unroll
        for (int j = 1; j < NI; j++)
            if (!absent<NO, NI>(i, j)) acc = fmaf(m.d[i][j], x[j], acc);
        return acc;
    }
};

template <int NI, int MID>
struct Operands<double, NI, MID> {
    int2 b[NI];
    int emax;
    bool wild;
    __device__ __forceinline__ explicit Operands(const double (&v)[NI]) {
        int mo = 0, mx = 0;
#pragma unroll
        for (int j = 0; j < NI; j++)
            if (j != MID) mo = max(mo, hi_abs(v[j]));
        mx = MID < 0 ? mo : max(mo, hi_abs(v[MID < 0 ? 0 : MID]));
        wild = out_of_range(mx) || (MID >= 0 && lone_middle(mx, mo));
        emax = max(mx >> 20, 64);
#pragma unroll
        for (int j = 0; j < NI; j++) {
            b[j] = split<60>(v[j], emax);
            // (the bits of x itself where they are not split)
            if (wild) b[j] = make_int2(__double2hiint(v[j]), __double2loint(v[j]));
        }
    }
    template <bool CVT = false, int NO>
    __device__ __forceinline__ double row(const Mat<double, NO, NI> &m, int i) const {
        if (wild) {
            double y = 0.0;
#pragma unroll
            for (int j = 0; j < NI; j++)
                if (!absent<NO, NI>(i, j)) y = fma(m.d[i][j], __hiloint2double(b[j].x, b[j].y), y);
            return y;
        }
        Fx s;
        s.clear();
#pragma unroll
        for (int j = 0; j < NI; j++)
            if (!absent<NO, NI>(i, j)) s.mad(m.a[i][j], b[j]);
        return CVT ? s.value_cvt(emax - m.s - 1051) : s.value(emax - m.s - 1051);
    }
};

// ---- launch constants -----------------------------------------------------------

constexpr int ipow(int q, int n) { return n == 0 ? 1 : q * ipow(q, n - 1); }

template <typename T, int ND, int Q>
struct Line {
    static constexpr int NV = ND + 2, NP = ipow(Q, ND), L = NP / Q, NFP = 2 * ND * L;
    Mat<T, Q, Q + 2> grad;      // corrected derivative from (u, common lo, hi)
    Mat<T, 2, Q> interp;        // values at the low and high end
    Mat<T, 2, Q + 2> gradend;   // interp of grad: the derivative at the ends
    Mat<T, Q, Q + 2> div;       // derivative less own lift, from (F, Fc lo, hi)
    unsigned char fpt[ND][L][2];

    // First point of line l of direction d, and the distance of its points
    __device__ static __forceinline__ int stride(int d) { return d == 0 ? 1 : d == 1 ? Q : Q * Q; }
    __device__ static __forceinline__ int base(int d, int l) {
        return d == 0 ? l * Q : d == 1 ? (l / Q) * (Q * Q) + l % Q : l;
    }
};

// One thread's outputs of the divergence: the Q points of x-line l, from the
// fluxes of all directions along their lines and (LIFT) the common flux at the
// lines' ends.  Line of direction d > 0 through point i of x-line l:
template <int ND, int Q>
struct Cross {
    int line, row;      // and the point's place on it
    __device__ __forceinline__ Cross(int d, int l, int i) {
        const int y = l % Q, z = l / Q;
        row = d == 1 ? y : z;
        line = d == 1 ? (ND == 3 ? z * Q + i : i) : y * Q + i;
    }
};

// ---- kernels ------------------------------------------------------------------

// Elements and threads of a block of the kernels that keep elements in shared
// memory.  64 or 32 bytes of a variable's row per block (whole sectors), so
// that the gradients of two or three blocks' elements fit an SM; the groups of
// threads of one element (NT/E) divide the lines and points of an element into
// nearly full rounds (p = 3 hexahedra, FP64: 48 groups for 48 lines).
template <typename T, int ND, int Q>
struct Tile {
    static constexpr int E = 64 / (int)sizeof(T) / (ND == 3 && Q == 5 ? 2 : 1);
    static constexpr int NT = ND == 2 ? 256 : (sizeof(T) == 8 && Q == 4) ? 384 : 256;
    static constexpr int G = NT / E, MINB = NT == 384 ? 2 : 3;
};

// Rows of a matrix from a column on; ld in bytes, below 2^32 (checked on the
// host), so that a row's address is one multiply-add
template <typename T>
struct Rows {
    T *p;
    unsigned ld;
    __device__ __forceinline__ T &operator()(unsigned row) const {
        return *reinterpret_cast<T *>(
            reinterpret_cast<uintptr_t>(p) + (unsigned long long)row * ld);
    }
    __device__ __forceinline__ Rows at(int64_t col) const { return Rows{p + col, ld}; }
};

// u at both ends of every line.  A warp takes a line of 32 elements, of one
// variable (SPLIT: too few lines to fill the GPU otherwise) or of all, which
// saves most of the index arithmetic; the lines of one block of elements are
// consecutive, so that the three reads of a point are near each other in time.
constexpr int TE_WARPS = 8;

template <typename T, int ND, int Q, bool SPLIT>
__global__ void __launch_bounds__(TE_WARPS * 32)
te_interp_kernel(const __grid_constant__ Line<T, ND, Q> P, int64_t neles, unsigned nchunk,
                 Rows<const T> u, Rows<T> f) {
    b200::dependent_entry(u.p, f.p);
    using K = Line<T, ND, Q>;
    constexpr int NV = K::NV, VS = SPLIT ? NV : 1;
    const int lane = threadIdx.x & 31;
    const unsigned blk = blockIdx.x / nchunk;
    const int t = (int)(blockIdx.x - blk * nchunk) * TE_WARPS + (threadIdx.x >> 5);
    if (t >= VS * ND * K::L || (int64_t)blk * 32 + lane >= neles) return;
    const int v0 = t % VS, d = t / VS / K::L, l = t / VS % K::L;
    const int p0 = K::base(d, l), st = K::stride(d);
    const int64_t col = ((int64_t)blk * NV + v0) * 32 + lane;
    const T *pu[Q];
    T *pf[2];
#pragma unroll
    for (int i = 0; i < Q; i++) pu[i] = &u.at(col)(p0 + i * st);
#pragma unroll
    for (int e = 0; e < 2; e++) pf[e] = &f.at(col)(P.fpt[d][l][e]);
#pragma unroll
    for (int v = 0; v < NV / VS; v++) {
        T x[Q];
#pragma unroll
        for (int i = 0; i < Q; i++) x[i] = pu[i][v * 32];
        const Operands<T, Q> b(x);
#pragma unroll
        for (int e = 0; e < 2; e++) pf[e][v * 32] = b.template row<true>(P.interp, e);
    }
}

// Fluxes of one element in shared memory, component c of point p at
// sm[(c NPS + p) E], and the common flux of flux point q at ends[(v NFS + q) E];
// NPS and NFS odd, so that two neighbouring components or points lie in
// different halves of the banks.
template <typename T, int ND, int Q, int E>
struct SmemFlux {
    static constexpr int NV = ND + 2, NPS = ipow(Q, ND) | 1,
                         NFS = (2 * ND * ipow(Q, ND - 1)) | 1;
    const Line<T, ND, Q> &P;
    const T *sm, *ends;     // + element
    int v;
    __device__ __forceinline__ const T *at(int d, int p) const {
        return sm + ((d * NV + v) * NPS + p) * E;
    }
    __device__ __forceinline__ const T *end_at(int d, int l, int e) const {
        return ends + (v * NFS + P.fpt[d][l][e]) * E;
    }
    __device__ __forceinline__ T flux(int d, int p) const { return *at(d, p); }
    __device__ __forceinline__ T end(int d, int l, int e) const { return *end_at(d, l, e); }
    // value j of line l of direction d: its points, then its ends
    __device__ __forceinline__ const T *on(int d, int l, int j) const {
        return j < Q ? at(d, P.base(d, l) + j * P.stride(d)) : end_at(d, l, j - Q);
    }
};

// Exponents of the lines of an element in shared memory, as the products take
// them (-1: the line is formed by FMAs, its values left as they are); the
// variables next to each other, so that the groups of a warp, which take
// neighbouring ones, meet no bank twice
template <int ND, int Q, int E>
struct LineExp {
    static constexpr int NV = ND + 2, L = ipow(Q, ND - 1), N = ND * NV * L * E;
    int *p;             // + element
    __device__ __forceinline__ int &operator()(int d, int l, int v) const {
        return p[((d * L + l) * NV + v) * E];
    }
};

// The values of a line (LIFT: with its ends) in fixed point over their largest
// magnitude, in their own places: every value is an operand of one line's
// outputs alone
template <bool LIFT, int ND, int Q, int E>
__device__ __forceinline__ void fix_line(const SmemFlux<double, ND, Q, E> &g,
                                         const LineExp<ND, Q, E> &ex, int d, int l) {
    constexpr int N = LIFT ? Q + 2 : Q;
    double x[N];
    int mx = 0, mo = 0;
#pragma unroll
    for (int j = 0; j < N; j++) {
        x[j] = *g.on(d, l, j);
        mx = max(mx, hi_abs(x[j]));
        if (j != middle(Q)) mo = max(mo, hi_abs(x[j]));
    }
    const bool wild = out_of_range(mx) || (middle(Q) >= 0 && lone_middle(mx, mo));
    const int emax = max(mx >> 20, 64);
    ex(d, l, g.v) = wild ? -1 : emax;
    if (wild) return;
#pragma unroll
    for (int j = 0; j < N; j++)
        *reinterpret_cast<int2 *>(const_cast<double *>(g.on(d, l, j))) = split<60>(x[j], emax);
}

// All lines of the thread's element, over its G groups of threads: a line of
// every variable a group where that fills the rounds as well (p = 3 hexahedra),
// which saves index arithmetic, else a line and variable
template <bool LIFT, int G, int ND, int Q, int E>
__device__ __forceinline__ void fix_lines(SmemFlux<double, ND, Q, E> g,
                                          const LineExp<ND, Q, E> &ex, int grp) {
    constexpr int NV = ND + 2, L = ipow(Q, ND - 1), NL = ND * L;
    if constexpr ((NL + G - 1) / G * NV <= (NL * NV + G - 1) / G) {
        for (int t = grp; t < NL; t += G)
#pragma unroll 1
            for (g.v = 0; g.v < NV; g.v++) fix_line<LIFT>(g, ex, t / L, t % L);
    } else {
        for (int t = grp; t < NL * NV; t += G) {
            g.v = t % NV;
            fix_line<LIFT>(g, ex, t / NV / L, t / NV % L);
        }
    }
}
template <bool LIFT, int G, int ND, int Q, int E>
__device__ __forceinline__ void fix_lines(const SmemFlux<float, ND, Q, E> &,
                                          const LineExp<ND, Q, E> &, int) {}

// The divergence at the points of x-line l from the element's fluxes (and,
// LIFT, common fluxes) in shared memory
template <bool LIFT, int ND, int Q, int E>
__device__ __forceinline__ void smem_div(const Line<float, ND, Q> &P,
                                         const SmemFlux<float, ND, Q, E> &g,
                                         const LineExp<ND, Q, E> &, int l, float (&y)[Q]) {
    constexpr int N = LIFT ? Q + 2 : Q;
#pragma unroll
    for (int i = 0; i < Q; i++) y[i] = 0.0f;
#pragma unroll
    for (int j = 0; j < N; j++) {
        const float x = *g.on(0, l, j);
#pragma unroll
        for (int i = 0; i < Q; i++)
            if (!absent<Q, Q + 2>(i, j)) y[i] += P.div.d[i][j] * x;
    }
#pragma unroll
    for (int d = 1; d < ND; d++)
#pragma unroll
        for (int i = 0; i < Q; i++) {
            const Cross<ND, Q> c(d, l, i);
#pragma unroll
            for (int j = 0; j < N; j++)
                if (!absent<Q, Q + 2>(c.row, j)) y[i] += P.div.d[c.row][j] * *g.on(d, c.line, j);
        }
}

// One output whose lines are not all in fixed point: FP64 FMAs for those that are not
template <bool LIFT, int ND, int Q, int E>
__device__ __noinline__ double wild_div(const Line<double, ND, Q> &P, SmemFlux<double, ND, Q, E> g,
                                        LineExp<ND, Q, E> ex, int l, int i) {
    constexpr int N = LIFT ? Q + 2 : Q;
    double y = 0.0;
#pragma unroll 1
    for (int d = 0; d < ND; d++) {
        const Cross<ND, Q> c(d, l, i);
        const int line = d ? c.line : l, row = d ? c.row : i, e = ex(d, line, g.v);
        Fx s;
        s.clear();
        double f = 0.0;
#pragma unroll 1
        for (int j = 0; j < N; j++) {
            const double *x = g.on(d, line, j);
            if (absent<Q, Q + 2>(row, j)) continue;
            if (e < 0)
                f = fma(P.div.d[row][j], *x, f);
            else
                s.mad(P.div.a[row][j], *reinterpret_cast<const int2 *>(x));
        }
        y += e < 0 ? f : s.value_cvt(e - P.div.s - 1051);
    }
    return y;
}

template <bool LIFT, int ND, int Q, int E>
__device__ __forceinline__ void smem_div(const Line<double, ND, Q> &P,
                                         const SmemFlux<double, ND, Q, E> &g,
                                         const LineExp<ND, Q, E> &ex, int l, double (&y)[Q]) {
    constexpr int N = LIFT ? Q + 2 : Q;
    const auto fixed = [&](int d, int line, int j) {
        return *reinterpret_cast<const int2 *>(g.on(d, line, j));
    };
    Fx s[Q];
#pragma unroll
    for (int i = 0; i < Q; i++) s[i].clear();
#pragma unroll
    for (int j = 0; j < N; j++) {
        const int2 b = fixed(0, l, j);
#pragma unroll
        for (int i = 0; i < Q; i++)
            if (!absent<Q, Q + 2>(i, j)) s[i].mad(P.div.a[i][j], b);
    }
    const int e0 = ex(0, l, g.v);
    bool wild = false;
#pragma unroll
    for (int i = 0; i < Q; i++) {
        long long t[ND] = {s[i].total()};
        int e[ND] = {e0}, top = e0, low = e0;
#pragma unroll
        for (int d = 1; d < ND; d++) {
            const Cross<ND, Q> c(d, l, i);
            Fx r;
            r.clear();
            // (an absent entry is zero)
#pragma unroll
            for (int j = 0; j < N; j++) r.mad(P.div.a[c.row][j], fixed(d, c.line, j));
            t[d] = r.total();
            e[d] = ex(d, c.line, g.v);
            top = max(top, e[d]);
            low = min(low, e[d]);
        }
        long long sum = 0;
#pragma unroll
        for (int d = 0; d < ND; d++) sum += t[d] >> min(top - e[d], 63);
        y[i] = b200::fixed_to_f64(sum, top - P.div.s - 1051);
        wild |= low < 0;
    }
    if (wild) {
#pragma unroll
        for (int i = 0; i < Q; i++) y[i] = wild_div<LIFT>(P, g, ex, l, i);
    }
}

// The same at point p alone, from the values as they are: in two dimensions
// there are few lines for the threads of an element, and a point each, over its
// own operands' exponent, is a shorter chain than the x-line's (40 x 40 cells at
// p = 3, where the kernel is one chain of latencies)
template <int ND, int Q, int E>
__device__ __forceinline__ double smem_div_point(const Line<double, ND, Q> &P,
                                                 const SmemFlux<double, ND, Q, E> &g, int p) {
    double x[ND][Q + 2];
    int row[ND], mx = 0;
#pragma unroll
    for (int d = 0; d < ND; d++) {
        const int st = P.stride(d), b = p - (row[d] = p / st % Q) * st;
        const int l = d == 0 ? p / Q : d == 1 ? p / (Q * Q) * Q + p % Q : b;
#pragma unroll
        for (int j = 0; j < Q + 2; j++) {
            x[d][j] = j < Q ? g.flux(d, b + j * st) : g.end(d, l, j - Q);
            if (!absent<Q, Q + 2>(row[d], j)) mx = max(mx, hi_abs(x[d][j]));
        }
    }
    if (out_of_range(mx)) {
        double y = 0.0;
#pragma unroll
        for (int d = 0; d < ND; d++)
#pragma unroll
            for (int j = 0; j < Q + 2; j++)
                if (!absent<Q, Q + 2>(row[d], j)) y = fma(P.div.d[row[d]][j], x[d][j], y);
        return y;
    }
    const int emax = max(mx >> 20, 64);
    Fx s;
    s.clear();
#pragma unroll
    for (int d = 0; d < ND; d++)
#pragma unroll
        for (int j = 0; j < Q + 2; j++)
            // (an absent value may be of any size)
            if (!absent<Q, Q + 2>(row[d], j))
                s.mad(P.div.a[row[d]][j], split<58>(x[d][j], emax));
    return s.value_cvt(emax - P.div.s - 1049);
}

// The gradient in physical space, (1/|J|) S^T tg
template <int ND, typename T>
__device__ __forceinline__ void grad_to_phys(const T s[ND][ND], T rcp, const T tg[ND][ND + 2],
                                             T gr[ND][ND + 2]) {
#pragma unroll
    for (int i = 0; i < ND; i++) {
        T k[ND];
#pragma unroll
        for (int d = 0; d < ND; d++) k[d] = rcp * s[d][i];
#pragma unroll
        for (int v = 0; v < ND + 2; v++) {
            T acc = k[0] * tg[0][v];
#pragma unroll
            for (int d = 1; d < ND; d++) acc += k[d] * tg[d][v];
            gr[i][v] = acc;
        }
    }
}

// The flux ft in reference space into the element's shared memory (sme + c NPS
// E: component c of the point)
template <typename T, int ND, bool DIAG, int STRIDE>
__device__ __forceinline__ void put_tflux(T *sme, const T s[ND][ND], const T ft[ND][ND + 2]) {
#pragma unroll
    for (int v = 0; v < ND + 2; v++)
#pragma unroll
        for (int i = 0; i < ND; i++) {
            T acc = s[i][DIAG ? i : 0] * ft[DIAG ? i : 0][v];
#pragma unroll
            for (int k = 1; k < ND; k++)
                if (!DIAG) acc += s[i][k] * ft[k][v];
            sme[(i * (ND + 2) + v) * STRIDE] = acc;
        }
}

// facemask: bit 2 d + end, the faces whose gradient is wanted on any element;
// refgrad: it stays in reference space (the interface kernels transform it).
// r may be u, and gf's first component may be c: every element's values are
// read before they are written.
//
// What bounds it (p = 3 hexahedra, FP64): the flux, 105 FP64 operations a point
// on the narrow FP64 unit, and about as much issue time for the lines on the
// integer pipes; the blocks of an SM are in different phases, so that the two
// run side by side.
template <typename T, int ND, int Q, bool DIAG>
__global__ void __launch_bounds__((Tile<T, ND, Q>::NT), (Tile<T, ND, Q>::MINB))
te_gradflux_kernel(const __grid_constant__ Line<T, ND, Q> P, int64_t neles, b200::GasK<T> gas,
                   Rows<const T> u, Rows<const T> c, Rows<T> gf, unsigned facemask, int refgrad,
                   ElemGeom<T> geo, Rows<T> r) {
    b200::dependent_entry(u.p, c.p, gf.p, r.p);
    using K = Line<T, ND, Q>;
    constexpr int NV = K::NV, NP = K::NP, L = K::L, NFP = K::NFP, NPS = NP | 1;
    constexpr int E = Tile<T, ND, Q>::E, G = Tile<T, ND, Q>::G;
    constexpr bool FIXED = sizeof(T) == 8;
    constexpr int VU = FIXED ? 1 : NV;      // unrolling over the variables
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T *sm = reinterpret_cast<T *>(smem_raw);

    const int el = threadIdx.x % E, grp = threadIdx.x / E;
    const int64_t e = (int64_t)blockIdx.x * E + el;
    const bool live = e < neles;
    const int64_t col0 = soa_off(live ? e : 0, 0, NV);
    u = u.at(col0);
    c = c.at(col0);
    gf = gf.at(col0);
    r = r.at(col0);
    T *const sme = sm + el;
    const LineExp<ND, Q, E> ex{reinterpret_cast<int *>(sm + ND * NV * NPS * E) + el};

    // The corrected gradient along every line; for a diagonal metric, already
    // in physical space (unless it is wanted in reference space)
    T sd[ND] = {};
    if (DIAG && live) {
#pragma unroll
        for (int d = 0; d < ND; d++)
            sd[d] = geo.rcpdjac[e] * geo.smats[(int64_t)d * geo.lds + soa_off(e, d, ND)];
    }
    const bool scale = DIAG && !refgrad, own = DIAG || refgrad;
    for (int t = grp; t < ND * L; t += G) {
        const int d = t / L, l = t % L;
        const int p0 = K::base(d, l), st = K::stride(d);
        const int q0 = P.fpt[d][l][0], q1 = P.fpt[d][l][1];
        const T s = DIAG ? (d == 0 ? sd[0] : d == 1 ? sd[1] : sd[ND - 1]) : T(1);
        const T *pu[Q], *pc[2] = {&c(q0), &c(q1)};
        T *pg[2] = {&gf(d * NFP + q0), &gf(d * NFP + q1)};
#pragma unroll
        for (int i = 0; i < Q; i++) pu[i] = &u(p0 + i * st);
        T *out = sme + (d * NV * NPS + p0) * E;
#pragma unroll VU
        for (int v = 0; v < NV; v++) {
            T x[Q + 2];
#pragma unroll
            for (int i = 0; i < Q; i++) x[i] = live ? pu[i][v * 32] : T(0);
#pragma unroll
            for (int i = 0; i < 2; i++) x[Q + i] = live ? pc[i][v * 32] : T(0);
            const Operands<T, Q + 2, middle(Q)> b(x);
#pragma unroll
            for (int i = 0; i < Q; i++) {
                T y = b.row(P.grad, i);
                if (scale) y *= s;
                out[(v * NPS + i * st) * E] = y;
            }
            // The derivative along the line at its ends, where the metric
            // leaves it a component of its own.  (Where the first component's
            // rows are those of c, this thread alone reads the value that it
            // replaces.)
            if (own && live) {
#pragma unroll
                for (int i = 0; i < 2; i++)
                    if ((facemask >> (2 * d + i)) & 1) {
                        const T y = b.row(P.gradend, i);
                        pg[i][v * 32] = scale ? s * y : y;
                    }
            }
        }
    }
    __syncthreads();

    if (!DIAG && !refgrad) {
        for (int p = grp; p < NP; p += G) {
            T s[ND][ND] = {}, rcp = T(0), tg[ND][NV], gr[ND][NV];
            if (live) b200::elem_metrics<ND, T>(geo, NP, p, e, s, rcp, true);
#pragma unroll
            for (int d = 0; d < ND; d++)
#pragma unroll
                for (int v = 0; v < NV; v++) tg[d][v] = sme[((d * NV + v) * NPS + p) * E];
            grad_to_phys<ND, T>(s, rcp, tg, gr);
#pragma unroll
            for (int d = 0; d < ND; d++)
#pragma unroll
                for (int v = 0; v < NV; v++) sme[((d * NV + v) * NPS + p) * E] = gr[d][v];
        }
        __syncthreads();
    }

    // The gradient at the flux points that are read
    for (int t = grp; t < ND * L; t += G) {
        const int d = t / L, l = t % L;
        const unsigned need = (facemask >> (2 * d)) & 3;
        if (!need) continue;
        const int p0 = K::base(d, l), st = K::stride(d);
        const int q0 = P.fpt[d][l][0], q1 = P.fpt[d][l][1];
#pragma unroll 1
        for (int k = 0; k < ND; k++) {
            if (own && k == d) continue;
            const T *in = sme + (k * NV * NPS + p0) * E;
            T *pg[2] = {&gf(k * NFP + q0), &gf(k * NFP + q1)};
#pragma unroll VU
            for (int v = 0; v < NV; v++) {
                T x[Q];
#pragma unroll
                for (int i = 0; i < Q; i++) x[i] = in[(v * NPS + i * st) * E];
                const Operands<T, Q> b(x);
#pragma unroll
                for (int i = 0; i < 2; i++)
                    if (live && ((need >> i) & 1)) pg[i][v * 32] = b.row(P.interp, i);
            }
        }
    }
    __syncthreads();

    // The flux in reference space, in the place of the gradient
    for (int p = grp; p < NP; p += G) {
        T uu[NV], gr[ND][NV], ft[ND][NV], s[ND][ND] = {}, rcp = T(0);
        if (live) b200::elem_metrics<ND, T, DIAG>(geo, NP, p, e, s, rcp, !DIAG && refgrad);
        const T *pu = &u(p);
#pragma unroll
        for (int v = 0; v < NV; v++) uu[v] = live ? pu[v * 32] : T(1);
#pragma unroll
        for (int d = 0; d < ND; d++)
#pragma unroll
            for (int v = 0; v < NV; v++) gr[d][v] = sme[((d * NV + v) * NPS + p) * E];
        if (DIAG && refgrad) {
#pragma unroll
            for (int d = 0; d < ND; d++)
#pragma unroll
                for (int v = 0; v < NV; v++) gr[d][v] *= sd[d];
        } else if (refgrad) {
            T tg[ND][NV];
#pragma unroll
            for (int d = 0; d < ND; d++)
#pragma unroll
                for (int v = 0; v < NV; v++) tg[d][v] = gr[d][v];
            grad_to_phys<ND, T>(s, rcp, tg, gr);
        }
        b200::ns_flux<ND, T>(uu, gr, ft, gas);
        put_tflux<T, ND, DIAG, NPS * E>(sme + p * E, s, ft);
    }
    __syncthreads();
    // FP64: in fixed point over each line's largest flux (a value is an operand
    // of the outputs of a line, and is split once)
    if (FIXED) {
        fix_lines<false, G>(SmemFlux<T, ND, Q, E>{P, sme, nullptr, 0}, ex, grp);
        __syncthreads();
    }

    // The divergence along the lines of every direction
    for (int t = grp; t < NV * L; t += G) {
        const int v = t % NV, l = t / NV;
        const SmemFlux<T, ND, Q, E> g{P, sme, nullptr, v};
        T y[Q];
        smem_div<false>(P, g, ex, l, y);
#pragma unroll
        for (int i = 0; i < Q; i++)
            if (live) r.at(v * 32)(l * Q + i) = y[i];
    }
}

// Euler: flux at the points, divergence, lift and scaling.  r may be u.
template <typename T, int ND, int Q, bool DIAG>
__global__ void __launch_bounds__((Tile<T, ND, Q>::NT), (Tile<T, ND, Q>::MINB))
te_euler_kernel(const __grid_constant__ Line<T, ND, Q> P, int64_t neles, T gamma, Rows<const T> u,
                Rows<const T> fc, ElemGeom<T> geo, Rows<T> r) {
    b200::dependent_entry(u.p, fc.p, r.p);
    using K = Line<T, ND, Q>;
    constexpr int NV = K::NV, NP = K::NP, L = K::L, NFP = K::NFP;
    constexpr int E = Tile<T, ND, Q>::E, G = Tile<T, ND, Q>::G;
    using SF = SmemFlux<T, ND, Q, E>;
    constexpr int NPS = SF::NPS, NFS = SF::NFS;
    // (by points in two dimensions, FP64)
    constexpr bool POINTS = sizeof(T) == 8 && ND == 2, FIXED = sizeof(T) == 8 && !POINTS;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T *sm = reinterpret_cast<T *>(smem_raw);

    const int el = threadIdx.x % E, grp = threadIdx.x / E;
    const int64_t e = (int64_t)blockIdx.x * E + el;
    const bool live = e < neles;
    const int64_t col0 = soa_off(live ? e : 0, 0, NV);
    u = u.at(col0);
    fc = fc.at(col0);
    r = r.at(col0);
    T *const sme = sm + el, *const sce = sme + ND * NV * NPS * E;
    const LineExp<ND, Q, E> ex{
        reinterpret_cast<int *>(sm + (ND * NV * NPS + NV * NFS) * E) + el};

    // (from the last group on, so that in two dimensions other threads than
    // the points' take the flux points)
    for (int q = G - 1 - grp; q < NFP; q += G) {
        const T *pf = &fc(q);
#pragma unroll
        for (int v = 0; v < NV; v++) sce[(v * NFS + q) * E] = live ? pf[v * 32] : T(0);
    }
    for (int p = grp; p < NP; p += G) {
        T uu[NV], ft[ND][NV], s[ND][ND] = {}, rcp, pr, vel[ND];
        if (live) b200::elem_metrics<ND, T, DIAG>(geo, NP, p, e, s, rcp, false);
        const T *pu = &u(p);
#pragma unroll
        for (int v = 0; v < NV; v++) uu[v] = live ? pu[v * 32] : T(1);
        b200::inviscid_flux<ND, T>(uu, ft, pr, vel, gamma);
        put_tflux<T, ND, DIAG, NPS * E>(sme + p * E, s, ft);
    }
    __syncthreads();
    if (FIXED) {
        fix_lines<true, G>(SF{P, sme, sce, 0}, ex, grp);
        __syncthreads();
    }
    if (!live) return;

    if constexpr (POINTS) {
        for (int t = grp; t < NV * NP; t += G) {
            const int v = t % NV, p = t / NV;
            const T rj = geo.rcpdjac[(geo.linear >= b200::GEOM_PER_ELEMENT ? 0 : p * geo.ldr) + e];
            r.at(v * 32)(p) = -rj * smem_div_point(P, SF{P, sme, sce, v}, p);
        }
    } else {
    for (int t = grp; t < NV * L; t += G) {
        const int v = t % NV, l = t / NV;
        const SF g{P, sme, sce, v};
        T y[Q];
        smem_div<true>(P, g, ex, l, y);
#pragma unroll
        for (int i = 0; i < Q; i++) {
            const int p = l * Q + i;
            const T rj = geo.rcpdjac[(geo.linear >= b200::GEOM_PER_ELEMENT ? 0 : p * geo.ldr) + e];
            r.at(v * 32)(p) = -rj * y[i];
        }
    }
    }
}

// The lift at the points of x-line l from the common flux at its ends and at
// those of the lines across it; fc(d, line, end).  FP64: the two ends of the
// x-line over their own exponent, the others over theirs, and the two integer
// sums shifted to the larger, so that an output has its own operands' bits
template <int ND, int Q, typename F>
__device__ __forceinline__ void lift_line(const Line<float, ND, Q> &P, const F &fc, int l,
                                          float (&y)[Q]) {
#pragma unroll
    for (int i = 0; i < Q; i++) y[i] = 0.0f;
#pragma unroll
    for (int e = 0; e < 2; e++) {
        const float x = fc(0, l, e);
#pragma unroll
        for (int i = 0; i < Q; i++) y[i] += P.div.d[i][Q + e] * x;
    }
#pragma unroll
    for (int i = 0; i < Q; i++)
#pragma unroll
        for (int d = 1; d < ND; d++) {
            const Cross<ND, Q> c(d, l, i);
#pragma unroll
            for (int e = 0; e < 2; e++) y[i] += P.div.d[c.row][Q + e] * fc(d, c.line, e);
        }
}

template <int ND, int Q, typename F>
__device__ __forceinline__ void lift_line(const Line<double, ND, Q> &P, const F &fc, int l,
                                          double (&y)[Q]) {
    double x[2], c[Q][ND - 1][2];
    int row[ND - 1];
#pragma unroll
    for (int e = 0; e < 2; e++) x[e] = fc(0, l, e);
#pragma unroll
    for (int i = 0; i < Q; i++)
#pragma unroll
        for (int d = 1; d < ND; d++) {
            const Cross<ND, Q> cr(d, l, i);
            row[d - 1] = cr.row;
#pragma unroll
            for (int e = 0; e < 2; e++) c[i][d - 1][e] = fc(d, cr.line, e);
        }

    const int mx0 = max(hi_abs(x[0]), hi_abs(x[1])), e0 = max(mx0 >> 20, 64);
    int2 b0[2];
#pragma unroll
    for (int e = 0; e < 2; e++) b0[e] = split<60>(x[e], e0);
#pragma unroll
    for (int i = 0; i < Q; i++) {
        int mx = 0;
#pragma unroll
        for (int k = 0; k < 2 * (ND - 1); k++) mx = max(mx, hi_abs(c[i][k / 2][k % 2]));
        if (out_of_range(mx0) || out_of_range(mx)) {
            y[i] = fma(P.div.d[i][Q + 1], x[1], P.div.d[i][Q] * x[0]);
#pragma unroll
            for (int k = 0; k < 2 * (ND - 1); k++)
                y[i] = fma(P.div.d[row[k / 2]][Q + k % 2], c[i][k / 2][k % 2], y[i]);
            continue;
        }
        const int e1 = max(mx >> 20, 64), top = max(e0, e1);
        Fx s, r;
        s.clear();
        r.clear();
#pragma unroll
        for (int e = 0; e < 2; e++) s.mad(P.div.a[i][Q + e], b0[e]);
#pragma unroll
        for (int k = 0; k < 2 * (ND - 1); k++)
            r.mad(P.div.a[row[k / 2]][Q + k % 2], split<60>(c[i][k / 2][k % 2], e1));
        y[i] = b200::fixed_to_f64_cvt((s.total() >> min(top - e0, 63)) +
                                          (r.total() >> min(top - e1, 63)),
                                      top - P.div.s - 1051);
    }
}

// R = -(1/|J|) (R + M3 Fc): a warp takes an x-line and variable of 32 elements
template <typename T, int ND, int Q>
__global__ void __launch_bounds__(TE_WARPS * 32)
te_lift_kernel(const __grid_constant__ Line<T, ND, Q> P, int64_t neles, unsigned nchunk,
               Rows<const T> fc, const T *__restrict__ rcpdjac, int64_t ldj, Rows<T> r) {
    b200::dependent_entry(fc.p, r.p);
    using K = Line<T, ND, Q>;
    const int lane = threadIdx.x & 31;
    const unsigned blk = blockIdx.x / nchunk;
    const int t = (int)(blockIdx.x - blk * nchunk) * TE_WARPS + (threadIdx.x >> 5);
    const int64_t e = (int64_t)blk * 32 + lane;
    if (t >= K::NV * K::L || e >= neles) return;
    const int v = t % K::NV, l = t / K::NV;
    const int64_t col = ((int64_t)blk * K::NV + v) * 32 + lane;
    r = r.at(col);
    fc = fc.at(col);
    T old[Q], y[Q];
#pragma unroll
    for (int i = 0; i < Q; i++) old[i] = r(l * Q + i);
    lift_line(P, [&](int d, int line, int end) { return fc(P.fpt[d][line][end]); }, l, y);
#pragma unroll
    for (int i = 0; i < Q; i++) {
        const int p = l * Q + i;
        r(p) = -rcpdjac[p * ldj + e] * (y[i] + old[i]);
    }
}

// ---- host side ----------------------------------------------------------------

constexpr int QMAX = 5;

// The one-dimensional matrices in FP64, and the flux points of the lines
struct TeHandle {
    int ndims, q;
    double grad[QMAX * (QMAX + 2)], interp[2 * QMAX], div[QMAX * (QMAX + 2)];
    unsigned char fpt[3 * QMAX * QMAX * 2];
};

template <typename T, int ND, int Q>
Line<T, ND, Q> line_of(const TeHandle &h) {
    Line<T, ND, Q> p;
    set_mat(p.grad, h.grad);
    set_mat(p.interp, h.interp);
    double ge[2 * (Q + 2)];
    for (int e = 0; e < 2; e++)
        for (int j = 0; j < Q + 2; j++) {
            double x = 0.0;
            for (int i = 0; i < Q; i++) x += h.interp[e * Q + i] * h.grad[i * (Q + 2) + j];
            ge[e * (Q + 2) + j] = x;
        }
    set_mat(p.gradend, ge);
    set_mat(p.div, h.div, true);
    memcpy(p.fpt, h.fpt, sizeof(p.fpt));
    return p;
}

// fn(integral constants ND, Q) for the handle's shape
template <typename F>
bool with_shape(const TeHandle &h, F &&fn) {
#define B200_TE(nd, nq)                                                      \
    if (h.ndims == nd && h.q == nq) {                                        \
        fn(std::integral_constant<int, nd>(), std::integral_constant<int, nq>()); \
        return true;                                                         \
    }
    B200_TE(2, 3) B200_TE(2, 4) B200_TE(2, 5)
    B200_TE(3, 3) B200_TE(3, 4) B200_TE(3, 5)
#undef B200_TE
    return false;
}

template <typename Fn>
int opt_in(Fn fn, size_t smem) {
    return b200::check_cuda(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 (int)smem), "te: smem attribute");
}

// Shared memory of an element block: the fluxes, with ends the common flux, and
// in FP64 the lines' exponents
template <typename T, int ND, int Q>
constexpr size_t te_smem(bool ends) {
    using SF = SmemFlux<T, ND, Q, Tile<T, ND, Q>::E>;
    constexpr int E = Tile<T, ND, Q>::E;
    return (size_t)(ND * SF::NV * SF::NPS + (ends ? SF::NV * SF::NFS : 0)) * E * sizeof(T) +
           (sizeof(T) == 8 ? LineExp<ND, Q, E>::N * sizeof(int) : 0);
}

template <typename T>
int te_opt_in(const TeHandle &h) {
    int rc = 0;
    with_shape(h, [&](auto nd, auto nq) {
        constexpr int ND = nd(), Q = nq();
        constexpr size_t s = te_smem<T, ND, Q>(false), se = te_smem<T, ND, Q>(true);
        rc = opt_in(te_gradflux_kernel<T, ND, Q, true>, s);
        if (!rc) rc = opt_in(te_gradflux_kernel<T, ND, Q, false>, s);
        if (!rc) rc = opt_in(te_euler_kernel<T, ND, Q, true>, se);
        if (!rc) rc = opt_in(te_euler_kernel<T, ND, Q, false>, se);
    });
    return rc;
}

// Rows with a leading dimension of ld values, which has to fit the kernels'
// 32 bits of bytes
template <typename T>
bool rows(Rows<T> &r, T *p, int64_t ld) {
    r = Rows<T>{p, (unsigned)(ld * (int64_t)sizeof(T))};
    return ld >= 0 && ld * (int64_t)sizeof(T) < (1ll << 32);
}

int too_wide(const char *what) {
    return b200::set_error(B200_ERR_UNSUPPORTED, "%s: rows of 4 GiB and more", what);
}

int check_te(const void *handle, const char *what, std::initializer_list<const void *> ptrs) {
    if (!handle) return b200::set_error(B200_ERR_ARG, "%s: null handle", what);
    for (const void *p : ptrs)
        if (!p) return b200::set_error(B200_ERR_ARG, "%s: null pointer", what);
    return B200_OK;
}

template <typename T>
int te_interp(void *handle, int64_t neles, const T *u, int64_t ldu, T *f, int64_t ldf,
              cudaStream_t st) {
    int rc = check_te(handle, "te_interp", {u, f});
    if (rc || neles <= 0) return rc;
    const TeHandle &h = *(const TeHandle *)handle;
    Rows<const T> ur;
    Rows<T> fr;
    if (!rows(ur, u, ldu) || !rows(fr, f, ldf)) return too_wide("te_interp");
    with_shape(h, [&](auto nd, auto nq) {
        constexpr int ND = nd(), Q = nq();
        using K = Line<T, ND, Q>;
        const unsigned nblk = b200::ceil_div(neles, 32);
        // (a warp per line and variable below 16 warps an SM)
        const bool split = (int64_t)nblk * ND * K::L < b200::SM_COUNT * 16;
        const unsigned nchunk = b200::ceil_div(ND * K::L * (split ? K::NV : 1), TE_WARPS);
        const auto P = line_of<T, ND, Q>(h);
        if (split)
            b200::launch(te_interp_kernel<T, ND, Q, true>, nblk * nchunk, TE_WARPS * 32, 0, st, P, neles, nchunk, ur, fr);
        else
            b200::launch(te_interp_kernel<T, ND, Q, false>, nblk * nchunk, TE_WARPS * 32, 0, st, P, neles, nchunk, ur, fr);
    });
    B200_CHECK_LAUNCH("te_interp");
    return B200_OK;
}

int te_geom(int linear, const void *smats, const void *rcpdjac) {
    if (linear != b200::GEOM_STORED && linear != b200::GEOM_PER_ELEMENT &&
        linear != b200::GEOM_DIAGONAL)
        return b200::set_error(B200_ERR_ARG, "te: the metric terms must be stored");
    if (!smats || !rcpdjac) return b200::set_error(B200_ERR_ARG, "te: null metric terms");
    return B200_OK;
}

template <typename T>
int te_gradflux_ns(void *handle, int64_t neles, int linear, const b200_gas_t *gas, const T *u,
                   int64_t ldu, const T *c, int64_t ldc, T *gf, int64_t ldg, unsigned facemask,
                   int refgrad, const T *smats, int64_t lds, const T *rcpdjac, int64_t ldj, T *r,
                   int64_t ldr, cudaStream_t st) {
    int rc = check_te(handle, "te_gradflux", {gas, u, c, gf, r});
    if (!rc) rc = te_geom(linear, smats, rcpdjac);
    if (rc || neles <= 0) return rc;
    const TeHandle &h = *(const TeHandle *)handle;
    const auto g = b200::gas_consts<T>(*reinterpret_cast<const Gas *>(gas));
    if (g.shifted)
        return b200::set_error(B200_ERR_UNSUPPORTED, "te_gradflux: takes unshifted states");
    const auto geo = b200::make_geom<T>(linear, smats, lds, rcpdjac, ldj, nullptr, 0, nullptr, 0);
    Rows<const T> ur, cr;
    Rows<T> gr, rr;
    if (!rows(ur, u, ldu) || !rows(cr, c, ldc) || !rows(gr, gf, ldg) || !rows(rr, r, ldr))
        return too_wide("te_gradflux");
    with_shape(h, [&](auto nd, auto nq) {
        constexpr int ND = nd(), Q = nq(), NT = Tile<T, ND, Q>::NT;
        const unsigned grid = b200::ceil_div(neles, Tile<T, ND, Q>::E);
        constexpr size_t s = te_smem<T, ND, Q>(false);
        const auto P = line_of<T, ND, Q>(h);
        if (linear == b200::GEOM_DIAGONAL)
            b200::launch(te_gradflux_kernel<T, ND, Q, true>, grid, NT, s, st, P, neles, g, ur, cr, gr, facemask, refgrad, geo, rr);
        else
            b200::launch(te_gradflux_kernel<T, ND, Q, false>, grid, NT, s, st, P, neles, g, ur, cr, gr, facemask, refgrad, geo, rr);
    });
    B200_CHECK_LAUNCH("te_gradflux");
    return B200_OK;
}

template <typename T>
int te_euler(void *handle, int64_t neles, int linear, double gamma, const T *u, int64_t ldu,
             const T *fc, int64_t ldf, const T *smats, int64_t lds, const T *rcpdjac, int64_t ldj,
             T *r, int64_t ldr, cudaStream_t st) {
    int rc = check_te(handle, "te_euler", {u, fc, r});
    if (!rc) rc = te_geom(linear, smats, rcpdjac);
    if (rc || neles <= 0) return rc;
    const TeHandle &h = *(const TeHandle *)handle;
    const auto geo = b200::make_geom<T>(linear, smats, lds, rcpdjac, ldj, nullptr, 0, nullptr, 0);
    Rows<const T> ur, fr;
    Rows<T> rr;
    if (!rows(ur, u, ldu) || !rows(fr, fc, ldf) || !rows(rr, r, ldr)) return too_wide("te_euler");
    with_shape(h, [&](auto nd, auto nq) {
        constexpr int ND = nd(), Q = nq(), NT = Tile<T, ND, Q>::NT;
        const unsigned grid = b200::ceil_div(neles, Tile<T, ND, Q>::E);
        constexpr size_t s = te_smem<T, ND, Q>(true);
        const auto P = line_of<T, ND, Q>(h);
        if (linear == b200::GEOM_DIAGONAL)
            b200::launch(te_euler_kernel<T, ND, Q, true>, grid, NT, s, st, P, neles, (T)gamma, ur, fr, geo, rr);
        else
            b200::launch(te_euler_kernel<T, ND, Q, false>, grid, NT, s, st, P, neles, (T)gamma, ur, fr, geo, rr);
    });
    B200_CHECK_LAUNCH("te_euler");
    return B200_OK;
}

template <typename T>
int te_lift(void *handle, int64_t neles, const T *fc, int64_t ldf, const T *rcpdjac, int64_t ldj,
            T *r, int64_t ldr, cudaStream_t st) {
    int rc = check_te(handle, "te_lift", {fc, rcpdjac, r});
    if (rc || neles <= 0) return rc;
    const TeHandle &h = *(const TeHandle *)handle;
    Rows<const T> fr;
    Rows<T> rr;
    if (!rows(fr, fc, ldf) || !rows(rr, r, ldr)) return too_wide("te_lift");
    with_shape(h, [&](auto nd, auto nq) {
        constexpr int ND = nd(), Q = nq();
        using K = Line<T, ND, Q>;
        const unsigned nchunk = b200::ceil_div(K::NV * K::L, TE_WARPS);
        b200::launch(te_lift_kernel<T, ND, Q>, b200::ceil_div(neles, 32) * nchunk, TE_WARPS * 32, 0, st, line_of<T, ND, Q>(h), neles, nchunk, fr, rcpdjac, ldj, rr);
    });
    B200_CHECK_LAUNCH("te_lift");
    return B200_OK;
}

}  // namespace

extern "C" {

int b200_te_create(int ndims, int q, const double *grad, const double *interp, const double *div,
                   const int *fpt, void **handle) {
    if (!grad || !interp || !div || !fpt || !handle)
        return b200::set_error(B200_ERR_ARG, "te_create: null pointer");
    TeHandle *h = (TeHandle *)calloc(1, sizeof(TeHandle));
    if (!h) return b200::set_error(B200_ERR_STATE, "te_create: out of host memory");
    h->ndims = ndims;
    h->q = q;
    if (!with_shape(*h, [](auto, auto) {})) {
        free(h);
        return b200::set_error(B200_ERR_UNSUPPORTED, "te_create: %d-D, %d points a line", ndims, q);
    }
    // (finite, and with a row sum that the fixed-point form takes)
    double top = 0.0;
    for (int i = 0; i < q * (q + 2); i++) top = fmax(top, fmax(fabs(grad[i]), fabs(div[i])));
    bool fine = top >= 0.5 && top <= 1e6;
    for (int i = 0; i < q * (q + 2); i++) fine = fine && isfinite(grad[i]) && isfinite(div[i]);
    for (int i = 0; i < 2 * q; i++) fine = fine && fabs(interp[i]) <= 1e6;
    const int mid = (q / 2) * (q + 2) + q / 2;
    if (q & 1) fine = fine && grad[mid] == 0.0 && div[mid] == 0.0;
    const int nf = 2 * ndims * (ndims == 2 ? q : q * q);
    for (int i = 0; i < nf; i++) fine = fine && fpt[i] >= 0 && fpt[i] < nf;
    if (!fine) {
        free(h);
        return b200::set_error(B200_ERR_ARG, "te_create: operators out of range");
    }
    memcpy(h->grad, grad, sizeof(double) * q * (q + 2));
    memcpy(h->interp, interp, sizeof(double) * 2 * q);
    memcpy(h->div, div, sizeof(double) * q * (q + 2));
    for (int i = 0; i < nf; i++) h->fpt[i] = (unsigned char)fpt[i];
    int rc = te_opt_in<double>(*h);
    if (!rc) rc = te_opt_in<float>(*h);
    if (rc) {
        free(h);
        return rc;
    }
    *handle = h;
    return B200_OK;
}

int b200_te_destroy(void *handle) {
    free(handle);
    return B200_OK;
}

#define B200_TE_API(T, sfx)                                                                     \
    int b200_te_interp_##sfx(void *h, int64_t neles, const T *u, int64_t ldu, T *f, int64_t ldf, \
                             void *stream) {                                                    \
        return te_interp<T>(h, neles, u, ldu, f, ldf, (cudaStream_t)stream);                    \
    }                                                                                           \
    int b200_te_gradflux_ns_##sfx(void *h, int64_t neles, int linear, const b200_gas_t *gas,     \
                                  const T *u, int64_t ldu, const T *c, int64_t ldc, T *gf,      \
                                  int64_t ldg, unsigned facemask, int refgrad, const T *smats,  \
                                  int64_t lds, const T *rcpdjac, int64_t ldj, T *r,             \
                                  int64_t ldr, void *stream) {                                  \
        return te_gradflux_ns<T>(h, neles, linear, gas, u, ldu, c, ldc, gf, ldg, facemask,       \
                                 refgrad, smats, lds, rcpdjac, ldj, r, ldr,                     \
                                 (cudaStream_t)stream);                                         \
    }                                                                                           \
    int b200_te_euler_##sfx(void *h, int64_t neles, int linear, double gamma, const T *u,        \
                            int64_t ldu, const T *fc, int64_t ldf, const T *smats, int64_t lds, \
                            const T *rcpdjac, int64_t ldj, T *r, int64_t ldr, void *stream) {   \
        return te_euler<T>(h, neles, linear, gamma, u, ldu, fc, ldf, smats, lds, rcpdjac, ldj, r, \
                           ldr, (cudaStream_t)stream);                                          \
    }                                                                                           \
    int b200_te_lift_##sfx(void *h, int64_t neles, const T *fc, int64_t ldf, const T *rcpdjac,   \
                           int64_t ldj, T *r, int64_t ldr, void *stream) {                      \
        return te_lift<T>(h, neles, fc, ldf, rcpdjac, ldj, r, ldr, (cudaStream_t)stream);        \
    }

B200_TE_API(double, f64)
B200_TE_API(float, f32)

}  // extern "C"
