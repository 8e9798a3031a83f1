// Metric terms of the elements, as the element kernels read them.
#pragma once

#include <type_traits>

#include "common.cuh"
#include "physics.cuh"

namespace b200 {

template <typename T>
struct ElemGeom {
    const T *smats;  int64_t lds;
    const T *rcpdjac; int64_t ldr;
    const T *verts;  int64_t ldv;
    const T *upts;   int64_t ldup;
    int linear;
};

// Geometry modes (the `linear` argument of the element kernels)
enum { GEOM_STORED = 0, GEOM_VERTICES = 1, GEOM_PER_ELEMENT = 2, GEOM_DIAGONAL = 3 };

// Metric terms at solution point `upt` of element `e`: from the vertices
// (GEOM_VERTICES, multilinear elements), from the stored per-point smats
// and 1/|J| (GEOM_STORED), or from one stored set per element
// (GEOM_PER_ELEMENT: affine elements, whose Jacobian is constant, keep
// only the rows of their first point: io-shapes (ndims, 1, ndims, neles)
// and (1, neles)).  DIAG (GEOM_DIAGONAL: per-element terms of elements
// aligned with the axes, whose off-diagonal S are zero) is a compile-time
// form of the kernels: the two transforms then take 30 FP64 operations a
// point in 3-D instead of 99 (tflux_ns at 26^3 elements, p = 3: 416 us
// before both the shared flux expressions and this form).
template <int ND, typename T, bool DIAG = false>
__device__ __forceinline__ void elem_metrics(const ElemGeom<T> &g, int nupts, int upt,
                                             int64_t e, T s[ND][ND], T &rcpdjac,
                                             bool need_rcp) {
    if (DIAG || g.linear >= GEOM_PER_ELEMENT) {
        nupts = 1;
        upt = 0;
    }
    if (DIAG) {
#pragma unroll
        for (int i = 0; i < ND; i++)
#pragma unroll
            for (int j = 0; j < ND; j++)
                s[i][j] = i == j ? g.smats[(int64_t)i * g.lds + soa_off(e, i, ND)] : T(0);
        rcpdjac = need_rcp ? g.rcpdjac[e] : T(0);
    } else if (g.linear == GEOM_VERTICES) {
        T V[1 << ND][ND], x[ND], d;
#pragma unroll
        for (int v = 0; v < (1 << ND); v++)
#pragma unroll
            for (int k = 0; k < ND; k++) V[v][k] = g.verts[v * g.ldv + soa_off(e, k, ND)];
#pragma unroll
        for (int k = 0; k < ND; k++) x[k] = g.upts[upt * g.ldup + k];
        linear_smats<ND, T>(V, x, s, d);
        rcpdjac = need_rcp ? T(1) / d : T(0);
    } else {
#pragma unroll
        for (int i = 0; i < ND; i++)
#pragma unroll
            for (int j = 0; j < ND; j++)
                s[i][j] = g.smats[(int64_t)(i * nupts + upt) * g.lds + soa_off(e, j, ND)];
        rcpdjac = need_rcp ? g.rcpdjac[(int64_t)upt * g.ldr + e] : T(0);
    }
}

template <typename T>
inline ElemGeom<T> make_geom(int linear, const T *smats, int64_t lds, const T *rcpdjac, int64_t ldr,
                      const T *verts, int64_t ldv, const T *upts, int64_t ldup) {
    ElemGeom<T> g;
    g.smats = smats; g.lds = lds;
    g.rcpdjac = rcpdjac; g.ldr = ldr;
    g.verts = verts; g.ldv = ldv;
    g.upts = upts; g.ldup = ldup;
    g.linear = linear;
    return g;
}

// A launch over the number of dimensions and the diagonal form of the
// metrics, both compile-time: fn(integral constants); false for ndims other
// than 2 or 3
template <typename F>
bool with_form(int ndims, int linear, F &&fn) {
    using b2 = std::integral_constant<int, 2>;
    using b3 = std::integral_constant<int, 3>;
    if (ndims == 2 && linear == GEOM_DIAGONAL)
        fn(b2(), std::true_type());
    else if (ndims == 2)
        fn(b2(), std::false_type());
    else if (ndims == 3 && linear == GEOM_DIAGONAL)
        fn(b3(), std::true_type());
    else if (ndims == 3)
        fn(b3(), std::false_type());
    else
        return false;
    return true;
}

}  // namespace b200
