// Shared helpers for the pyfrb200 CUDA library.
//
// Data layout (identical to the reference CUDA backend, SoA size 32,
// pyfr/backends/base/types.py:58-75 and pyfr/backends/cuda/base.py:55-59):
// a field of io-shape (nrow, nvars, neles) is stored row-major with
// `ld` scalars per row; inside a row, elements are grouped in blocks of 32
// and the variables of one block are contiguous:
//     a[row*ld + (e/32)*32*nvars + v*32 + e%32]
// so a warp that reads one variable of 32 consecutive elements touches one
// contiguous 256-byte (FP64) segment.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#define B200_SOASZ 32

namespace b200 {

// Record an error message for b200_get_last_error(); returns the code.
int set_error(int code, const char *fmt, ...);
int check_cuda(cudaError_t err, const char *what);

__host__ __device__ __forceinline__ int64_t soa_off(int64_t e, int v, int nv) {
    return (e / B200_SOASZ) * B200_SOASZ * nv + v * B200_SOASZ + (e % B200_SOASZ);
}

// Gather-index load from an int32 or int64 view mapping.
__device__ __forceinline__ int64_t load_ix(const void *map, int ix64, int64_t i) {
    return ix64 ? __ldg(static_cast<const long long *>(map) + i)
                : (int64_t)__ldg(static_cast<const int *>(map) + i);
}

// SMs of the GPU (GB300), for the sizes at which a grid fills it
constexpr int SM_COUNT = 152;

// Launches by programmatic dependent launch: a kernel may be set up while the
// one before it on the stream ends, and waits at dependent_entry until the
// kernels before have finished and their writes are visible, which closes most
// of the gap between short kernels (the 2-D vortex on 40 x 40 cells at p = 3,
// FP64, 100 kernels a call: 372 -> 352 us; the largest steps are the same).
// The kernels do not let their dependents start earlier than that: with
// griddepcontrol.launch_dependents at the start of every kernel the same call
// took 523 us, the waiting blocks standing in the way of running ones.  Only the
// pieces of one large tensor-core operator do (early_dependents: their
// operator's copy into shared memory then overlaps: a step of 12^3 hexahedra at
// p = 4, eight pieces a right-hand side, 589 -> 536 us).
//
// Every kernel that is launched so calls dependent_entry first, with every
// pointer to memory that other kernels write: no access through it can be
// moved before the wait, whatever the qualifiers of the pointer.
template <typename... P>
__device__ __forceinline__ void dependent_entry(P &...p) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    ((void)([&] { asm volatile("" : "+l"(p)); }()), ...);
}

__device__ __forceinline__ void early_dependents() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// brief: a kernel whose length the gap before it matters to
template <typename... P, typename... A>
inline void launch_if(bool brief, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem,
                      cudaStream_t st, A &&...a) {
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c = {};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = st;
    c.attrs = attr;
    // (in captured graphs, where the chains of short kernels are: a single
    // kernel launched from the host again and again, a 20 x 40 tensor-core
    // apply of 24 us, takes 1.4% longer so)
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    c.numAttrs = brief && cudaStreamIsCapturing(st, &cap) == cudaSuccess &&
                 cap == cudaStreamCaptureStatusActive;
    // (a failure is left for the caller's cudaGetLastError)
    (void)cudaLaunchKernelEx(&c, kernel, static_cast<P>(a)...);
}

// (beyond 32 blocks an SM nothing is gained: a step of 32^3 hexahedra is as
// long, and its graph's instantiation up to 0.3 ms longer)
template <typename... P, typename... A>
inline void launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                   A &&...a) {
    launch_if((uint64_t)grid.x * grid.y * grid.z <= SM_COUNT * 32, kernel, grid, block, smem, st,
              static_cast<A &&>(a)...);
}

inline unsigned ceil_div(int64_t a, int64_t b) { return (unsigned)((a + b - 1) / b); }

// FP32 <-> FP64 conversions on the integer pipes.  GB300's FP64 unit is
// narrow (about 2 operations per clock per SM) and executes the hardware
// conversions too, so a bandwidth-bound kernel that widens and narrows
// every element is FP64-bound.  These build the result from the IEEE 754
// binary32/binary64 encodings (1/8/23 and 1/11/52 bits, exponent biases 127
// and 1023) for the normal range and for signed zeros, which is where
// solution and RHS values live; subnormal, infinite and NaN operands take
// the hardware conversion.  Both are exact in the sense of IEEE 754: the
// widening is exact and the narrowing rounds to nearest, ties to even.
__device__ __forceinline__ double widen_f32(float f) {
    const uint32_t u = __float_as_uint(f);
    const uint32_t a = u & 0x7fffffffu;
    const uint64_t s = (uint64_t)(u & 0x80000000u) << 32;
    if (a - 0x00800000u < 0x7f000000u)  // biased exponent in [1, 254]
        return __longlong_as_double((long long)(s | ((uint64_t)a << 29) +
                                                         ((uint64_t)(1023 - 127) << 52)));
    if (a == 0) return __longlong_as_double((long long)s);
    return (double)f;
}

__device__ __forceinline__ float narrow_f64(double d) {
    const uint64_t u = (uint64_t)__double_as_longlong(d);
    const uint64_t a = u & 0x7fffffffffffffffull;
    const uint32_t s = (uint32_t)(u >> 32) & 0x80000000u;
    // Binary64 exponents 897..1150 are the binary32 normals 1..254
    if (a - (897ull << 52) < (254ull << 52)) {
        uint32_t r = (uint32_t)((a >> 29) - (896ull << 23));
        const uint32_t rem = (uint32_t)a & 0x1fffffffu;
        r += (uint32_t)(rem > 0x10000000u) | ((uint32_t)(rem == 0x10000000u) & r);
        return __uint_as_float(s | r);
    }
    if (a == 0) return __uint_as_float(s);
    return (float)d;
}

// A double in [2^-100, 2^100) by magnitude to a float by truncation, and a
// normal float to a double, on the integer pipes (the encodings above).
__device__ __forceinline__ float trunc_f64(double d) {
    const uint32_t hi = (uint32_t)__double2hiint(d), lo = (uint32_t)__double2loint(d);
    return __uint_as_float((hi & 0x80000000u) |
                           (__funnelshift_l(lo, hi & 0x7fffffffu, 3) - (896u << 23)));
}

__device__ __forceinline__ double widen_normal(float f) {
    const uint32_t u = __float_as_uint(f);
    return __hiloint2double((int)((u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + (896u << 20))),
                            (int)(u << 29));
}

// Whether |d| lies in [2^-100, 2^100): there a single-precision estimate of
// 1/d or 1/sqrt(d) and its argument are normal floats
__device__ __forceinline__ bool mid_range(double d) {
    return ((uint32_t)__double2hiint(d) & 0x7fffffffu) - ((1023u - 100) << 20) < (200u << 20);
}

// 1/d in FP64 without an IEEE division: a single-precision estimate
// (rcp.approx.ftz.f32 of the truncated operand, relative error e about
// 2^-22) refined by one step of Chebyshev's third-order iteration,
// r (1 + e + e^2) with e = 1 - d r, whose error e^3 is below FP64's
// rounding: 3 FP64 FMAs where an IEEE division spends about ten FP64
// operations, fix-up tests and a slow path, on a GPU whose FP64 unit is
// narrow (2 operations per clock and SM).  Operands outside mid_range, zeros,
// infinities and NaNs take the IEEE division.
__device__ __forceinline__ double rcp_f64(double d) {
    if (!mid_range(d)) return 1.0 / d;
    float r0;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"(trunc_f64(d)));
    const double r = widen_normal(r0);
    const double e = fma(-d, r, 1.0);
    return fma(r, fma(e, e, e), r);
}

// sqrt(x) in FP64: the single-precision estimate y of 1/sqrt(x), h = x y and
// two Newton (Heron) steps with the fixed slope y/2, s <- s + (x - s^2) y/2,
// which take the error from 2^-22 to below FP64's rounding: 5 FP64
// operations.  Operands outside mid_range, negative ones, zeros, infinities
// and NaNs take the IEEE square root.
__device__ __forceinline__ double sqrt_f64(double x) {
    if (!mid_range(x) || __double2hiint(x) < 0) return sqrt(x);
    float y0;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y0) : "f"(trunc_f64(x)));
    const double y2 = widen_normal(0.5f * y0);
    double s = x * widen_normal(y0);
    s = fma(fma(-s, s, x), y2, s);
    return fma(fma(-s, s, x), y2, s);
}

// The reciprocal and square root of the flux kernels: in FP64 the forms
// above, in FP32 the IEEE operations
__device__ __forceinline__ double rcp(double x) { return rcp_f64(x); }
__device__ __forceinline__ float rcp(float x) { return 1.0f / x; }
__device__ __forceinline__ double root(double x) { return sqrt_f64(x); }
__device__ __forceinline__ float root(float x) { return sqrtf(x); }
// a/b (in FP64 within one rounding more than the IEEE quotient's)
__device__ __forceinline__ double quot(double a, double b) { return a * rcp_f64(b); }
__device__ __forceinline__ float quot(float a, float b) { return a / b; }

}  // namespace b200

// Status codes of the C ABI
#define B200_OK 0
#define B200_ERR_CUDA 1
#define B200_ERR_ARG 2
#define B200_ERR_UNSUPPORTED 3
#define B200_ERR_STATE 4

#define B200_CHECK_LAUNCH(what)                                              \
    do {                                                                     \
        cudaError_t e_ = cudaGetLastError();                                 \
        if (e_ != cudaSuccess) return b200::check_cuda(e_, what);            \
    } while (0)
