// Complex arithmetic on float2 / double2 and small helpers shared by all kernels.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace ifdda {

// Programmatic dependent launch.  A kernel launched with it may start while
// the kernel before it on the stream is still finishing: its blocks run their
// prologue (constant tables, prefetches of constant data), then pdl_wait()
// blocks until the previous kernel has completed and its writes are visible
// to all its loads, also where L1 held the line from before (probed with plain,
// read-only and L2 loads, the reader resident while the writer's grid read and
// then wrote the words, 1 to 5 kernels apart: none old of 4e10 each).  So the
// status and the state of a solve are read with plain loads: from L2 instead,
// the same line for every warp, they made FP32 solves on 64^3 7% slower.
// pdl_trigger() lets the next kernel's blocks be scheduled once every block
// of this one has called it.  Without the launch attribute both are no-ops.
//
// Every block calls pdl_wait() before it reads anything the previous kernel
// wrote, before it triggers and before it exits.  So a kernel runs beside its
// direct predecessor only, and everything before that one is complete when it
// starts.  Triggering first instead lets a whole chain of waiting kernels
// occupy the SMs, and the blocks of a small grid then land where there is
// room, several on one SM: a product on 24^3 in FP64 took 19.8 instead of
// 12.8 us, one on 32^3 in FP32 21.7 instead of 14.0 us (64^3: no difference).
// A kernel whose vectors the next one reads through the read-only path (ldg)
// triggers after it has written them, so that they do not change while the
// reader runs.  The reader's early return of a finished solve stands between
// the wait and its first such load: without it the compiler, which takes what
// is read this way for constant, might move the load ahead of the wait.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename T> struct cvec;
template <> struct cvec<float> { using type = float2; };
template <> struct cvec<double> { using type = double2; };
template <typename T> using cplx = typename cvec<T>::type;

__host__ __device__ __forceinline__ float2 mk(float a, float b) { return make_float2(a, b); }
__host__ __device__ __forceinline__ double2 mk(double a, double b) { return make_double2(a, b); }

template <class C> __host__ __device__ __forceinline__ C cadd(C a, C b) { return mk(a.x + b.x, a.y + b.y); }
template <class C> __host__ __device__ __forceinline__ C csub(C a, C b) { return mk(a.x - b.x, a.y - b.y); }
// The products are written as the fused multiply-adds they become, so that
// every instance of the code rounds alike (left to the compiler, which of the
// two products is fused may differ from one copy of a loop body to the next).
template <class C> __host__ __device__ __forceinline__ C cmul(C a, C b) {
    return mk(fma(a.x, b.x, -(a.y * b.y)), fma(a.x, b.y, a.y * b.x));
}
// conj(a) * b
template <class C> __host__ __device__ __forceinline__ C cmulc(C a, C b) {
    return mk(a.x * b.x + a.y * b.y, a.x * b.y - a.y * b.x);
}
template <class C, class S> __host__ __device__ __forceinline__ C cscale(C a, S s) { return mk(a.x * s, a.y * s); }
template <class C> __host__ __device__ __forceinline__ C cconj(C a) { return mk(a.x, -a.y); }
// Two complex FP32 values, real parts and imaginary parts together: the
// element of the mat-vec's y and z passes in FP32.  Sums and products by
// constants of both values are one packed instruction (add / mul / fma
// .f32x2), which takes one issue slot for the work of two; loads and stores
// move 16 bytes.
struct __align__(16) cpair {
    float2 re, im;
};
// scalar type and twiddle (plain complex) type of an FFT element
template <class E> struct elem_traits;
template <> struct elem_traits<float2> { using T = float; using W = float2; };
template <> struct elem_traits<double2> { using T = double; using W = double2; };
template <> struct elem_traits<cpair> { using T = float; using W = float2; };
// element of the y and z passes for scalar T
template <class T> struct yz_elem;
template <> struct yz_elem<float> { using type = cpair; };
template <> struct yz_elem<double> { using type = double2; };

template <class E> __host__ __device__ __forceinline__ E czero() {
    if constexpr (sizeof(typename elem_traits<E>::W) == sizeof(E)) {
        using T = typename elem_traits<E>::T;
        return mk(T(0), T(0));
    } else {
        return E{make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
    }
}

// a + s i b, s real
template <class C, class T> __host__ __device__ __forceinline__ C cfma_i(C a, C b, T s) {
    return mk(fma(b.y, -s, a.x), fma(b.x, s, a.y));
}
#if defined(__CUDA_ARCH__)
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
#else  // host compilation pass only: never run
__device__ inline float2 add2(float2 a, float2) { return a; }
__device__ inline float2 mul2(float2 a, float2) { return a; }
__device__ inline float2 fma2(float2 a, float2, float2) { return a; }
#endif
// a - b, as one packed fma (the product is exact, so it rounds as a subtraction)
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return fma2(b, make_float2(-1.f, -1.f), a); }
__device__ __forceinline__ cpair cadd(cpair a, cpair b) { return cpair{add2(a.re, b.re), add2(a.im, b.im)}; }
__device__ __forceinline__ cpair csub(cpair a, cpair b) { return cpair{sub2(a.re, b.re), sub2(a.im, b.im)}; }
__device__ __forceinline__ cpair cscale(cpair a, float s) {
    const float2 ss = make_float2(s, s);
    return cpair{mul2(a.re, ss), mul2(a.im, ss)};
}
// by one complex number for both values (a table twiddle): plain products,
// whose operands need no packing
__device__ __forceinline__ cpair cmul(cpair a, float2 w) {
    return cpair{make_float2(fmaf(a.re.x, w.x, -(a.im.x * w.y)), fmaf(a.re.y, w.x, -(a.im.y * w.y))),
                 make_float2(fmaf(a.re.x, w.y, a.im.x * w.x), fmaf(a.re.y, w.y, a.im.y * w.x))};
}
// by a compile-time constant c + i s
template <class C, class T> __host__ __device__ __forceinline__ C cmulk(C a, T c, T s) {
    return mk(fma(a.x, c, -(a.y * s)), fma(a.x, s, a.y * c));
}
__device__ __forceinline__ cpair cmulk(cpair a, float c, float s) {
    const float2 c2 = make_float2(c, c), s2 = make_float2(s, s), n2 = make_float2(-s, -s);
    return cpair{fma2(a.im, n2, mul2(a.re, c2)), fma2(a.im, c2, mul2(a.re, s2))};
}
// a + SIGN i b
template <int SIGN, class C> __host__ __device__ __forceinline__ C cadd_i(C a, C b) {
    return SIGN > 0 ? mk(a.x - b.y, a.y + b.x) : mk(a.x + b.y, a.y - b.x);
}
template <int SIGN> __device__ __forceinline__ cpair cadd_i(cpair a, cpair b) {
    return SIGN > 0 ? cpair{sub2(a.re, b.im), add2(a.im, b.re)} : cpair{add2(a.re, b.im), sub2(a.im, b.re)};
}
// a + s b, s real
template <class C, class T> __host__ __device__ __forceinline__ C cfma_s(C a, C b, T s) {
    return mk(fma(b.x, s, a.x), fma(b.y, s, a.y));
}
__device__ __forceinline__ cpair cfma_s(cpair a, cpair b, float s) {
    const float2 ss = make_float2(s, s);
    return cpair{fma2(b.re, ss, a.re), fma2(b.im, ss, a.im)};
}

__device__ __forceinline__ cpair cfma_i(cpair a, cpair b, float s) {
    const float2 ss = make_float2(s, s), ns = make_float2(-s, -s);
    return cpair{fma2(b.im, ns, a.re), fma2(b.re, ss, a.im)};
}

// Global load that asks L2 to fetch the PF bytes (128 or 256; 0: a plain
// load) around the address from DRAM (PTX ld .L2::<PF>B): for narrow rows
// that neighbouring blocks read at the same time, the DRAM accesses become
// wider bursts.
template <int PF> __device__ __forceinline__ float2 ld_l2pf(const float2* p) {
    float2 v;
    if constexpr (PF == 256)
        asm volatile("ld.global.L2::256B.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
    else if constexpr (PF == 128)
        asm volatile("ld.global.L2::128B.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
    else
        v = *p;
    return v;
}
template <int PF> __device__ __forceinline__ double2 ld_l2pf(const double2* p) {
    double2 v;
    if constexpr (PF == 256)
        asm volatile("ld.global.L2::256B.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
    else if constexpr (PF == 128)
        asm volatile("ld.global.L2::128B.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
    else
        v = *p;
    return v;
}

template <int PF> __device__ __forceinline__ cpair ld_l2pf(const cpair* p) {
    cpair v;
    if constexpr (PF == 256)
        asm volatile("ld.global.L2::256B.v4.f32 {%0, %1, %2, %3}, [%4];"
                     : "=f"(v.re.x), "=f"(v.re.y), "=f"(v.im.x), "=f"(v.im.y)
                     : "l"(p));
    else
        v = *p;
    return v;
}

__host__ __device__ __forceinline__ double2 to_d(float2 a) { return make_double2(a.x, a.y); }
__host__ __device__ __forceinline__ double2 to_d(double2 a) { return a; }
template <class C> __host__ __device__ __forceinline__ C from_d(double2 a);
template <> __host__ __device__ __forceinline__ float2 from_d<float2>(double2 a) { return make_float2((float)a.x, (float)a.y); }
template <> __host__ __device__ __forceinline__ double2 from_d<double2>(double2 a) { return a; }

__host__ __device__ __forceinline__ double2 zdiv(double2 a, double2 b) {
    // a / b with scaling against overflow (Smith's algorithm)
    if (fabs(b.x) >= fabs(b.y)) {
        double r = b.y / b.x, den = b.x + b.y * r;
        return make_double2((a.x + a.y * r) / den, (a.y - a.x * r) / den);
    } else {
        double r = b.x / b.y, den = b.x * r + b.y;
        return make_double2((a.x * r + a.y) / den, (a.y * r - a.x) / den);
    }
}
__host__ __device__ __forceinline__ bool zisnull(double2 a) { return a.x == 0.0 && a.y == 0.0; }
__host__ __device__ __forceinline__ double zabs(double2 a) { return hypot(a.x, a.y); }

}  // namespace ifdda
