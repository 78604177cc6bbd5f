// nbc_math.cuh -- small vector algebra for the engine's kernels.
//
// The operations mirror the helpers the reference's kernels use
// (src/type.h:10-305): Length() returns 0 when the squared length is at or
// below 1e-32, Quat2IvDCM is the body->world rotation of a quaternion stored
// (x, y, z, w) with w the scalar part, Quat2DCM its transpose.
#pragma once
#include <cuda_runtime.h>

namespace nbc {

template <typename R> struct V3 { R x, y, z; };

template <typename R> __host__ __device__ __forceinline__ V3<R> v3(R x, R y, R z) { return {x, y, z}; }

// Sums and products with their rounding written out: which product of a sum is
// fused is otherwise the compiler's choice, and changes with the code around
// it; the step's results should not change with the kernel it runs in.  Sums
// of vectors are not fused with anything; what is fused says so (fma1: a s +
// c; fma2: a b + c d, the first product fused; fma3; dot, cross, len_floor).
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double sub_rn(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ float sub_rn(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
template <typename R> __device__ __forceinline__ R fma2(R a, R b, R c, R d) {   // a b + c d
    return fma_rn(a, b, mul_rn(c, d));
}
template <typename R> __device__ __forceinline__ R fma3(R a, R b, R c, R d, R e, R f) {   // a b + c d + e f
    return fma_rn(e, f, fma2(a, b, c, d));
}
template <typename R> __device__ __forceinline__ V3<R> operator+(V3<R> a, V3<R> b) {
    return {add_rn(a.x, b.x), add_rn(a.y, b.y), add_rn(a.z, b.z)};
}
template <typename R> __device__ __forceinline__ V3<R> operator-(V3<R> a, V3<R> b) {
    return {sub_rn(a.x, b.x), sub_rn(a.y, b.y), sub_rn(a.z, b.z)};
}
template <typename R> __device__ __forceinline__ V3<R> operator-(V3<R> a) { return {-a.x, -a.y, -a.z}; }
template <typename R> __device__ __forceinline__ V3<R> operator*(R s, V3<R> a) {
    return {mul_rn(s, a.x), mul_rn(s, a.y), mul_rn(s, a.z)};
}
template <typename R> __device__ __forceinline__ V3<R> fma1(R s, V3<R> a, V3<R> c) {   // s a + c
    return {fma_rn(s, a.x, c.x), fma_rn(s, a.y, c.y), fma_rn(s, a.z, c.z)};
}
template <typename R> __device__ __forceinline__ V3<R> fma2(R s, V3<R> a, R t, V3<R> b) {   // s a + t b
    return {fma2(s, a.x, t, b.x), fma2(s, a.y, t, b.y), fma2(s, a.z, t, b.z)};
}
template <typename R> __device__ __forceinline__ R dot(V3<R> a, V3<R> b) { return fma3(a.x, b.x, a.y, b.y, a.z, b.z); }
template <typename R> __device__ __forceinline__ V3<R> cross(V3<R> a, V3<R> b) {
    return {fma2(a.y, b.z, -a.z, b.y), fma2(a.z, b.x, -a.x, b.z), fma2(a.x, b.y, -a.y, b.x)};
}
template <typename R> __device__ __forceinline__ R len_floor(V3<R> a) {
    const R t = dot(a, a);
    return t > R(1e-32) ? sqrt(t) : R(0);
}
// the same with the y product fused first (the boundary laws' lengths)
template <typename R> __device__ __forceinline__ R len2_yx(V3<R> a) { return fma3(a.y, a.y, a.x, a.x, a.z, a.z); }
template <typename R> __device__ __forceinline__ R len_floor_yx(V3<R> a) {
    const R t = len2_yx(a);
    return t > R(1e-32) ? sqrt(t) : R(0);
}
template <typename R, typename S> __host__ __device__ __forceinline__ V3<R> cvt(V3<S> a) {
    return {R(a.x), R(a.y), R(a.z)};
}

// Real4 storage type of each precision
template <typename R> struct Vec4;
template <> struct Vec4<float> { using T = float4; };
template <> struct Vec4<double> { using T = double4; };
template <typename R> using R4 = typename Vec4<R>::T;

template <typename R> __device__ __forceinline__ V3<R> xyz(R4<R> a) { return {a.x, a.y, a.z}; }
__device__ __forceinline__ V3<double> xyzd(double4 a) { return {a.x, a.y, a.z}; }
template <typename R> __device__ __forceinline__ R4<R> pack(V3<R> a, R w) {
    R4<R> o; o.x = a.x; o.y = a.y; o.z = a.z; o.w = w; return o;
}

// 32-byte records in one access (sm_100 loads and stores 256 bits a lane): a
// gather of 32 scattered records costs the L1 one tag lookup per lane instead
// of two.  p is 32-byte aligned.  The asm is volatile so that it keeps its
// place between barriers; nothing written by the same kernel is read this way
// unless a barrier lies between.
__device__ __forceinline__ double4 ld32(const double4* p) {
    double4 v;
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ void st32(double4* p, double4 v) {
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(v.x), "d"(v.y), "d"(v.z), "d"(v.w) : "memory");
}
// two adjacent Real4 (a contact slot, a spring record): 32 bytes in FP32,
// two 32-byte halves in FP64
__device__ __forceinline__ void ld_pair(const float4* p, float4& a, float4& b) {
    asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
                 : "l"(p));
}
__device__ __forceinline__ void ld_pair(const double4* p, double4& a, double4& b) {
    a = ld32(p);
    b = ld32(p + 1);
}
__device__ __forceinline__ void st_pair(float4* p, float4 a, float4 b) {
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(a.x), "f"(a.y), "f"(a.z),
                 "f"(a.w), "f"(b.x), "f"(b.y), "f"(b.z), "f"(b.w)
                 : "memory");
}
__device__ __forceinline__ void st_pair(double4* p, double4 a, double4 b) {
    st32(p, a);
    st32(p + 1, b);
}

// a 32-byte record of eight integers
__device__ __forceinline__ void ld_rec(const int4* p, int4& a, int4& b) {
    asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w)
                 : "l"(p));
}
__device__ __forceinline__ void st_rec(int4* p, int4 a, int4 b) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(a.x), "r"(a.y), "r"(a.z),
                 "r"(a.w), "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w)
                 : "memory");
}

// body->world rotation (Quat2IvDCM, src/type.h:238-250) applied to u
__device__ __forceinline__ V3<double> rot_b2w(double4 q, V3<double> u) {
    const double m00 = __fma_rn(q.w, q.w, fma3(q.x, q.x, -q.y, q.y, -q.z, q.z));
    const double m11 = __fma_rn(q.w, q.w, fma3(-q.x, q.x, q.y, q.y, -q.z, q.z));
    const double m22 = __fma_rn(q.w, q.w, fma3(-q.x, q.x, -q.y, q.y, q.z, q.z));
    const double m10 = 2.0 * fma2(q.x, q.y, q.z, q.w), m01 = 2.0 * fma2(q.x, q.y, -q.z, q.w);
    const double m20 = 2.0 * fma2(q.x, q.z, -q.y, q.w), m02 = 2.0 * fma2(q.x, q.z, q.y, q.w);
    const double m21 = 2.0 * fma2(q.y, q.z, q.x, q.w), m12 = 2.0 * fma2(q.y, q.z, -q.x, q.w);
    return {fma3(m00, u.x, m01, u.y, m02, u.z), fma3(m11, u.y, m10, u.x, m12, u.z),
            fma3(m20, u.x, m21, u.y, m22, u.z)};
}
// world->body rotation (Quat2DCM, src/type.h:223-236) applied to u
__device__ __forceinline__ V3<double> rot_w2b(double4 q, V3<double> u) {
    const double m00 = __fma_rn(q.w, q.w, fma3(q.x, q.x, -q.y, q.y, -q.z, q.z));
    const double m11 = __fma_rn(q.w, q.w, fma3(-q.x, q.x, q.y, q.y, -q.z, q.z));
    const double m22 = __fma_rn(q.w, q.w, fma3(-q.x, q.x, -q.y, q.y, q.z, q.z));
    const double m10 = 2.0 * fma2(q.x, q.y, -q.z, q.w), m01 = 2.0 * fma2(q.x, q.y, q.z, q.w);
    const double m20 = 2.0 * fma2(q.x, q.z, q.y, q.w), m02 = 2.0 * fma2(q.x, q.z, -q.y, q.w);
    const double m21 = 2.0 * fma2(q.y, q.z, -q.x, q.w), m12 = 2.0 * fma2(q.y, q.z, q.x, q.w);
    return {fma3(m00, u.x, m01, u.y, m02, u.z), fma3(m10, u.x, m11, u.y, m12, u.z),
            fma3(m20, u.x, m21, u.y, m22, u.z)};
}

}  // namespace nbc
