// Four consecutive columns of a row in a lane's registers: loads and stores of 256 bits in FP64 (128 in
// FP32) on a boundary of that width.
#pragma once

#include "device.cuh"

namespace fereg {

template <class T>
struct V4 {
    T a, b, c, d;
};
__device__ __forceinline__ V4<double> ld4(const double* p) {
    V4<double> v;
    asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v.a), "=d"(v.b), "=d"(v.c), "=d"(v.d) : "l"(p));
    return v;
}
__device__ __forceinline__ V4<float> ld4(const float* p) {
    const float4 x = __ldg(reinterpret_cast<const float4*>(p));
    return V4<float>{x.x, x.y, x.z, x.w};
}
// L2-coherent load of values written earlier in the same pass sequence (t)
__device__ __forceinline__ V4<double> ld4cg(const double* p) {
    V4<double> v;
    asm("ld.global.cg.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v.a), "=d"(v.b), "=d"(v.c), "=d"(v.d) : "l"(p));
    return v;
}
__device__ __forceinline__ V4<float> ld4cg(const float* p) {
    const float4 x = __ldcg(reinterpret_cast<const float4*>(p));
    return V4<float>{x.x, x.y, x.z, x.w};
}
__device__ __forceinline__ void st4(double* p, const V4<double>& v) {
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(v.a), "d"(v.b), "d"(v.c), "d"(v.d) : "memory");
}
__device__ __forceinline__ void st4(float* p, const V4<float>& v) {
    *reinterpret_cast<float4*>(p) = make_float4(v.a, v.b, v.c, v.d);
}
template <class T>
__device__ __forceinline__ void add4(V4<T>& s, const V4<T>& v) {
    s.a += v.a;
    s.b += v.b;
    s.c += v.c;
    s.d += v.d;
}
template <class T>
__device__ __forceinline__ void fma4(V4<T>& s, T w, const V4<T>& v) {
    s.a += w * v.a;
    s.b += w * v.b;
    s.c += w * v.c;
    s.d += w * v.d;
}
// to shared memory (16-byte boundaries)
__device__ __forceinline__ void st4s(double* p, const V4<double>& v) {
    reinterpret_cast<double2*>(p)[0] = make_double2(v.a, v.b);
    reinterpret_cast<double2*>(p)[1] = make_double2(v.c, v.d);
}
__device__ __forceinline__ void st4s(float* p, const V4<float>& v) {
    *reinterpret_cast<float4*>(p) = make_float4(v.a, v.b, v.c, v.d);
}

}  // namespace fereg
