// Typed vector loads of the quantisers' inputs (fp32, bf16, fp16), widened to fp32.
#pragma once
#include "common.cuh"
#include <type_traits>

namespace cinn {

template <typename T> struct Elem;
template <> struct Elem<__nv_bfloat16> {
    static __device__ __forceinline__ float to_f(__nv_bfloat16 v) { return __bfloat162float(v); }
    static __device__ __forceinline__ void load8(const __nv_bfloat16* p, float (&v)[8]) {
        uint4 r = *reinterpret_cast<const uint4*>(p);
        uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            v[2 * i] = __uint_as_float(w[i] << 16);
            v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
        }
    }
    static __device__ __forceinline__ void load4(const __nv_bfloat16* p, float (&v)[4]) {
        uint2 r = *reinterpret_cast<const uint2*>(p);
        v[0] = __uint_as_float(r.x << 16); v[1] = __uint_as_float(r.x & 0xffff0000u);
        v[2] = __uint_as_float(r.y << 16); v[3] = __uint_as_float(r.y & 0xffff0000u);
    }
};
template <> struct Elem<__half> {
    static __device__ __forceinline__ float to_f(__half v) { return __half2float(v); }
    static __device__ __forceinline__ void load8(const __half* p, float (&v)[8]) {
        uint4 r = *reinterpret_cast<const uint4*>(p);
        const __half2* h = reinterpret_cast<const __half2*>(&r);
#pragma unroll
        for (int i = 0; i < 4; ++i) { float2 f = __half22float2(h[i]); v[2 * i] = f.x; v[2 * i + 1] = f.y; }
    }
    static __device__ __forceinline__ void load4(const __half* p, float (&v)[4]) {
        uint2 r = *reinterpret_cast<const uint2*>(p);
        const __half2* h = reinterpret_cast<const __half2*>(&r);
        float2 a = __half22float2(h[0]), b = __half22float2(h[1]);
        v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
    }
};
template <> struct Elem<float> {
    static __device__ __forceinline__ float to_f(float v) { return v; }
    static __device__ __forceinline__ void load8(const float* p, float (&v)[8]) {
        float4 a = *reinterpret_cast<const float4*>(p);
        float4 b = *reinterpret_cast<const float4*>(p + 4);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    }
    static __device__ __forceinline__ void load4(const float* p, float (&v)[4]) {
        float4 a = *reinterpret_cast<const float4*>(p);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    }
};

// eight elements as they are stored
template <typename T> struct Raw8 { uint4 a; };
template <> struct Raw8<float> { float4 a, b; };

template <typename T>
__device__ __forceinline__ Raw8<T> load_raw8(const T* p) {
    Raw8<T> r;
    if constexpr (sizeof(T) == 4) {
        r.a = __ldcs(reinterpret_cast<const float4*>(p));
        r.b = __ldcs(reinterpret_cast<const float4*>(p) + 1);
    } else {
        r.a = __ldcs(reinterpret_cast<const uint4*>(p));
    }
    return r;
}
template <typename T>
__device__ __forceinline__ Raw8<T> zero_raw8() {
    Raw8<T> r;
    if constexpr (sizeof(T) == 4) { r.a = make_float4(0.f, 0.f, 0.f, 0.f); r.b = r.a; }
    else r.a = make_uint4(0u, 0u, 0u, 0u);
    return r;
}
template <typename T>
__device__ __forceinline__ void unpack_raw8(const Raw8<T>& r, float (&v)[8]) {
    if constexpr (sizeof(T) == 4) {
        v[0] = r.a.x; v[1] = r.a.y; v[2] = r.a.z; v[3] = r.a.w; v[4] = r.b.x; v[5] = r.b.y; v[6] = r.b.z; v[7] = r.b.w;
    } else if constexpr (std::is_same<T, __nv_bfloat16>::value) {
        const uint32_t w[4] = {r.a.x, r.a.y, r.a.z, r.a.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) { v[2 * i] = __uint_as_float(w[i] << 16); v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u); }
    } else {
        const __half2* h = reinterpret_cast<const __half2*>(&r.a);
#pragma unroll
        for (int i = 0; i < 4; ++i) { const float2 f = __half22float2(h[i]); v[2 * i] = f.x; v[2 * i + 1] = f.y; }
    }
}

}  // namespace cinn
