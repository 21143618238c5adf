// Small arithmetic helpers: two fp32 operations per instruction, three-way maximum, exponential, warp maximum.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <cstdint>

namespace et {

// 2^x on the special-function unit; results flush to zero below 2^-126.
__device__ __forceinline__ float ex2_fast(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
// The larger of two values; not a number if one of them is not.
__device__ __forceinline__ float max_nan(float a, float b) {
    float d;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
    return d;
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    float2 d;
    asm("{\n.reg .b64 x, y, z, w;\nmov.b64 x, {%2, %3};\nmov.b64 y, {%4, %5};\nmov.b64 z, {%6, %7};\n"
        "fma.rn.f32x2 w, x, y, z;\nmov.b64 {%0, %1}, w;\n}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    float2 d;
    asm("{\n.reg .b64 x, y, w;\nmov.b64 x, {%2, %3};\nmov.b64 y, {%4, %5};\nadd.rn.f32x2 w, x, y;\nmov.b64 {%0, %1}, w;\n}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    float2 d;
    asm("{\n.reg .b64 x, y, w;\nmov.b64 x, {%2, %3};\nmov.b64 y, {%4, %5};\nmul.rn.f32x2 w, x, y;\nmov.b64 {%0, %1}, w;\n}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
// Largest value of a warp, in every lane.
__device__ __forceinline__ float warp_max(float v) {
    float m;
    asm("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(m) : "f"(v));
    return m;
}

}  // namespace et
