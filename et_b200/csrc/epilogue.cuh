// What the linears do with an accumulator: bias, tanh-GELU, fp16.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <cstdint>
#include "ptx.cuh"

namespace et {

// tanh-GELU of two values in packed fp16 arithmetic: 0.5 x (1 + tanh(x (c1 + c2 x^2))), six packed operations and
// one special-function op per pair, no conversion. The epilogue is bound by the conversion unit (fp32 <-> fp16
// conversions and special functions run at 16 per clock per SM): with the polynomial in fp32 and conversions
// around the tanh a 128 x 384 GELU tile took ~9000 clocks against ~4400 without GELU. The result is stored as fp16
// anyway; tanh saturates, so the rounding of its argument does not grow with |x| (an argument that overflows to
// infinity gives tanh = +-1, the correct limit).
__device__ __forceinline__ half2 gelu_tanh_h2(half2 x) {
    const half2 c1 = __float2half2_rn(0.7978845608028654f), c2 = __float2half2_rn(0.7978845608028654f * 0.044715f);
    const half2 u = __hmul2(x, __hfma2(__hmul2(x, x), c2, c1));
    uint32_t t;
    asm("tanh.approx.f16x2 %0, %1;" : "=r"(t) : "r"(*reinterpret_cast<const uint32_t*>(&u)));
    const half2 hx = __hmul2(x, __float2half2_rn(0.5f));
    return __hfma2(hx, *reinterpret_cast<const half2*>(&t), hx);
}

// One 32-column unit of an epilogue: its accumulators, then its results. The caller writes them under the 64-byte swizzle
// (16-byte chunk ^= (row / 2) % 4).
__device__ __forceinline__ void epi_load(uint32_t taddr, bool two, uint32_t (&acc)[32]) {
    if (two) {
        tmem_ld32(taddr, acc);
        tmem_ld_wait(acc);
    } else {
        uint32_t lo[16];
        tmem_ld16(taddr, lo);
        tmem_ld_wait(lo);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            acc[i] = lo[i];
            acc[16 + i] = 0u;
        }
    }
}
template <bool kGelu>
__device__ __forceinline__ void epi_convert_regs(const uint32_t (&acc)[32], const uint4 (&bv)[4], uint4 (&ov)[4]) {
    const half2* bh = reinterpret_cast<const half2*>(bv);
    half2* oh = reinterpret_cast<half2*>(ov);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        if constexpr (kGelu) {
            // one conversion per pair: the accumulator is packed first and the bias is added in packed fp16
            oh[i] = gelu_tanh_h2(__hadd2(__floats2half2_rn(__uint_as_float(acc[2 * i]), __uint_as_float(acc[2 * i + 1])), bh[i]));
        } else {
            // Mixed-precision additions: the sums of the converted bias, without its conversions. What an epilogue's warps execute competes
            // with the issuing warps of the resident kernel (with conversions 17771 x 768 -> 2304 at 75 % took 33.5 instead of 32.8 us).
            float lo, hi;
            asm("{\n.reg .b16 l, h;\nmov.b32 {l, h}, %2;\nadd.rn.f32.f16 %0, l, %3;\nadd.rn.f32.f16 %1, h, %4;\n}"
                : "=f"(lo), "=f"(hi)
                : "r"(reinterpret_cast<const uint32_t*>(bv)[i]), "f"(__uint_as_float(acc[2 * i])), "f"(__uint_as_float(acc[2 * i + 1])));
            oh[i] = __floats2half2_rn(lo, hi);
        }
    }
}

}  // namespace et
