// Residual add + LayerNorm, in place: in_out <- LN(in_out + skip) * gamma + beta.
// Replaces kernels/skip_layernorm.cu:4-112 of the reference (both its kernels).
//
// Bandwidth kernel: 6*size bytes per row (read x, read skip, write). One warp owns a row, reads
// it with 16-byte loads into registers, reduces with shuffles only (no shared memory, no block
// barrier), does all arithmetic in fp32 (sum, two-pass variance, eps 1e-6 as the reference) and
// writes 16 bytes per lane. gamma/beta are re-read per row through the read-only cache.
#include <algorithm>
#include "common.h"

namespace et {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) v += __shfl_xor_sync(0xffffffffu, v, m);
    return v;
}

// Which operations round together is stated, not left to the compiler, so that a row's result does not depend on the kernel that
// reduces it: the subtraction of the mean is one rounding with sum / size, and so are the squares of a lane's first chunk with their
// sum; the products of the other chunks are rounded before they are added. (Left to the compiler, sizes known at compile time
// changed 1e-5 of the results by one fp16 rounding, and 24 layers made of that a relative difference of 1e-3.)
__device__ __forceinline__ float centred(float v, float sum, float inv_n) { return __fmaf_rn(-sum, inv_n, v); }
__device__ __forceinline__ float plus_square(float sq, float d, int chunk) {
    return chunk == 0 ? __fmaf_rn(d, d, sq) : __fadd_rn(sq, __fmul_rn(d, d));
}
__device__ __forceinline__ float inv_std(float sq, float inv_n) { return rsqrtf(__fmaf_rn(sq, inv_n, 1e-6f)); }
__device__ __forceinline__ float scaled(float d, float rstd, float g, float b) { return __fmaf_rn(__fmul_rn(d, rstd), g, b); }

template <int CH>  // 16-byte chunks per lane; covers size <= CH*256
__global__ void __launch_bounds__(256, (CH <= 4 ? 3 : 1)) skip_layernorm_vec(half* __restrict__ in_out,
                                                          const half* __restrict__ skip,
                                                          const half* __restrict__ gamma,
                                                          const half* __restrict__ beta, int num,
                                                          int size) {
    pdl_launch_dependents();
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarp = (gridDim.x * blockDim.x) >> 5;
    const int nchunk = size >> 3;
    const float inv_n = 1.0f / (float)size;
    for (int row = warp; row < num; row += nwarp) {
        uint4* xr = reinterpret_cast<uint4*>(in_out + (size_t)row * size);
        const uint4* sr = reinterpret_cast<const uint4*>(skip + (size_t)row * size);
        uint4 xv[CH], sv[CH];
#pragma unroll
        for (int i = 0; i < CH; ++i) {
            const int c = lane + 32 * i;
            if (c < nchunk) {
                xv[i] = xr[c];
                sv[i] = skip ? __ldcs(sr + c) : make_uint4(0u, 0u, 0u, 0u);   // no residual: plain LayerNorm of the row
            }
        }
        float v[CH][8];
        float sum = 0.f;
#pragma unroll
        for (int i = 0; i < CH; ++i) {
            const int c = lane + 32 * i;
            const half2* xh = reinterpret_cast<const half2*>(&xv[i]);
            const half2* sh = reinterpret_cast<const half2*>(&sv[i]);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float2 a = __half22float2(xh[j]), s = __half22float2(sh[j]);
                v[i][2 * j] = c < nchunk ? a.x + s.x : 0.f;
                v[i][2 * j + 1] = c < nchunk ? a.y + s.y : 0.f;
                sum += v[i][2 * j] + v[i][2 * j + 1];
            }
        }
        sum = warp_sum(sum);
        float sq = 0.f;
#pragma unroll
        for (int i = 0; i < CH; ++i) {
            const int c = lane + 32 * i;
#pragma unroll
            for (int j = 0; j < 8; ++j)
                if (c < nchunk) sq = plus_square(sq, centred(v[i][j], sum, inv_n), i);
        }
        const float rstd = inv_std(warp_sum(sq), inv_n);
#pragma unroll
        for (int i = 0; i < CH; ++i) {
            const int c = lane + 32 * i;
            if (c < nchunk) {
                const uint4 g = __ldg(reinterpret_cast<const uint4*>(gamma) + c);
                const uint4 b = __ldg(reinterpret_cast<const uint4*>(beta) + c);
                const half2* gh = reinterpret_cast<const half2*>(&g);
                const half2* bh = reinterpret_cast<const half2*>(&b);
                uint4 o;
                half2* oh = reinterpret_cast<half2*>(&o);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 gg = __half22float2(gh[j]), bb = __half22float2(bh[j]);
                    oh[j] = __floats2half2_rn(scaled(centred(v[i][2 * j], sum, inv_n), rstd, gg.x, bb.x),
                                              scaled(centred(v[i][2 * j + 1], sum, inv_n), rstd, gg.y, bb.y));
                }
                xr[c] = o;
            }
        }
    }
}

// Rows of exactly CH * 256 elements: the next row is requested before this one's reductions, by as many blocks as an SM holds
// without spills (at 1024 elements a third one spilled 144 bytes: 17.8 us instead of 12.3 for 16384 rows); sizes known at compile time
// leave the registers for it. What bounds it is memory (6.2 to 6.7 TB/s from 60000 rows on), or L2 where the operands come from the
// linear before. Against the kernel above, with operands in L2: 8192 x 256 3.5 -> 3.0 us, x 512 5.5 -> 4.3, x 768 7.1 -> 5.6, x 1024
// 9.2 -> 6.9, x 1280 16.9 -> 8.3, x 2048 22.2 -> 11.6; from memory: 17771 x 768 15.4 -> 14.2, x 1024 21.9 -> 18.3, x 2048 50 -> 35,
// 131072 x 768 95.5 -> 96, x 1024 132 -> 124, x 2048 304 -> 240. Without a residual 17771 x 768 13.1 -> 10.4, x 2048 45.7 -> 25.5.
// kOne, for few rows, which a chain of latencies bounds: a warp has one row and requests gamma and beta with it, not behind its reductions, and
// small blocks spread the rows over the SMs.
constexpr int row_blocks(int ch) { return ch <= 1 ? 6 : ch <= 2 ? 4 : ch <= 3 ? 3 : ch <= 6 ? 2 : 1; }   // per SM
template <int CH, bool kSkip, bool kOne>
__global__ void __launch_bounds__(256, kOne ? 1 : row_blocks(CH)) skip_layernorm_rows(half* __restrict__ in_out, const half* __restrict__ skip,
                                                                       const half* __restrict__ gamma, const half* __restrict__ beta, int num) {
    pdl_launch_dependents();
    pdl_wait();
    constexpr int kSize = CH * 256;
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarp = (gridDim.x * blockDim.x) >> 5;
    const size_t step = (size_t)nwarp * (kSize / 8);
    uint4* xr = reinterpret_cast<uint4*>(in_out) + (size_t)warp * (kSize / 8) + lane;
    const uint4* sr = reinterpret_cast<const uint4*>(skip) + (size_t)warp * (kSize / 8) + lane;
    uint4 xv[CH], sv[CH];
    auto load = [&]() {
#pragma unroll
        for (int i = 0; i < CH; ++i) {
            xv[i] = xr[32 * i];
            if constexpr (kSkip) sv[i] = __ldcs(sr + 32 * i);
        }
    };
    uint4 gv[CH], bv[CH];   // kOne
    if (warp < num) {
        load();
        if constexpr (kOne) {
#pragma unroll
            for (int i = 0; i < CH; ++i) {
                gv[i] = __ldg(reinterpret_cast<const uint4*>(gamma) + lane + 32 * i);
                bv[i] = __ldg(reinterpret_cast<const uint4*>(beta) + lane + 32 * i);
            }
        }
    }
    for (int row = warp; row < num; row += nwarp) {
        uint4* const out = xr;
        float v[CH][8];
        float sum = 0.f;
#pragma unroll
        for (int i = 0; i < CH; ++i) {
            const half2* xh = reinterpret_cast<const half2*>(&xv[i]);
            const half2* sh = reinterpret_cast<const half2*>(&sv[i]);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float2 a = __half22float2(xh[j]), s = kSkip ? __half22float2(sh[j]) : make_float2(0.f, 0.f);
                v[i][2 * j] = a.x + s.x;
                v[i][2 * j + 1] = a.y + s.y;
                sum += v[i][2 * j] + v[i][2 * j + 1];
            }
        }
        if constexpr (!kOne) {
            xr += step;
            sr += step;
            if (row + nwarp < num) load();
        }
        sum = warp_sum(sum);
        float sq = 0.f;
#pragma unroll
        for (int i = 0; i < CH; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) sq = plus_square(sq, centred(v[i][j], sum, 1.0f / kSize), i);
        const float rstd = inv_std(warp_sum(sq), 1.0f / kSize);
#pragma unroll
        for (int i = 0; i < CH; ++i) {
            uint4 g, b;
            if constexpr (kOne) {
                g = gv[i];
                b = bv[i];
            } else {
                g = __ldg(reinterpret_cast<const uint4*>(gamma) + lane + 32 * i);
                b = __ldg(reinterpret_cast<const uint4*>(beta) + lane + 32 * i);
            }
            const half2* gh = reinterpret_cast<const half2*>(&g);
            const half2* bh = reinterpret_cast<const half2*>(&b);
            uint4 o;
            half2* oh = reinterpret_cast<half2*>(&o);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float2 gg = __half22float2(gh[j]), bb = __half22float2(bh[j]);
                oh[j] = __floats2half2_rn(scaled(centred(v[i][2 * j], sum, 1.0f / kSize), rstd, gg.x, bb.x),
                                          scaled(centred(v[i][2 * j + 1], sum, 1.0f / kSize), rstd, gg.y, bb.y));
            }
            out[32 * i] = o;
        }
        if constexpr (kOne) break;
    }
}

// Any size and alignment, by single elements: one warp per row, three passes over the row (17771 x 769: 33.7 us).
__global__ void __launch_bounds__(256) skip_layernorm_generic(half* __restrict__ in_out,
                                                              const half* __restrict__ skip,
                                                              const half* __restrict__ gamma,
                                                              const half* __restrict__ beta,
                                                              int num, int size) {
    pdl_launch_dependents();
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarp = (gridDim.x * blockDim.x) >> 5;
    const float inv_n = 1.0f / (float)size;
    for (int row = warp; row < num; row += nwarp) {
        half* x = in_out + (size_t)row * size;
        const half* s = skip + (size_t)row * size;
        float sum = 0.f;
        for (int i = lane; i < size; i += 32) sum += __half2float(x[i]) + (skip ? __half2float(s[i]) : 0.f);
        const float mean = warp_sum(sum) * inv_n;
        float sq = 0.f;
        for (int i = lane; i < size; i += 32) {
            const float d = __half2float(x[i]) + (skip ? __half2float(s[i]) : 0.f) - mean;
            sq += d * d;
        }
        const float rstd = rsqrtf(warp_sum(sq) * inv_n + 1e-6f);
        for (int i = lane; i < size; i += 32) {
            const float v = __half2float(x[i]) + (skip ? __half2float(s[i]) : 0.f);
            x[i] = __float2half_rn((v - mean) * rstd * __half2float(gamma[i]) +
                                   __half2float(beta[i]));
        }
    }
}

// The same for even sizes on 4-byte boundaries, two elements per access. What bounds it is the number of accesses: 17771 x 770 32.6 us by
// single elements, 18.0 here; 131072 x 770 321 -> 160; 4096 x 2050 53 -> 24; 2048 x 770 12.7 -> 7.9.
__global__ void __launch_bounds__(256) skip_layernorm_pairs(half* __restrict__ in_out, const half* __restrict__ skip, const half* __restrict__ gamma,
                                                            const half* __restrict__ beta, int num, int size) {
    pdl_launch_dependents();
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarp = (gridDim.x * blockDim.x) >> 5;
    const float inv_n = 1.0f / (float)size;
    const half2* const g2 = reinterpret_cast<const half2*>(gamma);
    const half2* const b2 = reinterpret_cast<const half2*>(beta);
    for (int row = warp; row < num; row += nwarp) {
        half2* x = reinterpret_cast<half2*>(in_out + (size_t)row * size);
        const half2* s = reinterpret_cast<const half2*>(skip + (size_t)row * size);
        auto value = [&](int i) {
            float2 v = __half22float2(x[i]);
            if (skip) {
                const float2 t = __half22float2(s[i]);
                v.x += t.x;
                v.y += t.y;
            }
            return v;
        };
        float sum = 0.f;
#pragma unroll 4
        for (int i = lane; i < size / 2; i += 32) {
            const float2 v = value(i);
            sum += v.x + v.y;
        }
        const float mean = warp_sum(sum) * inv_n;
        float sq = 0.f;
#pragma unroll 4
        for (int i = lane; i < size / 2; i += 32) {
            const float2 v = value(i);
            sq += (v.x - mean) * (v.x - mean) + (v.y - mean) * (v.y - mean);
        }
        const float rstd = rsqrtf(warp_sum(sq) * inv_n + 1e-6f);
#pragma unroll 4
        for (int i = lane; i < size / 2; i += 32) {
            const float2 v = value(i), g = __half22float2(g2[i]), b = __half22float2(b2[i]);
            x[i] = __floats2half2_rn((v.x - mean) * rstd * g.x + b.x, (v.y - mean) * rstd * g.y + b.y);
        }
    }
}

}  // namespace et

namespace et {
// in_out <- LN(in_out + skip) * gamma + beta; skip == nullptr leaves the residual out (the layer stack's last
// LayerNorm when the others are folded into the linears).
int layernorm_launch(half* x, const half* s, const half* g, const half* b, int num, int size, cudaStream_t st);
}

extern "C" int et_skip_layernorm(void* in_out, const void* skip, const void* gamma,
                                 const void* beta, int num, int size, void* stream) {
    ET_REQUIRE(in_out && skip && gamma && beta, "et_skip_layernorm: null pointer");
    ET_REQUIRE(num >= 0 && size > 0, "et_skip_layernorm: bad dimensions");
    return et::layernorm_launch(static_cast<half*>(in_out), static_cast<const half*>(skip), static_cast<const half*>(gamma),
                                static_cast<const half*>(beta), num, size, static_cast<cudaStream_t>(stream));
}

int et::layernorm_launch(half* x, const half* s, const half* g, const half* b, int num, int size, cudaStream_t st) {
    using namespace et;
    if (num == 0) return ET_OK;
    const int warps_needed = num;
    int blocks = (warps_needed + 7) / 8;
    const bool vec = size % 8 == 0 && size <= 2048 && aligned16(x) && (!s || aligned16(s)) &&
                     aligned16(g) && aligned16(b);
    const bool pairs = size % 2 == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(s) | reinterpret_cast<uintptr_t>(g) |
                                          reinterpret_cast<uintptr_t>(b)) & 3) == 0;
    // (skip_layernorm_rows aside:) blocks per SM, by what is resident there. Of skip_layernorm_vec for 257 to 1024 elements three blocks
    // of eight warps are (registers): a multiple of three, two waves, or eight where a warp would have more than six rows, as shorter
    // shares even out the SMs' shares of the bandwidth (60000 x 1000: 64.2 us with 24, 68.8 with six). Narrower rows leave room for eight
    // blocks: 131072 x 200 31.6 us with them, 33.1 with 24. Wider rows: 24 cost 60000 x 2000 158 us instead of 149 with eight. Pairs: six
    // are resident, and four waves of them do better than one and a third (17771 x 770 18.0 us, 19.6 with eight; 131072 x 770 160 and
    // 196). Single elements: eight are resident (17771 x 770 32.6 us, 45.7 with six, 35.6 with 24; 131072 x 770 361 with eight, 321 with 24).
    const bool long_share = num / 12 > sm_count() * 3 * 8;
    const int per_sm = !vec ? (pairs || long_share ? 24 : 8) : size <= 256 ? 8 : size <= 1024 ? (long_share ? 24 : 6) : (long_share ? 8 : 6);
    blocks = std::min(blocks, sm_count() * per_sm);
    if (vec && size % 256 == 0) {   // every lane's chunks are whole
        using RowsFn = void (*)(half*, const half*, const half*, const half*, int);
        static const RowsFn rows[8][2] = {{skip_layernorm_rows<1, false, false>, skip_layernorm_rows<1, true, false>}, {skip_layernorm_rows<2, false, false>, skip_layernorm_rows<2, true, false>},
                                          {skip_layernorm_rows<3, false, false>, skip_layernorm_rows<3, true, false>}, {skip_layernorm_rows<4, false, false>, skip_layernorm_rows<4, true, false>},
                                          {skip_layernorm_rows<5, false, false>, skip_layernorm_rows<5, true, false>}, {skip_layernorm_rows<6, false, false>, skip_layernorm_rows<6, true, false>},
                                          {skip_layernorm_rows<7, false, false>, skip_layernorm_rows<7, true, false>}, {skip_layernorm_rows<8, false, false>, skip_layernorm_rows<8, true, false>}};
        static const RowsFn one[8][2] = {{skip_layernorm_rows<1, false, true>, skip_layernorm_rows<1, true, true>}, {skip_layernorm_rows<2, false, true>, skip_layernorm_rows<2, true, true>},
                                         {skip_layernorm_rows<3, false, true>, skip_layernorm_rows<3, true, true>}, {skip_layernorm_rows<4, false, true>, skip_layernorm_rows<4, true, true>},
                                         {skip_layernorm_rows<5, false, true>, skip_layernorm_rows<5, true, true>}, {skip_layernorm_rows<6, false, true>, skip_layernorm_rows<6, true, true>},
                                         {skip_layernorm_rows<7, false, true>, skip_layernorm_rows<7, true, true>}, {skip_layernorm_rows<8, false, true>, skip_layernorm_rows<8, true, true>}};
        const int ch = size / 256;
        // One row a warp in blocks of two warps where all have a place at once and an SM gets up to seven rows of 768; of rows of up to 768 elements
        // up to 14, in blocks of one (128 x 768 2.22 -> 1.70 us, 1024 x 768 2.73 -> 2.22, 2048 x 768 2.92 -> 2.56, 300 x 1024 2.30 -> 1.81, 256 x 2048
        // 2.90 -> 2.30; but 1024 x 1024 2.69 and 2.67, 1500 x 1024 2.84 and 2.97).
        const long sms = sm_count(), elements = (long)num * size;
        const int one_warps = elements <= 5400 * sms ? 2 : size <= 768 && num <= 14 * sms ? 1 : 0;
        if (one_warps) {
            launch_pdl(one[ch - 1][s != nullptr], dim3((num + one_warps - 1) / one_warps), dim3(32 * one_warps), 0, st, x, s, g, b, num);
        } else {
            const dim3 grid(std::min((warps_needed + 7) / 8, sm_count() * row_blocks(ch)));
            launch_pdl(rows[ch - 1][s != nullptr], grid, dim3(256), 0, st, x, s, g, b, num);
        }
    } else if (vec) {
        const int ch = (size / 8 + 31) / 32;
        switch (ch) {
            case 1: launch_pdl(skip_layernorm_vec<1>, dim3(blocks), dim3(256), 0, st, x, s, g, b, num, size); break;
            case 2: launch_pdl(skip_layernorm_vec<2>, dim3(blocks), dim3(256), 0, st, x, s, g, b, num, size); break;
            case 3: launch_pdl(skip_layernorm_vec<3>, dim3(blocks), dim3(256), 0, st, x, s, g, b, num, size); break;
            case 4: launch_pdl(skip_layernorm_vec<4>, dim3(blocks), dim3(256), 0, st, x, s, g, b, num, size); break;
            case 5:
            case 6: launch_pdl(skip_layernorm_vec<6>, dim3(blocks), dim3(256), 0, st, x, s, g, b, num, size); break;
            default: launch_pdl(skip_layernorm_vec<8>, dim3(blocks), dim3(256), 0, st, x, s, g, b, num, size); break;
        }
    } else if (pairs) {
        launch_pdl(skip_layernorm_pairs, dim3(blocks), dim3(256), 0, st, x, s, g, b, num, size);
    } else {
        launch_pdl(skip_layernorm_generic, dim3(blocks), dim3(256), 0, st, x, s, g, b, num, size);
    }
    return cuda_status(cudaGetLastError(), "et_skip_layernorm launch");
}
