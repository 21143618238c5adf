// Fused additive mask + row softmax over attention score matrices, in place.
// Replaces the mask/softmax half of kernels/attention.cu:273-323 (scores read from HBM) and
// the device function kernels/attention.cu:10-48 of the reference.
//
// Bandwidth kernel: 4*L*L bytes per score matrix (fp16 read + write); the [L x L] mask is
// shared by every matrix and stays in L2. One warp per row, 16-byte accesses, the row held in
// registers, fp32 max / sum, true row max (a fully masked row yields zeros), ex2 with log2(e)
// folded into the argument. Keys at index >= valid_len are excluded and written as zero.
#include "common.h"

namespace et {

// 2^x on the special-function unit; inputs here are <= 0 or -inf, results flush to zero below 2^-126.
__device__ __forceinline__ float ex2_fast(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

template <int CH, int R>  // CH 16-byte chunks per lane (L <= CH*256); R rows per warp and iteration
__global__ void __launch_bounds__(256) softmax_mask_vec(half* __restrict__ scores,
                                                        const half* __restrict__ mask, long nrow,
                                                        int L, int valid) {
    pdl_launch_dependents();
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const long warp = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long nwarp = ((long)gridDim.x * blockDim.x) >> 5;
    const int nchunk = L >> 3;
    constexpr float kLog2e = 1.4426950408889634f;
    for (long row0 = warp * R; row0 < nrow; row0 += nwarp * R) {
        uint4 sv[R][CH], mv[R][CH];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const long row = row0 + r;
            const uint4* sr = reinterpret_cast<const uint4*>(scores + row * L);
            const uint4* mr = mask ? reinterpret_cast<const uint4*>(mask + (size_t)(row % L) * L) : nullptr;
#pragma unroll
            for (int i = 0; i < CH; ++i) {
                const int c = lane + 32 * i;
                sv[r][i] = make_uint4(0, 0, 0, 0);
                mv[r][i] = make_uint4(0, 0, 0, 0);
                if (row < nrow && c < nchunk) {
                    sv[r][i] = __ldcs(sr + c);
                    if (mr) mv[r][i] = __ldg(mr + c);
                }
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const long row = row0 + r;
            float v[CH][8];
            float mx = -INFINITY;
#pragma unroll
            for (int i = 0; i < CH; ++i) {
                const int c = lane + 32 * i;
                const half2* sh = reinterpret_cast<const half2*>(&sv[r][i]);
                const half2* mh = reinterpret_cast<const half2*>(&mv[r][i]);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 a = __half22float2(sh[j]), m = __half22float2(mh[j]);
                    const int k = c * 8 + 2 * j;
                    v[i][2 * j] = (c < nchunk && k < valid) ? a.x + m.x : -INFINITY;
                    v[i][2 * j + 1] = (c < nchunk && k + 1 < valid) ? a.y + m.y : -INFINITY;
                    mx = fmaxf(mx, fmaxf(v[i][2 * j], v[i][2 * j + 1]));
                }
            }
#pragma unroll
            for (int m = 16; m > 0; m >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, m));
            const float shift = (mx == -INFINITY) ? 0.f : mx * kLog2e;
            float sum = 0.f;
#pragma unroll
            for (int i = 0; i < CH; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    v[i][j] = ex2_fast(v[i][j] * kLog2e - shift);
                    sum += v[i][j];
                }
#pragma unroll
            for (int m = 16; m > 0; m >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, m);
            const float inv = sum > 0.f ? 1.0f / sum : 0.f;
            if (row < nrow) {
                uint4* sw = reinterpret_cast<uint4*>(scores + row * L);
#pragma unroll
                for (int i = 0; i < CH; ++i) {
                    const int c = lane + 32 * i;
                    if (c < nchunk) {
                        uint4 o;
                        half2* oh = reinterpret_cast<half2*>(&o);
#pragma unroll
                        for (int j = 0; j < 4; ++j)
                            oh[j] = __floats2half2_rn(v[i][2 * j] * inv, v[i][2 * j + 1] * inv);
                        __stcs(sw + c, o);
                    }
                }
            }
        }
    }
}

// Rows of any length and alignment (sequence lengths are rarely multiples of 8), at most CH * 256 - 14 elements: the row is
// covered by the 16-byte granules of memory that it touches, so that all of its traffic but the two edge granules moves in
// aligned 16-byte accesses. Edge granules are read whole where the tensor's bounds allow (the neighbouring row's elements
// are masked off) and written element by element. The mask row has an alignment of its own: the two granules that hold a
// lane's eight mask values are read (the second one is the next lane's first: an L1 hit) and shifted into place.
// HBM bound: 4 * L bytes per row. 128 matrices of 500 x 500 with a mask: 101 us by the three-pass kernel below, 25 us here.
__device__ __forceinline__ uint4 granule(const half* p, const half* lo, const half* hi) {
    if (p >= lo && p + 8 <= hi) return __ldg(reinterpret_cast<const uint4*>(p));
    __align__(16) half v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = (p + j >= lo && p + j < hi) ? p[j] : __float2half(0.f);
    return *reinterpret_cast<const uint4*>(v);
}
template <int CH, int R>
__global__ void __launch_bounds__(256) softmax_mask_shift(half* __restrict__ scores, const half* __restrict__ mask, long nrow,
                                                          int L, int valid) {
    pdl_launch_dependents();
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const long warp = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long nwarp = ((long)gridDim.x * blockDim.x) >> 5;
    constexpr float kLog2e = 1.4426950408889634f;
    const half* const send = scores + nrow * L;
    const half* const mend = mask ? mask + (size_t)L * L : nullptr;
    for (long row0 = warp * R; row0 < nrow; row0 += nwarp * R) {
        uint4 sv[R][CH];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const half* sr = scores + (row0 + r) * L;
            const int off = (int)((reinterpret_cast<uintptr_t>(sr) & 15) >> 1);   // elements of the first granule before the row
#pragma unroll
            for (int i = 0; i < CH; ++i) {
                const int k = (lane + 32 * i) * 8 - off;
                sv[r][i] = make_uint4(0, 0, 0, 0);
                if (row0 + r < nrow && k < L) {
                    const half* p = sr + k;
                    if (p >= scores && p + 8 <= send) sv[r][i] = __ldcs(reinterpret_cast<const uint4*>(p));
                    else sv[r][i] = granule(p, scores, send);
                }
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const long row = row0 + r;
            if (row >= nrow) break;
            half* sr = scores + row * L;
            const int off = (int)((reinterpret_cast<uintptr_t>(sr) & 15) >> 1);
            float v[CH][8];
            float mx = -INFINITY;
#pragma unroll
            for (int i = 0; i < CH; ++i) {
                const int k = (lane + 32 * i) * 8 - off;
                uint32_t m[4] = {0u, 0u, 0u, 0u};
                if (mask && k < L) {
                    const half* p = mask + (size_t)(row % L) * L + k;
                    const int sh = (int)((reinterpret_cast<uintptr_t>(p) & 15) >> 1);   // the same for the whole row
                    const uint4 a = granule(p - sh, mask, mend);
                    const uint4 b = sh ? granule(p - sh + 8, mask, mend) : make_uint4(0, 0, 0, 0);
                    uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
                    if (sh & 4)
#pragma unroll
                        for (int q = 0; q < 6; ++q) w[q] = w[q + 2];
                    if (sh & 2)
#pragma unroll
                        for (int q = 0; q < 5; ++q) w[q] = w[q + 1];
#pragma unroll
                    for (int q = 0; q < 4; ++q) m[q] = (sh & 1) ? __funnelshift_r(w[q], w[q + 1], 16) : w[q];
                }
                const half2* xh = reinterpret_cast<const half2*>(&sv[r][i]);
                const half2* mh = reinterpret_cast<const half2*>(m);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 a = __half22float2(xh[j]), b = __half22float2(mh[j]);
                    const int e = k + 2 * j;
                    v[i][2 * j] = (e >= 0 && e < valid) ? a.x + b.x : -INFINITY;
                    v[i][2 * j + 1] = (e + 1 >= 0 && e + 1 < valid) ? a.y + b.y : -INFINITY;
                    mx = fmaxf(mx, fmaxf(v[i][2 * j], v[i][2 * j + 1]));
                }
            }
#pragma unroll
            for (int m = 16; m > 0; m >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, m));
            const float shift = (mx == -INFINITY) ? 0.f : mx * kLog2e;
            float sum = 0.f;
#pragma unroll
            for (int i = 0; i < CH; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    v[i][j] = ex2_fast(v[i][j] * kLog2e - shift);
                    sum += v[i][j];
                }
#pragma unroll
            for (int m = 16; m > 0; m >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, m);
            const float inv = sum > 0.f ? 1.0f / sum : 0.f;
#pragma unroll
            for (int i = 0; i < CH; ++i) {
                const int k = (lane + 32 * i) * 8 - off;
                if (k >= L) continue;
                uint4 o;
                half2* oh = reinterpret_cast<half2*>(&o);
#pragma unroll
                for (int j = 0; j < 4; ++j) oh[j] = __floats2half2_rn(v[i][2 * j] * inv, v[i][2 * j + 1] * inv);
                if (k >= 0 && k + 8 <= L) {
                    __stcs(reinterpret_cast<uint4*>(sr + k), o);
                } else {
                    const half* ov = reinterpret_cast<const half*>(&o);
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        if (k + j >= 0 && k + j < L) sr[k + j] = ov[j];
                }
            }
        }
    }
}

// Rows above 2048 elements: one warp per row, three passes.
__global__ void __launch_bounds__(256) softmax_mask_generic(half* __restrict__ scores,
                                                            const half* __restrict__ mask,
                                                            long nrow, int L, int valid) {
    pdl_launch_dependents();
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const long warp = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long nwarp = ((long)gridDim.x * blockDim.x) >> 5;
    constexpr float kLog2e = 1.4426950408889634f;
    for (long row = warp; row < nrow; row += nwarp) {
        half* s = scores + row * L;
        const half* m = mask ? mask + (size_t)(row % L) * L : nullptr;
        float mx = -INFINITY;
        for (int k = lane; k < valid; k += 32)
            mx = fmaxf(mx, __half2float(s[k]) + (m ? __half2float(m[k]) : 0.f));
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        const float shift = (mx == -INFINITY) ? 0.f : mx * kLog2e;
        float sum = 0.f;
        for (int k = lane; k < valid; k += 32)
            sum += exp2f((__half2float(s[k]) + (m ? __half2float(m[k]) : 0.f)) * kLog2e - shift);
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        const float inv = sum > 0.f ? 1.0f / sum : 0.f;
        for (int k = lane; k < L; k += 32) {
            float p = 0.f;
            if (k < valid)
                p = exp2f((__half2float(s[k]) + (m ? __half2float(m[k]) : 0.f)) * kLog2e - shift) *
                    inv;
            s[k] = __float2half_rn(p);
        }
    }
}

}  // namespace et

extern "C" int et_softmax_mask(void* scores, const void* mask, int nmat, int seq_len,
                               int valid_len, void* stream) {
    using namespace et;
    ET_REQUIRE(scores, "et_softmax_mask: null scores");
    ET_REQUIRE(nmat >= 0 && seq_len > 0, "et_softmax_mask: bad dimensions");
    ET_REQUIRE(valid_len >= 0 && valid_len <= seq_len, "et_softmax_mask: valid_len out of range");
    if (nmat == 0) return ET_OK;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    half* s = static_cast<half*>(scores);
    const half* m = static_cast<const half*>(mask);
    const long nrow = (long)nmat * seq_len;
    long blocks = (nrow + 15) / 16;          // 8 warps per block, 2 rows per warp and iteration
    const long cap = (long)sm_count() * 8;
    if (blocks > cap) blocks = cap;
    // Rows whose elements all sit in whole 16-byte granules take the plain form; the others the shifted one, up to the length
    // that eight granules per lane hold wherever a row starts.
    const bool vec = seq_len % 8 == 0 && seq_len <= 2048 && aligned16(s) && (!m || aligned16(m));
    const int granules = (seq_len + 14) / 8;   // touched by a row at the worst alignment
    if (!vec && granules <= 256 && (reinterpret_cast<uintptr_t>(s) & 1) == 0) {
        if (granules <= 32) launch_pdl(softmax_mask_shift<1, 4>, dim3((unsigned)blocks), dim3(256), 0, st, s, m, nrow, seq_len, valid_len);
        else if (granules <= 64) launch_pdl(softmax_mask_shift<2, 2>, dim3((unsigned)blocks), dim3(256), 0, st, s, m, nrow, seq_len, valid_len);
        else if (granules <= 128) launch_pdl(softmax_mask_shift<4, 1>, dim3((unsigned)blocks), dim3(256), 0, st, s, m, nrow, seq_len, valid_len);
        else launch_pdl(softmax_mask_shift<8, 1>, dim3((unsigned)blocks), dim3(256), 0, st, s, m, nrow, seq_len, valid_len);
    } else if (vec) {
        const int ch = (seq_len / 8 + 31) / 32;
        switch (ch) {
            case 1: launch_pdl(softmax_mask_vec<1, 2>, dim3((unsigned)blocks), dim3(256), 0, st, s, m, nrow, seq_len, valid_len); break;
            case 2: launch_pdl(softmax_mask_vec<2, 2>, dim3((unsigned)blocks), dim3(256), 0, st, s, m, nrow, seq_len, valid_len); break;
            case 3:
            case 4: launch_pdl(softmax_mask_vec<4, 2>, dim3((unsigned)blocks), dim3(256), 0, st, s, m, nrow, seq_len, valid_len); break;
            default: launch_pdl(softmax_mask_vec<8, 1>, dim3((unsigned)blocks), dim3(256), 0, st, s, m, nrow, seq_len, valid_len); break;
        }
    } else {
        launch_pdl(softmax_mask_generic, dim3((unsigned)blocks), dim3(256), 0, st, s, m, nrow, seq_len, valid_len);
    }
    return cuda_status(cudaGetLastError(), "et_softmax_mask launch");
}
