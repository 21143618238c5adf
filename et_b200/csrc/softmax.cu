// Fused additive mask + row softmax over attention score matrices, in place.
// Replaces the mask/softmax half of kernels/attention.cu:273-323 (scores read from HBM) and
// the device function kernels/attention.cu:10-48 of the reference.
//
// Bandwidth kernel: 4*L*L bytes per score matrix (fp16 read + write); the [L x L] mask is
// shared by every matrix and stays in L2. The row is held in registers, fp32 max / sum, true row max (a fully masked
// row yields zeros), ex2 with log2(e) folded into the argument. Keys at index >= valid_len are excluded and written as zero.
#include <algorithm>
#include <type_traits>
#include "common.h"
#include "vec_math.cuh"

namespace et {

constexpr float kLog2e = 1.4426950408889634f;

// A row is a head of up to 7 elements, whole 16-byte granules of memory, and a tail of up to 7 elements, whatever its
// length and alignment (sequence lengths are rarely multiples of 8). G lanes share a row: lane l holds granules l, l + G, ...
// (CH of them) and, for l < 8, head element l and tail element l. Nothing but valid elements is ever read, so the granules
// need no per-element checks; what lies beyond valid_len is only written. The mask row has an alignment of its own: a
// granule's eight mask values come as the two granules that hold them, shifted into place (five 4-byte loads instead: 40 us against 30, L1 wavefronts).
// Short rows leave lanes idle, hence G = 8 and 16; R rows per group are in flight at once (softmax_many_kernel, below, takes over where a
// group has many). Bound by HBM for rows above ~256
// elements, by instruction issue below (~60 per granule: two fp32 operations per instruction, 32-bit index arithmetic).
// Measured with a mask: 1024 matrices of 512 x 512 229 -> 173 us (6.2 TB/s; 64-bit modulo and scalar fp32 before), 128 of
// 500 x 500 101 us (three passes, 2-byte accesses) -> 32 us.
template <int G>
__device__ __forceinline__ float group_max(float v) {
    if constexpr (G == 32) {
        return warp_max(v);
    } else {
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
        return v;
    }
}
template <int G>
__device__ __forceinline__ float group_sum(float v) {
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ uint4 pack_row(const float2 (&v)[4], float inv) {
    const float2 i2 = make_float2(inv, inv);
    uint4 o;
    half2* oh = reinterpret_cast<half2*>(&o);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float2 p = mul2(v[j], i2);
        oh[j] = __floats2half2_rn(p.x, p.y);
    }
    return o;
}

// Rows in whole granules on both sides (length a multiple of 8, aligned tensors).
template <int G, int CH, int R>
__global__ void __launch_bounds__(256) softmax_mask_vec(half* __restrict__ scores, const half* __restrict__ mask, unsigned nrow,
                                                        int L, int valid) {
    pdl_launch_dependents();
    pdl_wait();
    const int lane = threadIdx.x & (G - 1);
    const unsigned group = (blockIdx.x * blockDim.x + threadIdx.x) / G;
    const unsigned ngroup = (gridDim.x * blockDim.x) / G;
    const int nchunk = L >> 3;
    const unsigned rounds = (nrow + ngroup * R - 1) / (ngroup * R);   // the same for all groups of a warp
    for (unsigned it = 0; it < rounds; ++it) {
        const unsigned row0 = (it * ngroup + group) * R;
        uint4 sv[R][CH], mv[R][CH];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const unsigned row = row0 + r;
            const uint4* sr = reinterpret_cast<const uint4*>(scores + (size_t)row * L);
            const uint4* mr = mask ? reinterpret_cast<const uint4*>(mask + (size_t)(row % (unsigned)L) * L) : nullptr;
#pragma unroll
            for (int i = 0; i < CH; ++i) {
                const int c = lane + G * i;
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
            const unsigned row = row0 + r;
            float2 v[CH][4];
            float mx = -INFINITY;
#pragma unroll
            for (int i = 0; i < CH; ++i) {
                const half2* sh = reinterpret_cast<const half2*>(&sv[r][i]);
                const half2* mh = reinterpret_cast<const half2*>(&mv[r][i]);
                const int left = valid - (lane + G * i) * 8;   // valid elements from this granule's first one on (valid <= L)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    v[i][j] = add2(__half22float2(sh[j]), __half22float2(mh[j]));
                    if (2 * j >= left) v[i][j].x = -INFINITY;
                    if (2 * j + 1 >= left) v[i][j].y = -INFINITY;
                    mx = max3(mx, v[i][j].x, v[i][j].y);
                }
            }
            mx = group_max<G>(mx);
            const float shift = (mx == -INFINITY) ? 0.f : -mx * kLog2e;
            const float2 l2 = make_float2(kLog2e, kLog2e), s2 = make_float2(shift, shift);
            float2 sum2 = make_float2(0.f, 0.f);
#pragma unroll
            for (int i = 0; i < CH; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 x = fma2(v[i][j], l2, s2);
                    v[i][j] = make_float2(ex2_fast(x.x), ex2_fast(x.y));
                    sum2 = add2(sum2, v[i][j]);
                }
            const float sum = group_sum<G>(sum2.x + sum2.y);
            const float inv = sum > 0.f ? 1.0f / sum : 0.f;
            if (row < nrow) {
                uint4* sw = reinterpret_cast<uint4*>(scores + (size_t)row * L);
#pragma unroll
                for (int i = 0; i < CH; ++i) {
                    const int c = lane + G * i;
                    if (c < nchunk) __stcs(sw + c, pack_row(v[i], inv));
                }
            }
        }
    }
}

// Two scores plus two mask values, in fp32.
__device__ __forceinline__ float2 scores_plus(uint32_t two, uint32_t mask) {
    float2 v = __half22float2(*reinterpret_cast<const half2*>(&two));
    asm("{\n.reg .b16 l, h;\nmov.b32 {l, h}, %2;\nadd.rn.f32.f16 %0, l, %0;\nadd.rn.f32.f16 %1, h, %1;\n}" : "+f"(v.x), "+f"(v.y) : "r"(mask));
    return v;
}

struct RowShape { int head, granules, tail; };
__device__ __forceinline__ RowShape row_shape(const half* row, int valid) {
    RowShape s;
    s.head = min((int)((16 - (reinterpret_cast<uintptr_t>(row) & 15)) & 15) >> 1, valid);
    s.granules = (valid - s.head) >> 3;
    s.tail = (valid - s.head) & 7;
    return s;
}

// The elements of a granule that lie inside [lo, hi); zeros for the others.
__device__ __forceinline__ uint4 edge_granule(const half* p, const half* lo, const half* hi) {
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint32_t l = p + 2 * j >= lo && p + 2 * j < hi ? __half_as_ushort(p[2 * j]) : 0u;
        const uint32_t h = p + 2 * j + 1 >= lo && p + 2 * j + 1 < hi ? __half_as_ushort(p[2 * j + 1]) : 0u;
        w[j] = l | (h << 16);
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}

template <int G, int CH, int R, bool kMask>
__global__ void __launch_bounds__(256) softmax_mask_kernel(half* __restrict__ scores, const half* __restrict__ mask,
                                                           unsigned nrow, int L, int valid) {
    pdl_launch_dependents();
    pdl_wait();
    const int lane = threadIdx.x & (G - 1);
    const unsigned group = (blockIdx.x * blockDim.x + threadIdx.x) / G;
    const unsigned ngroup = (gridDim.x * blockDim.x) / G;
    const half kNone = __ushort_as_half((unsigned short)0xfc00u);   // -inf
    // all groups of a warp make the same number of rounds (the reductions use the whole warp)
    const unsigned rounds = (nrow + ngroup * R - 1) / (ngroup * R);
    for (unsigned it = 0; it < rounds; ++it) {
        const unsigned row0 = (it * ngroup + group) * R;
        uint4 sv[R][CH], ma[R][CH], mb[R][CH];
        half se[R][2], me[R][2];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const unsigned row = row0 + r;
            const half* sr = scores + (size_t)row * L;
            const RowShape q = row_shape(sr, row < nrow ? valid : 0);
            const half* const mg = mask + (size_t)(row % (unsigned)L) * L + q.head;
            const half* const ml = reinterpret_cast<const half*>(reinterpret_cast<uintptr_t>(mg) & ~(uintptr_t)15);
            const bool split = ml != mg;   // the second granule exists: it holds the values from the first boundary on
#pragma unroll
            for (int i = 0; i < CH; ++i) {
                const int c = lane + G * i;
                sv[r][i] = make_uint4(0xfc00fc00u, 0xfc00fc00u, 0xfc00fc00u, 0xfc00fc00u);
                ma[r][i] = mb[r][i] = make_uint4(0u, 0u, 0u, 0u);
                if (c < q.granules) {
                    sv[r][i] = __ldcs(reinterpret_cast<const uint4*>(sr + q.head) + c);
                    if constexpr (kMask) {
                        // whole granules: the first one may begin in front of the row, with the previous row's end (for the
                        // mask's first row: within the same 16 bytes as its first element), the second one end behind it
                        if (c > 0 || row % (unsigned)L > 0 || !split) ma[r][i] = __ldg(reinterpret_cast<const uint4*>(ml) + c);
                        else ma[r][i] = edge_granule(ml, mask, mask + (size_t)L * L);
                        if (split) {
                            const half* t = ml + 8 * c + 8;
                            if (t + 8 <= mask + (size_t)L * L) mb[r][i] = __ldg(reinterpret_cast<const uint4*>(t));
                            else mb[r][i] = edge_granule(t, mask, mask + (size_t)L * L);
                        }
                    }
                }
            }
            se[r][0] = lane < q.head ? sr[lane] : kNone;
            se[r][1] = lane < q.tail ? sr[q.head + 8 * q.granules + lane] : kNone;
            me[r][0] = me[r][1] = __float2half(0.f);
            if constexpr (kMask) {
                if (lane < q.head) me[r][0] = __ldg(mg - q.head + lane);
                if (lane < q.tail) me[r][1] = __ldg(mg + 8 * q.granules + lane);
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const unsigned row = row0 + r;
            half* const sr = scores + (size_t)row * L;
            const RowShape q = row_shape(sr, row < nrow ? valid : 0);
            const int sh = !kMask ? 0
                                         : (int)((reinterpret_cast<uintptr_t>(mask + (size_t)(row % (unsigned)L) * L + q.head) & 15) >> 1);
            float2 v[CH][4];
            float2 e = make_float2(__half2float(se[r][0]) + __half2float(me[r][0]), __half2float(se[r][1]) + __half2float(me[r][1]));
#pragma unroll
            for (int i = 0; i < CH; ++i) {
                uint32_t w[8] = {ma[r][i].x, ma[r][i].y, ma[r][i].z, ma[r][i].w, mb[r][i].x, mb[r][i].y, mb[r][i].z, mb[r][i].w};
                if constexpr (kMask) {   // the same shift for the whole row
                    if (sh & 4) {
#pragma unroll
                        for (int k = 0; k < 6; ++k) w[k] = w[k + 2];
                    }
                    if (sh & 2) {
#pragma unroll
                        for (int k = 0; k < 5; ++k) w[k] = w[k + 1];
                    }
#pragma unroll
                    for (int k = 0; k < 4; ++k) w[k] = __funnelshift_r(w[k], w[k + 1], (sh & 1) * 16);
                }
                const half2* xh = reinterpret_cast<const half2*>(&sv[r][i]);
                const half2* mh = reinterpret_cast<const half2*>(w);
#pragma unroll
                for (int j = 0; j < 4; ++j) v[i][j] = kMask ? add2(__half22float2(xh[j]), __half22float2(mh[j])) : __half22float2(xh[j]);
            }
            float mx = fmaxf(e.x, e.y);
#pragma unroll
            for (int i = 0; i < CH; ++i)
                mx = max3(mx, max3(v[i][0].x, v[i][0].y, fmaxf(v[i][1].x, v[i][1].y)), max3(v[i][2].x, v[i][2].y, fmaxf(v[i][3].x, v[i][3].y)));
            mx = group_max<G>(mx);
            const float shift = (mx == -INFINITY) ? 0.f : -mx * kLog2e;
            const float2 l2 = make_float2(kLog2e, kLog2e), s2 = make_float2(shift, shift);
            e = fma2(e, l2, s2);
            e = make_float2(ex2_fast(e.x), ex2_fast(e.y));
            float2 sum2 = e;
#pragma unroll
            for (int i = 0; i < CH; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 x = fma2(v[i][j], l2, s2);
                    v[i][j] = make_float2(ex2_fast(x.x), ex2_fast(x.y));
                    sum2 = add2(sum2, v[i][j]);
                }
            const float sum = group_sum<G>(sum2.x + sum2.y);
            const float inv = sum > 0.f ? 1.0f / sum : 0.f;
#pragma unroll
            for (int i = 0; i < CH; ++i) {
                const int c = lane + G * i;
                if (c < q.granules) __stcs(reinterpret_cast<uint4*>(sr + q.head) + c, pack_row(v[i], inv));
            }
            if (lane < q.head) sr[lane] = __float2half_rn(e.x * inv);
            if (lane < q.tail) sr[q.head + 8 * q.granules + lane] = __float2half_rn(e.y * inv);
            if (valid < L && row < nrow)
                for (int k = valid + lane; k < L; k += G) sr[k] = __float2half(0.f);
        }
    }
}

// The order in which the rows of any alignment are taken: a row index of the matrices c, c + 8, c + 16, ... (whose rows have the same
// alignment whatever the length, so the mask row stays in registers), the next row index, the next c.
struct RowWalk {
    half* at;
    int r, n, c;
    __device__ __forceinline__ RowWalk(half* scores, unsigned index, int nmat, int L) {
        const unsigned full = (unsigned)nmat / 8, more = (unsigned)nmat % 8;   // classes below `more` have full + 1 matrices
        const unsigned split = more * (full + 1) * (unsigned)L;
        unsigned in, deep;
        if (index < split) {
            deep = full + 1;
            c = (int)(index / (deep * (unsigned)L));
            in = index - (unsigned)c * deep * (unsigned)L;
        } else {
            deep = max(full, 1u);
            const unsigned past = index - split;
            c = (int)(more + past / (deep * (unsigned)L));
            in = past % (deep * (unsigned)L);
        }
        r = (int)(in / deep);
        n = c + 8 * (int)(in % deep);
        at = scores + (size_t)n * L * L + (size_t)r * L;
    }
    __device__ __forceinline__ void next(half* scores, int nmat, int L) {
        n += 8;
        at += (size_t)8 * L * L;
        if (n < nmat) return;
        if (++r == L) { r = 0; ++c; }
        n = c;
        at = scores + (size_t)n * L * L + (size_t)r * L;
    }
};

// Many rows of any length and alignment: a group takes `rows / groups` of them in the order above, D of them in flight. A mask row is
// fetched, shifted and put in place once for all matrices of its class, and added by mixed-precision additions. What bounds it is the
// memory system at that size (aligned rows of 504 elements take 25.6 us, 128 matrices) and D times the registers; the kernel above, with
// the next row requested when one is done, is the faster one where a group has few rows or a mask row few matrices.
// 128 x 500 x 500 with a mask 32.1 -> 29.3 us, without 33.3 -> 26.4; 1024 x 500 x 500 with one 246 -> 212; 512 x 77 x 77 10.3 -> 8.7.
// (As blocks of rows that a warp of its own copies in and out in bulk: 32.8 us and slower at every length.)
template <int G, int CH, int D, bool kMask, int kPerSm>
__global__ void __launch_bounds__(256, kPerSm) softmax_many_kernel(half* __restrict__ scores, const half* __restrict__ mask, int nmat, int L,
                                                                   int valid, unsigned rows) {
    pdl_launch_dependents();
    pdl_wait();
    const int lane = threadIdx.x & (G - 1);
    const unsigned group = (blockIdx.x * blockDim.x + threadIdx.x) / G;
    const unsigned ngroup = (gridDim.x * blockDim.x) / G;
    const unsigned first = (unsigned)((unsigned long long)group * rows / ngroup);
    const int count = (int)((unsigned long long)(group + 1) * rows / ngroup - first);
    const int rounds = (int)((rows + ngroup - 1) / ngroup);   // the same for all groups of a warp (the reductions use the whole warp)
    RowWalk cur(scores, min(first, rows - 1), nmat, L), ahead = cur;
    uint4 slot[D][CH];
    half slot_e[D][2];
    auto load = [&](int d, bool there) {
        const RowShape q = row_shape(ahead.at, there ? valid : 0);
#pragma unroll
        for (int i = 0; i < CH; ++i) {
            slot[d][i] = make_uint4(0xfc00fc00u, 0xfc00fc00u, 0xfc00fc00u, 0xfc00fc00u);   // -inf
            if (lane + G * i < q.granules) slot[d][i] = __ldcs(reinterpret_cast<const uint4*>(ahead.at + q.head) + lane + G * i);
        }
        slot_e[d][0] = slot_e[d][1] = __ushort_as_half((unsigned short)0xfc00u);
        if (lane < q.head) slot_e[d][0] = ahead.at[lane];
        if (lane < q.tail) slot_e[d][1] = ahead.at[q.head + 8 * q.granules + lane];
        if (there) ahead.next(scores, nmat, L);
    };
    uint32_t m[CH][4];
    float me[2] = {0.f, 0.f};
    auto load_mask = [&](const RowShape& q) {
        const half* const mg = mask + (size_t)cur.r * L + q.head;
        const half* const ml = reinterpret_cast<const half*>(reinterpret_cast<uintptr_t>(mg) & ~(uintptr_t)15);
        const bool split = ml != mg;   // the second granule exists: it holds the values from the first boundary on
        const int sh = (int)((reinterpret_cast<uintptr_t>(mg) & 15) >> 1);
#pragma unroll
        for (int i = 0; i < CH; ++i) {
            const int c = lane + G * i;
            uint4 ma = make_uint4(0u, 0u, 0u, 0u), mb = ma;
            if (c < q.granules) {
                // whole granules: the first one may begin in front of the row, with the previous row's end (for the
                // mask's first row: within the same 16 bytes as its first element), the second one end behind it
                if (c > 0 || cur.r > 0 || !split) ma = __ldg(reinterpret_cast<const uint4*>(ml) + c);
                else ma = edge_granule(ml, mask, mask + (size_t)L * L);
                if (split) {
                    const half* t = ml + 8 * c + 8;
                    if (t + 8 <= mask + (size_t)L * L) mb = __ldg(reinterpret_cast<const uint4*>(t));
                    else mb = edge_granule(t, mask, mask + (size_t)L * L);
                }
            }
            uint32_t w[8] = {ma.x, ma.y, ma.z, ma.w, mb.x, mb.y, mb.z, mb.w};
            if (sh & 4) {
#pragma unroll
                for (int k = 0; k < 6; ++k) w[k] = w[k + 2];
            }
            if (sh & 2) {
#pragma unroll
                for (int k = 0; k < 5; ++k) w[k] = w[k + 1];
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                m[i][k] = __funnelshift_r(w[k], w[k + 1], (sh & 1) * 16);
            }
        }
        me[0] = lane < q.head ? __half2float(__ldg(mg - q.head + lane)) : 0.f;
        me[1] = lane < q.tail ? __half2float(__ldg(mg + 8 * q.granules + lane)) : 0.f;
    };
    // one row: slot d, then the slot is filled with the row D later
    auto row = [&](int d, bool there, bool more) {
        const RowShape q = row_shape(cur.at, there ? valid : 0);
        float2 v[CH][4];
        float2 e = make_float2(__half2float(slot_e[d][0]) + me[0], __half2float(slot_e[d][1]) + me[1]);
#pragma unroll
        for (int i = 0; i < CH; ++i) {
            const uint32_t w[4] = {slot[d][i].x, slot[d][i].y, slot[d][i].z, slot[d][i].w};
#pragma unroll
            for (int j = 0; j < 4; ++j) v[i][j] = kMask ? scores_plus(w[j], m[i][j]) : __half22float2(*reinterpret_cast<const half2*>(&w[j]));
        }
        load(d, more);
        float mx = fmaxf(e.x, e.y);
#pragma unroll
        for (int i = 0; i < CH; ++i)
            mx = max3(mx, max3(v[i][0].x, v[i][0].y, fmaxf(v[i][1].x, v[i][1].y)), max3(v[i][2].x, v[i][2].y, fmaxf(v[i][3].x, v[i][3].y)));
        mx = group_max<G>(mx);
        const float shift = (mx == -INFINITY) ? 0.f : -mx * kLog2e;
        const float2 l2 = make_float2(kLog2e, kLog2e), s2 = make_float2(shift, shift);
        e = fma2(e, l2, s2);
        e = make_float2(ex2_fast(e.x), ex2_fast(e.y));
        float2 sum2 = e;
#pragma unroll
        for (int i = 0; i < CH; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float2 x = fma2(v[i][j], l2, s2);
                v[i][j] = make_float2(ex2_fast(x.x), ex2_fast(x.y));
                sum2 = add2(sum2, v[i][j]);
            }
        const float sum = group_sum<G>(sum2.x + sum2.y);
        const float inv = sum > 0.f ? 1.0f / sum : 0.f;
#pragma unroll
        for (int i = 0; i < CH; ++i)
            if (lane + G * i < q.granules) __stcs(reinterpret_cast<uint4*>(cur.at + q.head) + lane + G * i, pack_row(v[i], inv));
        if (lane < q.head) cur.at[lane] = __float2half_rn(e.x * inv);
        if (lane < q.tail) cur.at[q.head + 8 * q.granules + lane] = __float2half_rn(e.y * inv);
        if (valid < L && there)
            for (int z = valid + lane; z < L; z += G) cur.at[z] = __float2half(0.f);
        if (there) cur.next(scores, nmat, L);
    };
#pragma unroll
    for (int d = 0; d < D; ++d) load(d, d < count);
    int mask_r = -1, mask_c = -1;
    for (int k0 = 0; k0 < rounds; k0 += D) {
#pragma unroll
        for (int d = 0; d < D; ++d) {
            if (k0 + d >= rounds) break;
            const bool there = k0 + d < count;
            if (kMask && (cur.r != mask_r || cur.c != mask_c)) {
                mask_r = cur.r;
                mask_c = cur.c;
                load_mask(row_shape(cur.at, there ? valid : 0));
            }
            row(d, there, k0 + d + D < count);
        }
    }
}

// Rows above 2048 elements: one warp per row, three passes.
__global__ void __launch_bounds__(256) softmax_mask_generic(half* __restrict__ scores,
                                                            const half* __restrict__ mask,
                                                            unsigned nrow, int L, int valid) {
    pdl_launch_dependents();
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const unsigned warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const unsigned nwarp = (gridDim.x * blockDim.x) >> 5;
    for (unsigned row = warp; row < nrow; row += nwarp) {
        half* s = scores + (size_t)row * L;
        const half* m = mask ? mask + (size_t)(row % (unsigned)L) * L : nullptr;
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
    // The kernels count rows in 32 bits: launches of whole matrices with at most 2^30 rows.
    const int per_launch = std::max(1, (1 << 30) / seq_len);
    // Rows in whole granules on both sides take the kernel without heads and tails. CH * G * 8 elements fit (beside a head and
    // a tail in the other one). Two rows in flight where their registers leave enough warps: not with a shifted mask (44 us
    // with two, 31 with one, at 128 x 500 x 500).
    const bool vec = seq_len % 8 == 0 && aligned16(s) && (!m || aligned16(m));
    auto run = [&](auto kernel, int group, int rows) {
        for (int at = 0, n; at < nmat; at += n) {
            n = std::min(per_launch, nmat - at);
            const unsigned nrow = (unsigned)n * (unsigned)seq_len;
            const long groups = ((long)nrow + rows - 1) / rows;
            const long blocks = std::min((groups * group + 255) / 256, (long)sm_count() * 8);
            launch_pdl(kernel, dim3((unsigned)blocks), dim3(256), 0, st, s + (size_t)at * seq_len * seq_len, m, nrow, seq_len, valid_len);
        }
    };
    // Five rows to each group that three blocks an SM have (whatever the grid), and for a mask six matrices of a class (softmax_mask_kernel and this one, us:
    // 30 x 509 x 509, four rows, 10.4 and 10.7; 500 x 45 x 45, two rows, 3.1 and 4.0; 16 x 1001 x 1001, two matrices, 18.8 and 24.4. Without a mask around the line, in
    // L2 / from memory: 36 x 500 x 500 7.0 / 10.6 and 8.3 / 10.2, 48 x 465 x 465 12.0 / 14.6 and 10.5 / 11.7, 64 x 300 x 300 11.4 / 12.7 and 9.5 / 9.5.)
    auto run_many = [&](auto kernel, int group, int per_sm) {
        if ((long)nmat * seq_len < 5L * sm_count() * 3 * (256 / group) || (m && nmat < 48)) return false;
        const int most = std::max(8, per_launch / 8 * 8);   // a launch begins with a matrix of the first one's alignment
        for (int at = 0, n; at < nmat; at += n) {
            n = std::min(most, nmat - at);
            const unsigned rows = (unsigned)n * (unsigned)seq_len;
            launch_pdl(kernel, dim3((unsigned)std::min(((long)rows * group + 255) / 256, (long)sm_count() * per_sm)), dim3(256), 0, st,
                       s + (size_t)at * seq_len * seq_len, m, n, seq_len, valid_len, rows);
        }
        return true;
    };
    auto pick = [&](auto masked) {
        constexpr bool kMask = decltype(masked)::value;
        constexpr int R = kMask ? 1 : 2;
        // Rows in flight per group against blocks per SM. A row of two granules a lane without a mask leaves registers for a fourth block when only one is in
        // flight, which is the faster way whether the rows were just written, lie in L2 or come from memory (us, three rows and three blocks -> one and four: 300 x 300 x 300
        // 31.5 -> 30.6, 370 39.3 -> 37.6, 500 60.8 -> 56.5; just written 512 x 465 x 465 83.1 -> 75.6; from memory 200 x 500 x 500 50.0 -> 41.6), but long rows want ten to a
        // group (64 x 478 x 478 from memory 14.4 -> 15.3, 48 x 500 x 500 12.4 -> 12.9; 128 x 478 x 478 26.5 -> 25.3). With a mask, and up to 256 elements, it is not: its rows pass again
        // and again 128 x 500 x 500 takes 29.3 -> 28.7 us, for the first time 39.0 -> 41.0, just written 24.2 -> 24.9; 512 x 233 x 233 just written 30.9 -> 32.8, without a mask 28.7 -> 29.1.
        const bool four = !kMask && (seq_len < 430 || (long)nmat * seq_len >= 10L * sm_count() * 4 * 8);
        if (seq_len <= 64 ? run_many(softmax_many_kernel<8, 1, 3, kMask, 3>, 8, 3)
            : seq_len <= 128 ? run_many(softmax_many_kernel<16, 1, 3, kMask, 3>, 16, 3)
            : seq_len <= 256 ? run_many(softmax_many_kernel<32, 1, 3, kMask, 3>, 32, 3)
            : seq_len <= 512 ? (four ? run_many(softmax_many_kernel<32, 2, 1, false, 4>, 32, 4) : run_many(softmax_many_kernel<32, 2, kMask ? 2 : 3, kMask, 3>, 32, 3)) : false)
            return;
        if (seq_len <= 64) run(softmax_mask_kernel<8, 1, R, kMask>, 8, R);
        else if (seq_len <= 128) run(softmax_mask_kernel<16, 1, R, kMask>, 16, R);
        else if (seq_len <= 256) run(softmax_mask_kernel<32, 1, R, kMask>, 32, R);
        else if (seq_len <= 512) run(softmax_mask_kernel<32, 2, R, kMask>, 32, R);
        else if (seq_len <= 1024) run(softmax_mask_kernel<32, 4, 1, kMask>, 32, 1);
        else run(softmax_mask_kernel<32, 8, 1, kMask>, 32, 1);
    };
    if (seq_len > 2048) {
        run(softmax_mask_generic, 32, 1);
    } else if (vec) {
        if (seq_len <= 64) run(softmax_mask_vec<8, 1, 2>, 8, 2);
        else if (seq_len <= 128) run(softmax_mask_vec<16, 1, 2>, 16, 2);
        else if (seq_len <= 256) run(softmax_mask_vec<32, 1, 2>, 32, 2);
        else if (seq_len <= 512) run(softmax_mask_vec<32, 2, 2>, 32, 2);
        else if (seq_len <= 1024) run(softmax_mask_vec<32, 4, 2>, 32, 2);
        else run(softmax_mask_vec<32, 8, 1>, 32, 1);
    } else if (m) {
        pick(std::true_type{});
    } else {
        pick(std::false_type{});
    }
    return cuda_status(cudaGetLastError(), "et_softmax_mask launch");
}
