// Tile-sparse linear  Y[T x N] = X[T x K] . W^T + bias  (optional tanh-GELU), W in 16x16 tile-BSR, for in_feat up to 1024: a
// slab of 128 tokens stays in tensor memory, whole, while the weight streams past it.
// Replaces, for those sizes, kernels/linear.cu:54-167 of the reference.
//
// Why: with A in tensor memory a kept tile is one UMMA 128x16x16 of ~9 clocks (four issuing warps), but bringing A there is
// dear: tcgen05.cp moves 64 bytes per clock and takes turns with the UMMAs on the tensor pipe (measured: 2048 UMMAs and 256
// copies of 4 KB take the sum of their times). The tile kernel (tile_gemm.cu) keeps 384 accumulator columns and streams A
// through the other 128 once per 384 output features: 512 clocks of copying per 128 x 128 chunk against ~350 of UMMAs at
// 80 % sparsity. Here A is copied once per slab and CTA: 768 inputs take 384 columns, and the other 128 hold two accumulators
// of 64 features, so that one is converted and stored while the next is multiplied. Inputs from 768 to 1024 stay in shared
// memory, as the A operand of UMMAs that read it there (~40 clocks a tile).
// What bounds it: for half-empty weights the UMMAs; at 75 % sparsity and above the stores, ~30 bytes per clock and SM
// (546 clocks per 128 x 64 tile), which is about what L2 takes from all SMs together.
//
// The weight is re-packed once into blocks of 64 features (x a part of the K range, so that two blocks per accumulator fit): per issuing warp
// a list of K slices, one byte per tile, then the tiles in UMMA layout. Roles: warp 0 copies activations, warps 2-3 weight
// blocks (a warp that has requested a copy goes on only after ~700 clocks), warp 1 moves activations to tensor memory, warps
// 4-11 issue and warps 12-27 convert and store. Copies of weights, issuing and converting come in two sets, one per accumulator: four issuing warps (one block-row of 16 features each), eight converting ones. The sets
// run apart: while one accumulator is handed over and drained, the other set issues. One elected lane issues a block's UMMAs in one go:
// ~120 clocks each (110 without the converting warps' stores); eight warps that do nothing else get one through in 55 to 60, which is
// the tensor pipe. As single predicated instructions they took ~145: 17771 x 768 -> 2304 at 75 % 32.8 us instead of 31.9, 8192 x 768 ->
// 2304 at 50 % 26.0 instead of 25.3; with those that read from shared memory outside the region 65536 x 1024 -> 3072 at 90 % 161.9
// instead of 157.4. A CTA takes (slab, range of features) items; the number of ranges is chosen at the launch so that the last wave is full.
// Every mbarrier wait is bounded; a role that gives up records a code and all threads meet at the common exit.
#include <algorithm>
#include <cstring>
#include <vector>
#include "common.h"
#include "epilogue.cuh"
#include "ptx.cuh"
#include "resident_gemm.h"
#include "tmap.h"

namespace et {

namespace {

constexpr int kSlab = 128;
constexpr int kKC = 128;                          // K elements per copied chunk: two 128-byte-swizzled panels
constexpr int kPanelBytes = kSlab * 64 * 2;       // 16 KB
constexpr int kChunkBytes = 2 * kPanelBytes;
constexpr int kTmemSlices = 48;                   // 16-wide K slices held in tensor memory (8 columns each)
constexpr int kMaxK = 1024;
constexpr int kMaxChunks = kMaxK / kKC;
constexpr int kTmemChunks = kTmemSlices * 16 / kKC;
constexpr int kGroupRows = 4;                     // block-rows per accumulator, one per issuing warp
constexpr int kAccCols = kGroupRows * 16;
constexpr uint32_t kAccAt = kTmemSlices * 8;
constexpr int kListBytes = 64;                    // entries per issuing warp and block
constexpr int kHeadBytes = 64 + kGroupRows * kListBytes;
constexpr int kMaxRing = 4;
constexpr int kSets = 2;                          // accumulators, each with its own issuing and converting warps and weight slots
constexpr int kFirstIssuer = 4, kIssuers = kSets * kGroupRows, kFirstEpi = kFirstIssuer + kIssuers, kEpiWarps = 16;
constexpr int kThreads = 32 * (kFirstEpi + kEpiWarps);
constexpr int kUnitBytes = 32 * 32 * 2;
constexpr int kSmemMax = 232448;

struct ResidentParams {
    const uint2* dir;         // [group][part]: {offset, size} in 16-byte units
    const uint8_t* stream;
    const half* bias;
    bool bias_given;          // the caller's, not the weight's own: the preceding kernel may still be writing it
    const uint8_t* empty;     // per group, a bit per block-row without tiles; null when there is none
    int T, N, K, groups, parts, ranges, items, slabs;
    int nx, nw, block_bytes;   // nw: weight slots per set
    int* err;
};

struct ResidentShared {
    uint64_t x_full[kMaxRing], x_empty[kMaxRing];   // chunk slots: landed / copied on to tensor memory
    uint64_t w_full[kSets][kMaxRing], w_empty[kSets][kMaxRing];   // weight blocks: landed / their UMMAs have completed (4 commits)
    uint64_t a_ready[kMaxChunks];                   // per chunk, once per item: in place for the UMMAs
    uint64_t a_free, tail_free;                     // the item's UMMAs have completed: its activations in tensor memory, in shared memory may be overwritten
    uint64_t acc_full[2], acc_empty[2];
    uint32_t tmem_base;
    volatile int abort;
};

// UMMAs of the lane that `leader` names, without a branch.
__device__ __forceinline__ void umma_ts_if(uint32_t leader, uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n.reg .pred p, q;\nsetp.ne.u32 p, %4, 0;\nsetp.ne.u32 q, %5, 0;\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}" ::"r"(d_tmem),
        "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(leader)
        : "memory");
}
__device__ __forceinline__ void umma_ss_if(uint32_t leader, uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n.reg .pred p, q;\nsetp.ne.u32 p, %4, 0;\nsetp.ne.u32 q, %5, 0;\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(leader)
        : "memory");
}
__device__ __forceinline__ void cp_128x256b(uint32_t taddr, uint64_t sdesc) {
    asm volatile("tcgen05.cp.cta_group::1.128x256b [%0], %1;" ::"r"(taddr), "l"(sdesc) : "memory");
}

// kEmpty: some block-row has no tiles.
template <bool kGelu, bool kEmpty>
__global__ void __launch_bounds__(kThreads, 1) resident_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmY,
                                                               const __grid_constant__ ResidentParams p) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int chunks = (p.K + kKC - 1) / kKC, tchunks = min(chunks, kTmemChunks);
    uint8_t* const tail = smem;                                                    // chunks beyond the tensor-memory part
    uint8_t* const xring = tail + (size_t)(chunks - tchunks) * kChunkBytes;
    uint8_t* const wring = xring + (size_t)p.nx * kChunkBytes;
    uint8_t* const epi = wring + (size_t)kSets * p.nw * p.block_bytes;             // a unit per converting warp
    ResidentShared* const sh = reinterpret_cast<ResidentShared*>(epi + kEpiWarps * kUnitBytes);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int G = gridDim.x;

    if (tid == 0) {
        for (int i = 0; i < kMaxRing; ++i) {
            mbar_init(&sh->x_full[i], 1); mbar_init(&sh->x_empty[i], 1);
            for (int k = 0; k < kSets; ++k) { mbar_init(&sh->w_full[k][i], 1); mbar_init(&sh->w_empty[k][i], kGroupRows); }
        }
        for (int i = 0; i < kMaxChunks; ++i) mbar_init(&sh->a_ready[i], 1);
        mbar_init(&sh->a_free, kIssuers);
        mbar_init(&sh->tail_free, kIssuers);
        for (int i = 0; i < 2; ++i) { mbar_init(&sh->acc_full[i], kGroupRows); mbar_init(&sh->acc_empty[i], kEpiWarps / 2); }
        sh->abort = 0;
        fence_mbar_init();
        prefetch_tmap(&tmX);
    }
    if (warp == 1) {
        tmem_alloc(&sh->tmem_base, 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh->tmem_base;
    auto give_up = [&](int code) {
        if (lane == 0) {
            if (!sh->abort) atomicExch(p.err, code);
            sh->abort = 1;
        }
    };
    // (A wait that gives up has lasted far longer than any copy: nothing is in flight when the CTA leaves.)

    if (warp == 0) {
        // ---- activations
        pdl_wait();
        bool ok = true;
        int xs = 0;
        uint32_t ph = 1, ptail = 1;
        for (int item = blockIdx.x; item < p.items && ok; item += G) {
            const int row = (item / p.ranges) * kSlab;
            for (int c = 0; c < tchunks; ++c) {
                ok = mbar_wait(&sh->x_empty[xs], ph);
                if (!ok) break;
                if (lane == 0) {
                    mbar_expect_tx(&sh->x_full[xs], kChunkBytes);
                    tma_load_3d(xring + (size_t)xs * kChunkBytes, &tmX, 0, row, 2 * c, &sh->x_full[xs]);
                }
                __syncwarp();
                if (++xs == p.nx) { xs = 0; ph ^= 1u; }
            }
            if (ok && tchunks < chunks) {
                ok = mbar_wait(&sh->tail_free, ptail);
                ptail ^= 1u;
                if (ok && lane == 0)
                    for (int c = tchunks; c < chunks; ++c) {
                        mbar_expect_tx(&sh->a_ready[c], kChunkBytes);
                        tma_load_3d(tail + (size_t)(c - tchunks) * kChunkBytes, &tmX, 0, row, 2 * c, &sh->a_ready[c]);
                    }
                __syncwarp();
            }
        }
        if (!ok) give_up(41);
    } else if (warp == 2 || warp == 3) {
        // ---- weight blocks of one set (they do not depend on the preceding kernel)
        const int set = warp - 2;
        bool ok = true;
        int ws = 0;
        uint32_t ph = 1, gs = 0;
        for (int item = blockIdx.x; item < p.items && ok; item += G) {
            const int r = item % p.ranges;
            const int g0 = r * p.groups / p.ranges, g1 = (r + 1) * p.groups / p.ranges;
            for (int g = g0; g < g1 && ok; ++g, ++gs) {
                if ((int)(gs & 1u) != set) continue;
                for (int b = g * p.parts; b < (g + 1) * p.parts; ++b) {
                    const uint2 d = __ldg(p.dir + b);
                    ok = mbar_wait(&sh->w_empty[set][ws], ph);
                    if (!ok) break;
                    if (lane == 0) {
                        mbar_expect_tx(&sh->w_full[set][ws], d.y * 16u);
                        bulk_load(wring + (size_t)(set * p.nw + ws) * p.block_bytes, p.stream + (size_t)d.x * 16u, d.y * 16u, &sh->w_full[set][ws]);
                    }
                    __syncwarp();
                    if (++ws == p.nw) { ws = 0; ph ^= 1u; }
                }
            }
        }
        if (!ok) give_up(42);
    } else if (warp == 1) {
        // ---- shared memory -> tensor memory. The columns are free when the previous item's UMMAs have completed: a copy is
        // guaranteed to run ahead of UMMAs issued after it, but not behind those issued before it.
        bool ok = true;
        int xs = 0, n = 0;
        uint32_t ph = 0;
        for (int item = blockIdx.x; item < p.items && ok; item += G, ++n) {
            if (n > 0) ok = mbar_wait(&sh->a_free, (uint32_t)(n - 1) & 1u);
            for (int c = 0; c < tchunks && ok; ++c) {
                ok = mbar_wait(&sh->x_full[xs], ph);
                if (!ok) break;
                tc_fence_after();
                if (elect_one()) {
                    const uint32_t xa = smem_u32(xring + (size_t)xs * kChunkBytes);
                    const int slices = min(8, p.K / 16 - 8 * c);
                    for (int s = 0; s < slices; ++s)
                        cp_128x256b(tmem + (uint32_t)(8 * c + s) * 8, make_smem_desc(xa + (s >> 2) * kPanelBytes + (s & 3) * 32, 16, 1024, 2));
                    umma_commit(&sh->a_ready[c]);
                    umma_commit(&sh->x_empty[xs]);
                }
                __syncwarp();
                if (++xs == p.nx) { xs = 0; ph ^= 1u; }
            }
        }
        if (!ok) give_up(43);
    } else if (warp >= kFirstIssuer && warp < kFirstEpi) {
        // ---- UMMAs: every second group, block-row w of it
        const int w = (warp - kFirstIssuer) & 3, set = (warp - kFirstIssuer) >> 2;
        const uint64_t b_desc0 = make_smem_desc(0, 128, 256, 0);   // no swizzle: 128 B between core matrices along K, 256 B along N
        const uint64_t t_desc0 = make_smem_desc(smem_u32(tail), 16, 1024, 2);
        constexpr uint32_t idesc = make_idesc_f16(128, 16);
        const uint32_t d = tmem + kAccAt + set * kAccCols + (uint32_t)w * 16;
        const uint32_t leader = elect_one() ? 1u : 0u;
        bool ok = true;
        int ws = 0, n = 0;
        uint32_t ph = 0, gs = 0;
        for (int item = blockIdx.x; item < p.items && ok; item += G, ++n) {
            const int r = item % p.ranges;
            const int g0 = r * p.groups / p.ranges, g1 = (r + 1) * p.groups / p.ranges;
            int ready = 0;   // chunks of the item known to be in place: the set's first group follows them one by one
            for (int g = g0; g < g1 && ok; ++g, ++gs) {
                if ((int)(gs & 1u) != set) continue;
                ok = mbar_wait(&sh->acc_empty[set], ((gs >> 1) & 1u) ^ 1u);
                if (!ok) break;
                uint32_t accumulate = 0;   // the block-row's first UMMA overwrites
                for (int part = 0; part < p.parts; ++part) {
                    ok = mbar_wait(&sh->w_full[set][ws], ph);
                    if (!ok) break;
                    tc_fence_after();
                    const uint8_t* blk = wring + (size_t)(set * p.nw + ws) * p.block_bytes;
                    // (a reduction over equal values: the compiler then knows it to be the same for the warp, and so the descriptors)
                    const uint32_t hdr = __reduce_max_sync(0xffffffffu, reinterpret_cast<const uint32_t*>(blk)[w]);
                    const int nts = (hdr >> 16) & 0xff, nall = hdr >> 24;
                    const uint8_t* list = blk + 64 + w * kListBytes;
                    const uint64_t bd = b_desc0 + ((smem_u32(blk) + kHeadBytes + (hdr & 0xffffu) * 512u) >> 4);
                    auto issue_one = [&](int i) {
                        const uint32_t k = list[i];
                        if (k < (uint32_t)kTmemSlices) {
                            umma_ts_if(leader, d, tmem + k * 8u, bd + (uint64_t)(i * 32), idesc, accumulate);
                        } else {
                            const uint32_t t = k - kTmemSlices;
                            umma_ss_if(leader, d, t_desc0 + (uint64_t)(((t >> 2) * kPanelBytes + (t & 3) * 32) >> 4), bd + (uint64_t)(i * 32), idesc, accumulate);
                        }
                        accumulate = 1;
                    };
                    if (ready == chunks) {
                        // by one lane in one go: the tiles whose activations are in tensor memory, then those that read them from shared memory
                        if (leader && nall > 0) {
                            auto ts = [&](int i, uint32_t k, uint32_t acc) { umma_f16_ts(d, tmem + k * 8u, bd + (uint64_t)(i * 32), idesc, acc); };
                            uint32_t acc = accumulate;
                            int i = 0;
#pragma unroll 1
                            for (; i + 4 <= nts; i += 4) {
                                const uint32_t k4 = *reinterpret_cast<const uint32_t*>(list + i);
                                ts(i, k4 & 0xffu, acc);
                                ts(i + 1, (k4 >> 8) & 0xffu, 1u);
                                ts(i + 2, (k4 >> 16) & 0xffu, 1u);
                                ts(i + 3, k4 >> 24, 1u);
                                acc = 1;
                            }
                            if (i < nts) {
                                const uint32_t k4 = *reinterpret_cast<const uint32_t*>(list + i);
                                ts(i, k4 & 0xffu, acc);
                                if (i + 1 < nts) ts(i + 1, (k4 >> 8) & 0xffu, 1u);
                                if (i + 2 < nts) ts(i + 2, (k4 >> 16) & 0xffu, 1u);
                                acc = 1;
                            }
#pragma unroll 1
                            for (i = nts; i < nall; ++i) {
                                const uint32_t t = list[i] - kTmemSlices;
                                umma_f16(d, t_desc0 + (uint64_t)(((t >> 2) * kPanelBytes + (t & 3) * 32) >> 4), bd + (uint64_t)(i * 32), idesc, acc);
                                acc = 1;
                            }
                        }
                        __syncwarp();
                        if (nall > 0) accumulate = 1;
                    } else {
                        int i = 0;
                        for (const int c1 = (part + 1) * chunks / p.parts; ready < c1; ++ready) {
                            ok = mbar_wait(&sh->a_ready[ready], (uint32_t)n & 1u);
                            if (!ok) break;
                            tc_fence_after();
                            for (; i < nall && list[i] < 8 * (ready + 1); ++i) issue_one(i);
                        }
                        if (!ok) break;
                    }
                    if (leader) {
                        umma_commit(&sh->w_empty[set][ws]);
                        if (part + 1 == p.parts) umma_commit(&sh->acc_full[set]);
                    }
                    __syncwarp();
                    if (++ws == p.nw) { ws = 0; ph ^= 1u; }
                }
            }
            // (a set without a group in this item has still to see every chunk's phase)
            for (; ready < chunks && ok; ++ready) ok = mbar_wait(&sh->a_ready[ready], (uint32_t)n & 1u);
            if (leader) {
                if (tchunks < chunks) umma_commit(&sh->tail_free);
                umma_commit(&sh->a_free);
            }
            __syncwarp();
        }
        if (!ok) give_up(44);
    } else if (warp >= kFirstEpi) {
        // ---- convert and store: set s has accumulator s, its eight warps a quarter of the rows and half of the columns each
        const int e = warp - kFirstEpi, q = warp & 3, set = e >> 3, half_of = (e >> 2) & 1;
        const uint32_t src = tmem + ((uint32_t)(q * 32) << 16) + kAccAt + set * kAccCols + half_of * 32;
        const bool bias_vec = (reinterpret_cast<uintptr_t>(p.bias) & 15) == 0;
        uint8_t* const buf = epi + (size_t)e * kUnitBytes;
        bool ok = true;
        uint32_t gs = 0;
        // (the weight's own bias is read without waiting: 4808 x 768 -> 2304 at 90 % 12.68 us, 12.83 with the wait)
        if (p.bias_given) pdl_wait();
        for (int item = blockIdx.x; item < p.items && ok; item += G) {
            const int r = item % p.ranges;
            const int g0 = r * p.groups / p.ranges, g1 = (r + 1) * p.groups / p.ranges;
            const int row = (item / p.ranges) * kSlab + q * 32;
            for (int g = g0; g < g1; ++g, ++gs) {
                if ((int)(gs & 1u) != set) continue;
                const int col = g * kAccCols + half_of * 32;
                const int cols = min(32, p.N - col);   // 32, 16, or nothing of this half exists
                uint4 bv[4];
                if (bias_vec) {
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        bv[c] = c * 8 < cols ? __ldg(reinterpret_cast<const uint4*>(p.bias + col) + c) : make_uint4(0u, 0u, 0u, 0u);
                } else {
                    half* b = reinterpret_cast<half*>(bv);
#pragma unroll
                    for (int c = 0; c < 32; ++c) b[c] = c < cols ? __ldg(p.bias + col + c) : __float2half(0.f);
                }
                const uint32_t e2 = kEmpty ? (__ldg(p.empty + g) >> (2 * half_of)) & 3u : 0u;
                ok = mbar_wait(&sh->acc_full[set], (gs >> 1) & 1u);
                if (!ok) break;
                tc_fence_after();
                if (item + G >= p.items && g + 2 >= g1) pdl_launch_dependents();   // the next kernel's set-up overlaps the last stores
                uint32_t acc[32];
                tmem_ld32(src, acc);
                tmem_ld_wait(acc);
                tc_fence_before();
                __syncwarp();
                if (elect_one()) mbar_arrive(&sh->acc_empty[set]);
                __syncwarp();
                if (kEmpty && e2) {   // what the zero tile of a block-row without tiles left is the bias alone, whatever the activations are
#pragma unroll
                    for (int i = 0; i < 32; ++i)
                        if ((e2 >> (i >> 4)) & 1u) acc[i] = 0u;
                }
                uint4 ov[4];
                epi_convert_regs<kGelu>(acc, bv, ov);
                if (lane == 0) tma_store_wait_read();   // the buffer's previous store has read it
                __syncwarp();
                epi_write(buf, lane, ov);
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) {
                    if (cols > 0 && row < p.T) tma_store_2d(&tmY, buf, col, row);
                    tma_store_commit();
                }
            }
        }
        if (lane == 0) tma_store_wait_read();
        if (!ok) give_up(45);
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 1) tmem_dealloc(tmem, 512);
}

}  // namespace

struct ResidentWeight {
    int K = 0, N = 0, groups = 0, parts = 1, block_bytes = 0, nx = 0, nw = 0;
    double group_clocks = 0;   // modelled, per group of 64 features and slab
    uint2* d_dir = nullptr;
    uint8_t* d_stream = nullptr;
    const uint8_t* d_empty = nullptr;   // behind the stream
    size_t bytes = 0;
};

// Clocks per group, fitted to launches of 128 to 32768 tokens (within 15 %): half of an accumulator's round (issuing, the last
// UMMAs' completion, hand-over to the converting warps and back), which grows with the tiles; a tile whose activations are
// read from shared memory counts for many.
static double group_clocks(int K, double density) {
    const double ts = kGroupRows * density * std::min(K / 16, kTmemSlices), ss = kGroupRows * density * std::max(0, K / 16 - kTmemSlices);
    return std::max(1000.0, 700.0 + 12.5 * ts) + 90.0 * ss;
}
static double launch_clocks(int slabs, int groups, int K, double per_group, int* ranges) {
    double best = 0;
    const double start = ((K + kKC - 1) / kKC) * 540.0 + 2000.0;   // copying a slab into place, per item
    for (int r = 1; r <= groups; ++r) {
        const int waves = (slabs * r + sm_count() - 1) / sm_count();
        const double c = 7500.0 + waves * (start + ((groups + r - 1) / r) * per_group);
        if (best == 0 || c < best * 0.999) { best = c; *ranges = r; }
    }
    return best;
}

double resident_cost(int tokens, int N, int K, double density) {
    if (K > kMaxK) return 1e30;
    int r = 1;
    return launch_clocks(std::max(1, (tokens + kSlab - 1) / kSlab), (N + kAccCols - 1) / kAccCols, K, group_clocks(K, density), &r);
}

int resident_pack(ResidentWeight** out, int K, int N, const half* data, const int* row_ptr, const int* row_offset) {
    *out = nullptr;
    if (K > kMaxK) return fail(ET_ERR_UNSUPPORTED, "resident linear: in_feat above 1024");
    const int NBR = N / 16, chunks = (K + kKC - 1) / kKC;
    auto* w = new ResidentWeight();
    w->K = K; w->N = N; w->groups = (NBR + kGroupRows - 1) / kGroupRows;
    w->group_clocks = group_clocks(K, (double)row_ptr[NBR] / std::max(1.0, (double)NBR * (K / 16)));
    const int avail = kSmemMax - 1024 - (int)sizeof(ResidentShared) - kEpiWarps * kUnitBytes - std::max(0, chunks - kTmemChunks) * kChunkBytes;
    std::vector<uint2> dir;
    std::vector<uint8_t> stream;
    // the fewest parts of the K range with which two blocks per set fit beside at least two slots for activations
    for (int parts = 1; parts <= chunks; ++parts) {
        dir.clear();
        stream.clear();
        size_t largest = 0;
        for (int g = 0; g < w->groups; ++g)
            for (int part = 0; part < parts; ++part) {
                const int s0 = part * chunks / parts * 8, s1 = (part + 1) * chunks / parts * 8;   // K slices of this part
                struct Ent { int slice, tile; };
                std::vector<Ent> lists[kGroupRows];
                size_t n = 0;
                for (int lb = 0; lb < kGroupRows; ++lb) {
                    const int r = g * kGroupRows + lb;
                    if (r >= NBR) continue;
                    for (int i = row_ptr[r]; i < row_ptr[r + 1]; ++i) {
                        const int s = row_offset[i] / 16;
                        if (s >= s0 && s < s1) lists[lb].push_back({s, i});
                    }
                    std::sort(lists[lb].begin(), lists[lb].end(), [](const Ent& a, const Ent& b) { return a.slice < b.slice; });
                    // a block-row without tiles gets one of zeros: its accumulator is then written like the others
                    if (part == 0 && row_ptr[r] == row_ptr[r + 1]) lists[lb].push_back({0, -1});
                    if (lists[lb].size() > kListBytes) { delete w; return fail(ET_ERR_UNSUPPORTED, "resident linear: a tile is listed twice"); }
                    n += lists[lb].size();
                }
                const size_t bytes = kHeadBytes + n * 512, off = stream.size();
                stream.resize(off + bytes, 0);
                uint8_t* blk = stream.data() + off;
                uint32_t start = 0;
                for (int lb = 0; lb < kGroupRows; ++lb) {
                    uint32_t nts = 0;
                    for (size_t i = 0; i < lists[lb].size(); ++i) {
                        const Ent& t = lists[lb][i];
                        nts += t.slice < kTmemSlices;
                        blk[64 + lb * kListBytes + i] = (uint8_t)t.slice;
                        if (t.tile < 0) continue;
                        uint8_t* dst = blk + kHeadBytes + (size_t)(start + i) * 512;
                        for (int r = 0; r < 16; ++r)
                            for (int k = 0; k < 16; k += 8)
                                std::memcpy(dst + (r / 8) * 256 + (k / 8) * 128 + (r % 8) * 16, data + (size_t)t.tile * 256 + r * 16 + k, 16);
                    }
                    reinterpret_cast<uint32_t*>(blk)[lb] = start | (nts << 16) | ((uint32_t)lists[lb].size() << 24);
                    start += (uint32_t)lists[lb].size();
                }
                dir.push_back(make_uint2((uint32_t)(off / 16), (uint32_t)(bytes / 16)));
                largest = std::max(largest, bytes);
            }
        w->parts = parts;
        w->block_bytes = (int)((largest + 127) / 128 * 128);
        for (int nx : {4, 3, 2})
            if (!w->nx && nx * kChunkBytes + kSets * 2 * w->block_bytes <= avail) { w->nx = nx; w->nw = 2; }
        if (w->nx) break;
    }
    if (!w->nx) { delete w; return fail(ET_ERR_UNSUPPORTED, "resident linear: weight blocks exceed shared memory"); }
    w->bytes = stream.size();
    std::vector<uint8_t> empty(w->groups, 0);
    for (int r = 0; r < NBR; ++r)
        if (row_ptr[r] == row_ptr[r + 1]) empty[r / kGroupRows] |= (uint8_t)(1u << (r % kGroupRows));
    const bool any_empty = std::any_of(empty.begin(), empty.end(), [](uint8_t e) { return e != 0; });
    if (any_empty) stream.insert(stream.end(), empty.begin(), empty.end());
    if (cudaMalloc(&w->d_dir, dir.size() * sizeof(uint2)) != cudaSuccess || cudaMalloc(&w->d_stream, stream.size()) != cudaSuccess) {
        resident_free(w);
        return fail(ET_ERR_CUDA, "resident linear: cudaMalloc failed");
    }
    cudaMemcpy(w->d_dir, dir.data(), dir.size() * sizeof(uint2), cudaMemcpyHostToDevice);
    const int rc = cuda_status(cudaMemcpy(w->d_stream, stream.data(), stream.size(), cudaMemcpyHostToDevice), "resident linear: upload");
    if (rc) { resident_free(w); return rc; }
    if (any_empty) w->d_empty = w->d_stream + w->bytes;
    *out = w;
    return ET_OK;
}

void resident_free(ResidentWeight* w) {
    if (!w) return;
    cudaFree(w->d_dir);
    cudaFree(w->d_stream);
    delete w;
}

size_t resident_bytes(const ResidentWeight* w) { return w->bytes; }

int resident_run(const ResidentWeight* w, half* Y, const half* X, const half* bias, bool bias_given, int T, int gelu, int* err, cudaStream_t st) {
    CUtensorMap tm, tmy;
    if (!make_tmap_panels_f16(&tm, X, (uint64_t)T, (uint64_t)w->K, (uint64_t)w->K, kSlab, 2) ||
        !make_tmap_2d_f16(&tmy, Y, (uint64_t)T, (uint64_t)w->N, (uint64_t)w->N, 32, 32, 64))
        return fail(ET_ERR_CUDA, "resident linear: cuTensorMapEncodeTiled failed");
    static PerDeviceOnce once;
    using KernelFn = void (*)(CUtensorMap, CUtensorMap, ResidentParams);
    static const KernelFn kernels[2][2] = {{resident_kernel<false, false>, resident_kernel<false, true>},
                                           {resident_kernel<true, false>, resident_kernel<true, true>}};
    const cudaError_t attr_err = once.run([] {
        cudaError_t e = cudaSuccess;
        for (int i = 0; i < 4 && e == cudaSuccess; ++i)
            e = cudaFuncSetAttribute(kernels[i >> 1][i & 1], cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax);
        return e;
    });
    if (attr_err != cudaSuccess) return cuda_status(attr_err, "resident linear: shared memory opt-in");
    ResidentParams p;
    p.dir = w->d_dir; p.stream = w->d_stream; p.bias = bias; p.bias_given = bias_given; p.empty = w->d_empty;
    p.T = T; p.N = w->N; p.K = w->K; p.groups = w->groups; p.parts = w->parts;
    p.slabs = (T + kSlab - 1) / kSlab;
    launch_clocks(p.slabs, w->groups, w->K, w->group_clocks, &p.ranges);
    p.items = p.slabs * p.ranges;
    p.nx = w->nx; p.nw = w->nw; p.block_bytes = w->block_bytes; p.err = err;
    const int chunks = (w->K + kKC - 1) / kKC;
    const size_t smem = (size_t)(std::max(0, chunks - kTmemChunks) + w->nx) * kChunkBytes + (size_t)kSets * w->nw * w->block_bytes + kEpiWarps * kUnitBytes + sizeof(ResidentShared) + 1024;
    return cuda_status(launch_pdl(kernels[gelu ? 1 : 0][w->d_empty ? 1 : 0], dim3((unsigned)std::min(p.items, sm_count())),
                                  dim3(kThreads), smem, st, tm, tmy, p),
                       "resident linear launch");
}

}  // namespace et
