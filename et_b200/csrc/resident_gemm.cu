// Tile-sparse linear  Y[T x N] = X[T x K] . W^T + bias  (optional tanh-GELU), W in 16x16 tile-BSR, for in_feat up to 1024: a
// slab of 128 tokens stays in tensor memory, whole, while the weight streams past it.
// Replaces, for those sizes, kernels/linear.cu:54-167 of the reference.
//
// Why: with A in tensor memory a kept tile is one UMMA 128x16x16 of ~9 clocks (eight issuing warps, or six), but bringing A there is
// dear: tcgen05.cp moves 64 bytes per clock and takes turns with the UMMAs on the tensor pipe (measured: 2048 UMMAs and 256
// copies of 4 KB take the sum of their times). The tile kernel (tile_gemm.cu) keeps 384 accumulator columns and streams A
// through the other 128 once per 384 output features: 512 clocks of copying per 128 x 128 chunk against ~350 of UMMAs at
// 80 % sparsity. Here A is copied once per slab and CTA: 768 inputs take 384 columns, and the other 128 hold four accumulators
// of 32 features, so that some are converted and stored while others are multiplied. Inputs beyond 768 (832 with three accumulators) stay in shared
// memory, as the A operand of UMMAs that read it there (~50 clocks a tile).
// What bounds it: with K = 768 the stores at 75 % sparsity and above (17771 x 768 -> 2304 at 75 % 26.1 us, of which 17 are the bytes at the copy
// bandwidth; without its stores 23), with GELU the converting warps (37.9 us; a warp has 16 packed tanh to a unit, 256 clocks of the special-function
// unit alone, ~870 with the three other warps of its scheduler), with K = 1024 the UMMAs that read shared memory.
//
// The weight is re-packed once into blocks of 32 features, or of a part of such a group's tiles where a block would exceed its slot: per issuing warp
// a list of K slices, one byte per tile, then the tiles in UMMA layout. Roles: a warp copies activations, one moves them to tensor memory, and each accumulator has
// a warp that copies its weight blocks (one that has requested a copy goes on only after ~700 clocks), two that issue (a block-row of 16 features each) and four that
// convert and store. These sets run apart: while one accumulator is handed over and drained, the others' UMMAs are issued. With two accumulators of 64 features (and each
// half handed over by itself) 8192 x 768 -> 2304 at 50 % took 21.1 us (20.5 now), 17771 x 768 -> 2304 at 75 % 26.8 (26.1), handed over whole 27.9. A CTA
// takes (slab, range of features) items; the number of ranges is chosen at the launch so that the last wave is full.
// Tried and dropped (17771 x 768 -> 2304, 27.9 us then): one issuing warp for 32 features 35, two for 64 29.2, a token that lets the sets
// issue in turn 33, stores from registers or through shared memory instead of TMA stores 34, one TMA store per 128 x 64 tile by warps of their own 28.7;
// two warps that copy activations +1 %; lane 0 instead of an elected lane for the UMMAs 30.1 (26.7), for tcgen05.cp 300 x 1024 -> 1024 at 90 % 7.2 (5.8).
// Every mbarrier wait is bounded; a role that gives up records a code and all threads meet at the common exit.
#include <algorithm>
#include <cstring>
#include <type_traits>
#include <vector>
#include "common.h"
#include "epilogue.cuh"
#include "ptx.cuh"
#include "resident_gemm.h"
#include "tmap.h"

namespace et {

namespace {

constexpr int kSlab = 128;
constexpr int kPanelBytes = kSlab * 64 * 2;       // 16 KB: 64 K elements, 128-byte-swizzled
constexpr int kMaxK = 1024;
constexpr int kListBytes = 64;                    // entries per issuing warp and block: a byte for each K slice of kMaxK
constexpr int kMaxRing = 8;                       // slots for chunks, at most
constexpr int kSlots = 2;                         // weight slots per set
constexpr uint32_t kLast = 0x8000u;               // in a block's header: the last block of its group
constexpr int kRows = 2;                          // block-rows per group of features and accumulator, one per issuing warp
constexpr int kAccCols = 16 * kRows;
constexpr int kHeadBytes = 64 + kRows * kListBytes;
// How tensor memory is shared out: 16-wide K slices of the activations (8 columns each), and accumulators, each with its own copying, two
// issuing and four converting warps ("a set").
template <int kSets_, int kSlices_, int kPanels_, int kLeastRing_>
struct Shape {
    static constexpr int kSets = kSets_, kSlices = kSlices_;
    static constexpr int kPanels = kPanels_;          // per copied chunk of activations
    static constexpr int kLeastRing = kLeastRing_;    // slots for chunks, at least
    static constexpr int kChunkSlices = 4 * kPanels, kChunkBytes = kPanels * kPanelBytes, kMaxChunks = kMaxK / 16 / kChunkSlices, kTmemChunks = kSlices / kChunkSlices;
    static constexpr uint32_t kAccAt = kSlices * 8;
    static constexpr int kFirstCopier = 2, kFirstIssuer = kFirstCopier + kSets, kIssuers = kSets * kRows, kFirstEpi = kFirstIssuer + kIssuers, kEpiWarps = kSets * 4;
    static constexpr int kThreads = 32 * (kFirstEpi + kEpiWarps);
    static_assert(kSlices % kChunkSlices == 0 && kAccAt + kSets * kAccCols <= 512, "tensor memory");
};
// Up to 768 inputs all fit beside four accumulators. Beyond that a tile of what does not fit costs ~50 clocks instead of ~9: one accumulator less holds
// four slices more, in chunks of one panel so that the ring leaves room for weights (131072 x 1024 -> 4096 + GELU at 80 % 374 instead of 423 us, 32768 x 1024 -> 3072 77.5
// instead of 88.9, at 90 % 65.6 instead of 63.9; with two accumulators and 56 slices 418, 87 and 81).
using Narrow = Shape<4, 48, 2, 2>;
using Wide = Shape<3, 52, 1, 3>;
constexpr int kUnitBytes = 32 * 32 * 2;
constexpr int kSmemMax = 232448;

struct ResidentParams {
    const uint2* dir;         // per group: {offset of its blocks, their number << 16 | size of each}, in 16-byte units
    const uint8_t* stream;
    const half* bias;
    bool bias_given;          // the caller's, not the weight's own: the preceding kernel may still be writing it
    const uint8_t* empty;     // per group, a bit per block-row without tiles; null when there is none
    int T, N, K, groups, ranges, items, slabs;
    int nx, block_bytes;
    int* err;
};

template <typename F>
struct ResidentShared {
    uint64_t x_full[kMaxRing], x_empty[kMaxRing];   // chunk slots: landed / copied on to tensor memory
    uint64_t w_full[F::kSets][kSlots], w_empty[F::kSets][kSlots];   // weight blocks: landed / their UMMAs have completed (a commit of each issuing warp)
    uint64_t a_ready[F::kMaxChunks];                   // per chunk, once per item: in place for the UMMAs
    uint64_t a_free, tail_free;                     // the item's UMMAs have completed: its activations in tensor memory, in shared memory may be overwritten
    uint64_t acc_full[F::kSets], acc_empty[F::kSets];
    uint32_t tmem_base;
    volatile int abort;
    __align__(16) half bias[F::kEpiWarps][32];         // of the unit that a converting warp works on
};

__device__ __forceinline__ void cp_128x256b(uint32_t taddr, uint64_t sdesc) {
    asm volatile("tcgen05.cp.cta_group::1.128x256b [%0], %1;" ::"r"(taddr), "l"(sdesc) : "memory");
}

// kEmpty: some block-row has no tiles.
template <typename F, bool kGelu, bool kEmpty>
__global__ void __launch_bounds__(F::kThreads, 1) resident_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmY,
                                                               const __grid_constant__ ResidentParams p) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    constexpr int kSets = F::kSets, kChunkBytes = F::kChunkBytes;
    const int chunks = (p.K / 16 + F::kChunkSlices - 1) / F::kChunkSlices, tchunks = min(chunks, F::kTmemChunks);
    uint8_t* const tail = smem;                                                    // chunks beyond the tensor-memory part
    uint8_t* const xring = tail + (size_t)(chunks - tchunks) * kChunkBytes;
    uint8_t* const wring = xring + (size_t)p.nx * kChunkBytes;
    uint8_t* const epi = wring + (size_t)kSets * kSlots * p.block_bytes;           // a unit per converting warp
    ResidentShared<F>* const sh = reinterpret_cast<ResidentShared<F>*>(epi + F::kEpiWarps * kUnitBytes);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int G = gridDim.x;

    if (tid == 0) {
        for (int i = 0; i < kMaxRing; ++i) { mbar_init(&sh->x_full[i], 1); mbar_init(&sh->x_empty[i], 1); }
        for (int i = 0; i < F::kMaxChunks; ++i) mbar_init(&sh->a_ready[i], 1);
        mbar_init(&sh->a_free, F::kIssuers);
        mbar_init(&sh->tail_free, F::kIssuers);
        for (int k = 0; k < kSets; ++k) {
            for (int i = 0; i < kSlots; ++i) { mbar_init(&sh->w_full[k][i], 1); mbar_init(&sh->w_empty[k][i], kRows); }
            mbar_init(&sh->acc_full[k], kRows);
            mbar_init(&sh->acc_empty[k], 4);
        }
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
        const uint32_t full0 = smem_u32(&sh->x_full[0]), empty0 = smem_u32(&sh->x_empty[0]), ring0 = smem_u32(xring);
        bool ok = true;
        int xs = 0;
        uint32_t ph = 1, ptail = 1;
        for (int item = blockIdx.x; item < p.items && ok; item += G) {
            const int row = (item / p.ranges) * kSlab;
            for (int c = 0; c < tchunks; ++c) {
                ok = mbar_wait_at(empty0 + xs * 8, ph);
                if (!ok) break;
                if (elect_one()) {
                    mbar_expect_tx_at(full0 + xs * 8, kChunkBytes);
                    tma_load_3d_at(ring0 + xs * kChunkBytes, &tmX, 0, row, F::kPanels * c, full0 + xs * 8);
                }
                __syncwarp();
                if (++xs == p.nx) { xs = 0; ph ^= 1u; }
            }
            if (ok && tchunks < chunks) {
                ok = mbar_wait(&sh->tail_free, ptail);
                ptail ^= 1u;
                if (ok && elect_one())
                    for (int c = tchunks; c < chunks; ++c) {
                        mbar_expect_tx(&sh->a_ready[c], kChunkBytes);
                        tma_load_3d(tail + (size_t)(c - tchunks) * kChunkBytes, &tmX, 0, row, F::kPanels * c, &sh->a_ready[c]);
                    }
                __syncwarp();
            }
        }
        if (!ok) give_up(41);
    } else if (warp >= F::kFirstCopier && warp < F::kFirstIssuer) {
        // ---- weight blocks of one set (they do not depend on the preceding kernel)
        const int set = warp - F::kFirstCopier;
        bool ok = true;
        int ws = 0, turn = 0;   // the set of the item's first group
        uint32_t ph = 1;
        for (int item = blockIdx.x; item < p.items && ok; item += G) {
            const int r = item % p.ranges;
            const int g0 = r * p.groups / p.ranges, g1 = (r + 1) * p.groups / p.ranges;
            const int first = g0 + (set - turn + kSets) % kSets;
            turn = (turn + g1 - g0) % kSets;
            for (int g = first; g < g1 && ok; g += kSets) {
                const uint2 d = __ldg(p.dir + g);
                const uint32_t bytes = (d.y & 0xffffu) * 16u;
                const uint8_t* src = p.stream + (size_t)d.x * 16u;
                for (uint32_t left = d.y >> 16; left > 0; --left, src += bytes) {
                    ok = mbar_wait(&sh->w_empty[set][ws], ph);
                    if (!ok) break;
                    if (elect_one()) {
                        mbar_expect_tx(&sh->w_full[set][ws], bytes);
                        bulk_load(wring + (size_t)(set * kSlots + ws) * p.block_bytes, src, bytes, &sh->w_full[set][ws]);
                    }
                    __syncwarp();
                    if (++ws == kSlots) { ws = 0; ph ^= 1u; }
                }
            }
        }
        if (!ok) give_up(42);
    } else if (warp == 1) {
        // ---- shared memory -> tensor memory. The columns are free when the previous item's UMMAs have completed: a copy is
        // guaranteed to run ahead of UMMAs issued after it, but not behind those issued before it.
        const uint32_t full0 = smem_u32(&sh->x_full[0]), empty0 = smem_u32(&sh->x_empty[0]), ready0 = smem_u32(&sh->a_ready[0]);
        const uint64_t x_desc0 = make_smem_desc(smem_u32(xring), 16, 1024, 2);
        const int slices = min(p.K / 16, F::kSlices);
        bool ok = true;
        if (elect_one()) {
            int xs = 0, n = 0;
            uint32_t ph = 0;
            for (int item = blockIdx.x; item < p.items && ok; item += G, ++n) {
                if (n > 0) ok = mbar_wait(&sh->a_free, (uint32_t)(n - 1) & 1u);
                for (int c = 0; c < tchunks && ok; ++c) {
                    ok = mbar_wait_at(full0 + xs * 8, ph);
                    if (!ok) break;
                    tc_fence_after();
                    const uint64_t xd = x_desc0 + (uint32_t)xs * (kChunkBytes >> 4);
                    const uint32_t ta = tmem + c * F::kChunkSlices * 8;
                    if (slices - c * F::kChunkSlices >= F::kChunkSlices) {
#pragma unroll
                        for (int s = 0; s < F::kChunkSlices; ++s) cp_128x256b(ta + s * 8, xd + (((s >> 2) * kPanelBytes + (s & 3) * 32) >> 4));
                    } else {
                        for (int s = 0; s < slices - c * F::kChunkSlices; ++s) cp_128x256b(ta + s * 8, xd + (((s >> 2) * kPanelBytes + (s & 3) * 32) >> 4));
                    }
                    umma_commit_at(ready0 + c * 8);
                    umma_commit_at(empty0 + xs * 8);
                    if (++xs == p.nx) { xs = 0; ph ^= 1u; }
                }
            }
            if (!ok) {
                if (!sh->abort) atomicExch(p.err, 43);
                sh->abort = 1;
            }
        }
        __syncwarp();
    } else if (warp >= F::kFirstIssuer && warp < F::kFirstEpi) {
        // ---- UMMAs: every kSets-th group, block-row w of it. One lane is the whole role. What it executes between two UMMAs is what a
        // group waits for: shared memory by 32-bit addresses, pointers carried along, one loop per kind of block. (Generic pointers, addresses
        // made of indexes and a branch per case cost ~280 clocks for every wait on a barrier that had completed, 65 now, and ~95 per
        // UMMA of eight warps, 65 now, which is the tensor pipe: 17771 x 768 -> 2304 at 75 % 31.1 instead of 29.2 us.)
        const int w = (warp - F::kFirstIssuer) % kRows, set = (warp - F::kFirstIssuer) / kRows;
        const uint64_t t_desc0 = make_smem_desc(smem_u32(tail), 16, 1024, 2);
        const uint64_t b_desc0 = make_smem_desc(0, 128, 256, 0);   // no swizzle: 128 B between core matrices along K, 256 B along N
        const uint32_t b_hi = (uint32_t)(b_desc0 >> 32), b_lo = (uint32_t)b_desc0;
        constexpr uint32_t idesc = make_idesc_f16(128, 16);
        const uint32_t d = tmem + F::kAccAt + set * kAccCols + (uint32_t)w * 16;
        const uint32_t block_bytes = p.block_bytes, ring0 = smem_u32(wring) + set * kSlots * block_bytes, ring1 = ring0 + kSlots * block_bytes;
        const uint32_t full0 = smem_u32(&sh->w_full[set][0]), to_empty = smem_u32(&sh->w_empty[set][0]) - full0;
        const uint32_t acc_full = smem_u32(&sh->acc_full[set]), acc_empty = smem_u32(&sh->acc_empty[set]);
        if (elect_one()) {
            bool ok = true;
            int n = 0;
            uint32_t blk = ring0, full = full0, ph = 0, acc_ph = 1;
            int turn = 0;
            auto b_desc = [&](uint32_t at) { return (uint64_t)b_hi << 32 | at; };
            auto tail_desc = [&](uint32_t k) {
                const uint32_t t = k - F::kSlices;
                return t_desc0 + (uint64_t)(((t >> 2) * kPanelBytes + (t & 3) * 32) >> 4);
            };
            auto finish_block = [&](bool last) {
                umma_commit_at(full + to_empty);
                if (last) umma_commit_at(acc_full);
                blk += block_bytes;
                full += 8;
                if (blk == ring1) { blk = ring0; full = full0; ph ^= 1u; }
            };
            for (int item = blockIdx.x; item < p.items && ok; item += G, ++n) {
                const int r = item % p.ranges;
                const int g0 = r * p.groups / p.ranges, g1 = (r + 1) * p.groups / p.ranges;
                int left = (g1 - g0 - (set - turn + kSets) % kSets + kSets - 1) / kSets;   // groups of this set
                turn = (turn + g1 - g0) % kSets;
                int ready = 0;   // chunks of the item known to be in place
                auto follow = [&](int chunk) {
                    for (; ok && ready <= chunk; ++ready) {
                        ok = mbar_wait(&sh->a_ready[ready], (uint32_t)n & 1u);
                        tc_fence_after();
                    }
                };
                if (left > 0) {   // the set's first group follows the chunks
                    ok = mbar_wait_at(acc_empty, acc_ph);
                    acc_ph ^= 1u;
                    uint32_t accumulate = 0;   // the block-row's first UMMA overwrites
                    for (bool last = false; ok && !last;) {
                        ok = mbar_wait_at(full, ph);
                        if (!ok) break;
                        tc_fence_after();
                        const uint32_t hdr = lds32(blk + w * 4), list = blk + 64 + w * kListBytes, bd = b_lo + ((blk + kHeadBytes + (hdr & (kLast - 1)) * 512u) >> 4);
                        last = hdr & kLast;
                        const uint32_t nall = hdr >> 24;
                        for (uint32_t i = 0; i < nall; ++i) {
                            const uint32_t k = lds8(list + i);
                            follow(k / F::kChunkSlices);
                            if (!ok) break;
                            if (k < (uint32_t)F::kSlices) umma_f16_ts(d, tmem + k * 8u, b_desc(bd + i * 32), idesc, accumulate);
                            else umma_f16(d, tail_desc(k), b_desc(bd + i * 32), idesc, accumulate);
                            accumulate = 1;
                        }
                        if (last) follow(chunks - 1);
                        if (ok) finish_block(last);
                    }
                    --left;
                }
                bool fresh = true;   // the block is the first of its group
                uint32_t accumulate = 0;
#pragma unroll 1
                while (ok && left > 0) {
                    if (!mbar_wait_at(full, ph)) { ok = false; break; }
                    const uint32_t hdr = lds32(blk + w * 4);
                    uint32_t list = blk + 64 + w * kListBytes;
                    uint4 e = lds128(list);   // sixteen entries
                    if (fresh) {
                        if (!mbar_wait_at(acc_empty, acc_ph)) { ok = false; break; }
                        acc_ph ^= 1u;
                        accumulate = 0;
                    }
                    tc_fence_after();
                    // the tiles whose activations are in tensor memory, then those that read them from shared memory
                    int nts = (hdr >> 16) & 0xff, nss = (int)(hdr >> 24) - nts;
                    uint32_t bd = b_lo + ((blk + kHeadBytes + (hdr & (kLast - 1)) * 512u) >> 4);
                    auto ts = [&](uint32_t k, uint32_t off, uint32_t acc) { umma_f16_ts(d, tmem + k * 8u, b_desc(bd + off), idesc, acc); };
#pragma unroll 1
                    for (; nts >= 4; nts -= 4) {
                        ts(e.x & 0xffu, 0, accumulate);
                        ts((e.x >> 8) & 0xffu, 32, 1u);
                        ts((e.x >> 16) & 0xffu, 64, 1u);
                        ts(e.x >> 24, 96, 1u);
                        accumulate = 1;
                        bd += 128;
                        list += 4;
                        e.x = e.y; e.y = e.z; e.z = e.w;
                        if (!(list & 15)) e = lds128(list);
                    }
                    if (nts > 0) {
                        ts(e.x & 0xffu, 0, accumulate);
                        if (nts > 1) ts((e.x >> 8) & 0xffu, 32, 1u);
                        if (nts > 2) ts((e.x >> 16) & 0xffu, 64, 1u);
                        accumulate = 1;
                        bd += nts * 32;
                        list += nts;
                    }
#pragma unroll 1
                    for (; nss > 0; --nss) {
                        umma_f16(d, tail_desc(lds8(list)), b_desc(bd), idesc, accumulate);
                        accumulate = 1;
                        bd += 32;
                        ++list;
                    }
                    fresh = hdr & kLast;
                    finish_block(fresh);
                    if (fresh) --left;
                }
                // (a set without a group in this item has still to see every chunk's phase)
                follow(chunks - 1);
                if (tchunks < chunks) umma_commit(&sh->tail_free);
                umma_commit(&sh->a_free);
            }
            if (!ok) {
                if (!sh->abort) atomicExch(p.err, 44);
                sh->abort = 1;
            }
        }
        __syncwarp();
    } else if (warp >= F::kFirstEpi) {
        // ---- convert and store: set s has accumulator s, its four warps a quarter of the rows each
        const int e = warp - F::kFirstEpi, q = warp & 3, set = e >> 2;
        const uint32_t src = tmem + ((uint32_t)(q * 32) << 16) + F::kAccAt + set * kAccCols;
        const uint32_t acc_full = smem_u32(&sh->acc_full[set]), acc_empty = smem_u32(&sh->acc_empty[set]);
        const uint32_t bias_at = smem_u32(sh->bias[e]);
        uint8_t* const buf = epi + (size_t)e * kUnitBytes;
        const uint32_t to = smem_u32(buf) + lane * 64, swizzle = (lane >> 1) & 3;   // row `lane`: four 16-byte chunks under the 64-byte swizzle
        bool ok = true;
        uint32_t ph = 0;
        int turn = 0;
        // (the weight's own bias is read without waiting: 4808 x 768 -> 2304 at 90 % 12.68 us, 12.83 with the wait)
        if (p.bias_given) pdl_wait();
        for (int item = blockIdx.x; item < p.items && ok; item += G) {
            const int r = item % p.ranges;
            const int g0 = r * p.groups / p.ranges, g1 = (r + 1) * p.groups / p.ranges;
            const int row = (item / p.ranges) * kSlab + q * 32;
            const int g = g0 + (set - turn + kSets) % kSets;
            turn = (turn + g1 - g0) % kSets;
            int col = g * kAccCols;   // columns from N on do not exist
            // A lane has one column's bias, read a unit ahead; a unit passes them on through shared memory (as four wide loads by every lane
            // 17771 x 768 -> 2304 at 75 % 27.1 instead of 26.8 us).
            auto bias_of = [&](int c) { return c + lane < p.N ? __ldg(reinterpret_cast<const uint16_t*>(p.bias) + c + lane) : (uint16_t)0; };
            uint16_t b = g < g1 ? bias_of(col) : (uint16_t)0;
#pragma unroll 1
            for (int left = (g1 - g + kSets - 1) / kSets; left > 0; --left) {
                const uint32_t e2 = kEmpty ? __ldg(p.empty + col / kAccCols) : 0u;
                sts16(bias_at + lane * 2, b);
                if (!mbar_wait_at(acc_full, ph)) { ok = false; break; }
                ph ^= 1u;
                tc_fence_after();
                if (left == 1 && item + G >= p.items) pdl_launch_dependents();   // the next kernel's set-up overlaps the last stores
                uint32_t acc[32];
                tmem_ld32(src, acc);
                tmem_ld_wait(acc);
                tc_fence_before();
                __syncwarp();
                if (elect_one()) mbar_arrive_at(acc_empty);
                if (kEmpty && e2) {   // what the zero tile of a block-row without tiles left is the bias alone, whatever the activations are
#pragma unroll
                    for (int i = 0; i < 32; ++i)
                        if ((e2 >> (i >> 4)) & 1u) acc[i] = 0u;
                }
                uint4 bv[4], ov[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) bv[c] = lds128(bias_at + c * 16);
                epi_convert_regs<kGelu>(acc, bv, ov);
                if (left > 1) b = bias_of(col + kSets * kAccCols);
                tma_store_wait_read();   // the buffer's previous store has read it
                __syncwarp();
#pragma unroll
                for (int c = 0; c < 4; ++c) sts128(to + ((c ^ swizzle) << 4), ov[c]);
                fence_proxy_async_smem();
                __syncwarp();
                if (col < p.N && row < p.T && elect_one()) {
                    tma_store_2d(&tmY, buf, col, row);
                    tma_store_commit();
                }
                __syncwarp();
                col += kSets * kAccCols;
            }
        }
        tma_store_wait_read();
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
    int K = 0, N = 0, groups = 0, block_bytes = 0, nx = 0;
    bool wide = false;
    double group_clocks = 0;   // modelled, per group of features and slab
    uint2* d_dir = nullptr;
    uint8_t* d_stream = nullptr;
    const uint8_t* d_empty = nullptr;   // behind the stream
    size_t bytes = 0;
};

// Clocks per group, fitted to 342 launches of 128 to 65536 tokens (rms 11 %) together with the choice between the forms: an accumulator's round (issuing, the
// last UMMAs' completion, hand-over to the converting warps and back) over the number of accumulators, which grows with the tiles and is never
// shorter than the converting warps' round; a tile whose activations are read from shared memory counts for six.
template <typename F>
static double group_clocks(int K, double density) {
    constexpr bool narrow = std::is_same<F, Narrow>::value;
    const double ts = kRows * density * std::min(K / 16, F::kSlices), ss = kRows * density * std::max(0, K / 16 - F::kSlices);
    return narrow ? std::max(420.0, 274.0 + 10.5 * ts) : std::max(530.0, 164.0 + 10.0 * ts + 64.0 * ss);
}
static double launch_clocks(int slabs, int groups, int K, double per_group, int* ranges) {
    double best = 0;
    const double start = ((K + 127) / 128) * 350.0 + 4400.0;   // copying a slab into place, per item
    const int sms = sm_count();
    // Of the numbers of ranges with as many groups in the largest only the first can be the best (this runs at every launch: 128 groups all tried 0.61 us, 0.22 now).
    for (int r = 1;;) {
        const int most = (groups + r - 1) / r, waves = (slabs * r + sms - 1) / sms;
        const double c = 5200.0 + waves * (start + most * per_group);
        if (best == 0 || c < best * 0.999) { best = c; *ranges = r; }
        if (most == 1) return best;
        r = (groups + most - 2) / (most - 1);
    }
}

static bool is_wide(int K) { return K / 16 > Narrow::kSlices; }

double resident_cost(int tokens, int N, int K, double density) {
    if (K > kMaxK) return 1e30;
    int r = 1;
    const int slabs = std::max(1, (tokens + kSlab - 1) / kSlab), groups = (N / 16 + kRows - 1) / kRows;
    const bool wide = is_wide(K);
    double clocks = launch_clocks(slabs, groups, K, wide ? group_clocks<Wide>(K, density) : group_clocks<Narrow>(K, density), &r);
    // Measured / modelled from L2 and from memory (means over in_feat 768 and 1024): 0.94 and 1.20. With a quarter of the tiles or less 0.85 from L2 (and 0.95 in the tile form). A slab from memory takes
    // longer with the ring of single panels, which covers L2's latency (65536 x 1024 -> 512 at 90 % 47 us, tile 40; 65536 x 1024 -> 1024 62 and 70).
    const double far = beyond_l2(tokens, K, N);
    if (tokens >= 2048 && density <= 0.3) clocks *= 0.93 + 0.07 * far;
    return wide ? (1.0 + 0.12 * far) * clocks + (slabs + sm_count() - 1) / sm_count() * 3000.0 * far : (1.0 + 0.1 * far) * clocks;
}

template <typename F>
static int pack(ResidentWeight** out, int K, int N, const half* data, const int* row_ptr, const int* row_offset) {
    const int NBR = N / 16, chunks = (K / 16 + F::kChunkSlices - 1) / F::kChunkSlices;
    auto* w = new ResidentWeight();
    w->K = K; w->N = N; w->groups = (NBR + kRows - 1) / kRows;
    w->wide = std::is_same<F, Wide>::value;
    w->group_clocks = group_clocks<F>(K, (double)row_ptr[NBR] / std::max(1.0, (double)NBR * (K / 16)));
    const int avail = kSmemMax - 1024 - (int)sizeof(ResidentShared<F>) - F::kEpiWarps * kUnitBytes - std::max(0, chunks - F::kTmemChunks) * F::kChunkBytes;
    // Tiles of each group in the order of their K slices (a block-row without tiles gets one of zeros: its accumulator is then written like the others).
    struct Ent { int slice, row, tile; };
    std::vector<std::vector<Ent>> tiles(w->groups);
    size_t most = 0;
    for (int r = 0; r < NBR; ++r) {
        auto& v = tiles[r / kRows];
        if (r % kRows == 0) v.reserve(row_ptr[std::min(r + kRows, NBR)] - row_ptr[r] + kRows);
        if (row_ptr[r + 1] - row_ptr[r] > kListBytes) { delete w; return fail(ET_ERR_UNSUPPORTED, "resident linear: a tile is listed twice"); }
        for (int i = row_ptr[r]; i < row_ptr[r + 1]; ++i) v.push_back({row_offset[i] / 16, r % kRows, i});
        if (row_ptr[r] == row_ptr[r + 1]) v.push_back({0, r % kRows, -1});
        most = std::max(most, v.size());
    }
    size_t listed = 0;
    for (auto& v : tiles) {
        std::stable_sort(v.begin(), v.end(), [](const Ent& a, const Ent& b) { return a.slice < b.slice; });
        listed += v.size();
    }
    // Slots for activations as long as every group fits in one block beside them; two at least, and then the groups that do not fit are cut into
    // equal blocks. (Cut at the same K slices everywhere, into as many as the largest needs, 131072 x 1024 -> 1024 at 80 % took 150 instead of 141 us
    // when a kilobyte was short.)
    auto room = [&](int nx) { return (avail - nx * F::kChunkBytes) / (F::kSets * kSlots) / 128 * 128; };
    w->nx = F::kLeastRing;
    for (int nx = kMaxRing / F::kPanels; nx > F::kLeastRing; --nx)
        if (w->nx == F::kLeastRing && (long)room(nx) >= (long)(kHeadBytes + most * 512)) w->nx = nx;
    const size_t cap = (size_t)(room(w->nx) - kHeadBytes) / 512;
    std::vector<uint2> dir;
    std::vector<uint8_t> stream;
    stream.reserve(listed * 520 + tiles.size() * 3 * kHeadBytes);
    for (const auto& v : tiles) {
        const size_t parts = (v.size() + cap - 1) / cap, bytes = kHeadBytes + (v.size() + parts - 1) / parts * 512, off = stream.size();
        stream.resize(off + parts * bytes, 0);
        for (size_t part = 0; part < parts; ++part) {
            uint8_t* blk = stream.data() + off + part * bytes;
            const size_t first = part * v.size() / parts, end = (part + 1) * v.size() / parts;
            uint32_t at = 0;
            for (int lb = 0; lb < kRows; ++lb) {
                const uint32_t start = at;
                uint32_t nts = 0;
                for (size_t i = first; i < end; ++i) {
                    const Ent& t = v[i];
                    if (t.row != lb) continue;
                    nts += t.slice < F::kSlices;
                    blk[64 + lb * kListBytes + (at - start)] = (uint8_t)t.slice;
                    uint8_t* dst = blk + kHeadBytes + (size_t)at++ * 512;
                    if (t.tile < 0) continue;
                    for (int r = 0; r < 16; ++r)
                        for (int k = 0; k < 16; k += 8)
                            std::memcpy(dst + (r / 8) * 256 + (k / 8) * 128 + (r % 8) * 16, data + (size_t)t.tile * 256 + r * 16 + k, 16);
                }
                reinterpret_cast<uint32_t*>(blk)[lb] = start | (part + 1 == parts ? kLast : 0) | (nts << 16) | ((at - start) << 24);
            }
        }
        dir.push_back(make_uint2((uint32_t)(off / 16), (uint32_t)(parts << 16 | bytes / 16)));
        w->block_bytes = std::max(w->block_bytes, (int)((bytes + 127) / 128 * 128));
    }
    w->bytes = stream.size();
    std::vector<uint8_t> empty(w->groups, 0);
    for (int r = 0; r < NBR; ++r)
        if (row_ptr[r] == row_ptr[r + 1]) empty[r / kRows] |= (uint8_t)(1u << (r % kRows));
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

int resident_pack(ResidentWeight** out, int K, int N, const half* data, const int* row_ptr, const int* row_offset) {
    *out = nullptr;
    if (K > kMaxK) return fail(ET_ERR_UNSUPPORTED, "resident linear: in_feat above 1024");
    return is_wide(K) ? pack<Wide>(out, K, N, data, row_ptr, row_offset) : pack<Narrow>(out, K, N, data, row_ptr, row_offset);
}

void resident_free(ResidentWeight* w) {
    if (!w) return;
    cudaFree(w->d_dir);
    cudaFree(w->d_stream);
    delete w;
}

size_t resident_bytes(const ResidentWeight* w) { return w->bytes; }
int resident_block_rows() { return kRows; }
int resident_groups(const ResidentWeight* w) { return w->groups; }

template <typename F>
static int run(const ResidentWeight* w, half* Y, const half* X, const half* bias, bool bias_given, int T, int gelu, int* err, cudaStream_t st) {
    CUtensorMap tm, tmy;
    if (!make_tmap_panels_f16(&tm, X, (uint64_t)T, (uint64_t)w->K, (uint64_t)w->K, kSlab, F::kPanels) ||
        !make_tmap_2d_f16(&tmy, Y, (uint64_t)T, (uint64_t)w->N, (uint64_t)w->N, 32, 32, 64))
        return fail(ET_ERR_CUDA, "resident linear: cuTensorMapEncodeTiled failed");
    static PerDeviceOnce once;
    using KernelFn = void (*)(CUtensorMap, CUtensorMap, ResidentParams);
    static const KernelFn kernels[2][2] = {{resident_kernel<F, false, false>, resident_kernel<F, false, true>},
                                           {resident_kernel<F, true, false>, resident_kernel<F, true, true>}};
    const cudaError_t attr_err = once.run([] {
        cudaError_t e = cudaSuccess;
        for (int i = 0; i < 4 && e == cudaSuccess; ++i)
            e = cudaFuncSetAttribute(kernels[i >> 1][i & 1], cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax);
        return e;
    });
    if (attr_err != cudaSuccess) return cuda_status(attr_err, "resident linear: shared memory opt-in");
    ResidentParams p;
    p.dir = w->d_dir; p.stream = w->d_stream; p.bias = bias; p.bias_given = bias_given; p.empty = w->d_empty;
    p.T = T; p.N = w->N; p.K = w->K; p.groups = w->groups;
    p.slabs = (T + kSlab - 1) / kSlab;
    launch_clocks(p.slabs, w->groups, w->K, w->group_clocks, &p.ranges);
    p.items = p.slabs * p.ranges;
    p.nx = w->nx; p.block_bytes = w->block_bytes; p.err = err;
    const int chunks = (w->K / 16 + F::kChunkSlices - 1) / F::kChunkSlices;
    const size_t smem = (size_t)(std::max(0, chunks - F::kTmemChunks) + w->nx) * F::kChunkBytes + (size_t)F::kSets * kSlots * w->block_bytes + F::kEpiWarps * kUnitBytes + sizeof(ResidentShared<F>) + 1024;
    return cuda_status(launch_pdl(kernels[gelu ? 1 : 0][w->d_empty ? 1 : 0], dim3((unsigned)std::min(p.items, sm_count())),
                                  dim3(F::kThreads), smem, st, tm, tmy, p),
                       "resident linear launch");
}

int resident_run(const ResidentWeight* w, half* Y, const half* X, const half* bias, bool bias_given, int T, int gelu, int* err, cudaStream_t st) {
    return w->wide ? run<Wide>(w, Y, X, bias, bias_given, T, gelu, err, st) : run<Narrow>(w, Y, X, bias, bias_given, T, gelu, err, st);
}

}  // namespace et
