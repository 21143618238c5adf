// On-the-fly attention on the 5th-generation tensor cores (tcgen05 + TMEM + TMA) for heads of 64, dense or with compact,
// column-pruned operands: the path behind et_attention_otf / et_attention_batch / et_attention_prune and the encoder layers (the
// mma.sync kernel in attention.cu covers the remaining variants).
// Replaces kernels/attention.cu:51-134 and :149-271 of the reference for those cases.
//
// A work item is 128 queries of one head of one sequence; a block is 128 keys of it:
//   S = Q K^T        SS UMMAs 128x128x16 (x4), Q and K_j in shared memory (TMA, 128-byte swizzle), fp32 in 128 TMEM columns
//   softmax          four warps, one thread per query row. The scores stay in tensor memory: a first pass over them takes the
//                    maximum (and adds the mask), 64 columns at a time, a second one the exponentials, 32 columns at a time with
//                    the next 32 on their way; with the last ones read, Q K^T of the NEXT block (of the next item, at the end
//                    of one) may overwrite them. Reference point and sum in fp32 (log2 domain); if the
//                    maximum has grown by more than 2^8 the reference point moves and O is rescaled in place.
//                    P = 2^(s - reference) as packed fp16 in 64 TMEM columns of its own.
//   O += P V         TS UMMAs 128x64x16 (x8): A = P from tensor memory, B = V_j as loaded (rows = keys, MN-major)
//   epilogue         O / row sum -> fp16 -> global, rows beyond the sequence are not written
// Blocks that hold at most 64 keys take half of everything.
//
// What bounds it: the softmax warps, at two per scheduler. The special-function unit delivers 16 results per clock and SM
// whatever the format (measured: ex2.f32 16.0, ex2.f16x2 8.0 pairs), so a 128 x 128 block costs it 1024 clocks, against 512
// clocks of UMMAs and ~450 issue slots per warp; kPolyPairs of every 16 pairs of exponentials are evaluated on the FMA pipe
// (Cody-Waite reduction and a cubic). 64 x 512 tokens, 12 heads, with 0, 2, 4, 6, 8 pairs: 84.1, 81.2, 81.2, 84.0, 85.8 us, and 2.880, 2.884,
// 2.889, 2.895, 2.900e-4 away from 64 bits: two, the more exact of the two that are equally fast. Loads, maximum, exponentials and stores
// alone, two warps to a scheduler, take 1240 clocks a block; with everything else it is ~1640.
// Two CTAs share an SM (256 TMEM columns and ~100 KB of shared memory each), so that one's loads, maxima and hand-overs run
// under the other's exponentials.
// Both passes are loops over few columns: 110 registers, where a row's 128 scores unrolled in registers took 216, handed over by the other
// warps, and with a mask spilled 120 bytes (20 here). Held so 64 x 512 tokens took 83.4 us, 64 x 200 28.4 (26.2 here), 64 ragged sequences 58.9
// (54.8), 1 x 384 with a mask 9.6 (9.1), 64 x 384 with one 78.6 (69.4), 1 x 701 with one (16 heads, rows anywhere) 21.2 (17.4). Slower as well
// (64 x 512): two threads per row and sixteen softmax warps 83.5, the next block's scores fetched under the last exponentials 85.6, the second
// pass unrolled 82.4, half blocks of 64 keys 100 (and 1.035 times the error), exponentials ahead of the maximum 101.
// CTAs are persistent: the grid has one CTA per item, and a running CTA takes over the next one that has not started (cluster
// launch control), so that ragged batches balance themselves and an item's loads and first Q K^T are under way while the
// previous one is finished; its rows are written inside the next item's first block. Ragged batches that outlast a wave are taken
// longest first (sort_sequences).
// An additive mask is added to the scores as score + 8 x mask, one mixed-precision multiply-add per element (8 is 1 / scale), in the
// first pass, which writes them back. It comes by TMA where the rows allow it, otherwise two warps copy granules; with an SM per
// item two blocks' masks are held.
// Column-pruned operands come in two forms. kScatterV (the operator): V is compact, a head's columns start anywhere, results go
// to their original columns with zeros between. kCompact (the encoder layers, which lay their weights out for it): every head's
// columns of Q, K and V start at a multiple of 16 and are padded to one with zeros, so that Q K^T takes width / 16 steps, P V
// a UMMA of the width, and the result is stored compact; the next linear has its input features gathered accordingly.
//
// Every mbarrier wait is bounded; a wait that gives up sets the error word and the CTA leaves through the common exit.
#include <mutex>
#include "attention.h"
#include "common.h"
#include "ptx.cuh"
#include "tmap.h"
#include "vec_math.cuh"

namespace et {

namespace {

constexpr int kBQ = 128, kBK = 128, kHD = 64;
constexpr int kTile = kBQ * kHD * 2;      // 16 KB: a Q tile, a key block of K or of V
constexpr int kSoftmaxWarps = 4;          // one thread per query row
constexpr int kMaskWarps = 2;             // copy masks that do not come by TMA
constexpr int kThreads = 256;             // + a warp that requests the loads and hands out items, one that issues UMMAs, kMaskWarps
constexpr int kCtasPerSm = 2;
constexpr int kTmemCols = 256;            // S 128 | P 64 | O 64
constexpr uint32_t kSCol = 0, kPCol = 128, kOCol = 192;
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kRescaleStep = 8.f;       // log2 units by which a row maximum must grow before O is rescaled
constexpr int kItemRing = 4;
constexpr int kMaxSorted = 256;           // sequences of a ragged batch that a CTA keeps in order of length
constexpr int kLenClasses = 9;            // 8 or more key blocks, 7, ..., none
constexpr int kMaskPitch = 272;           // bytes: seventeen 16-byte granules hold 128 mask values at any alignment; conflict-free
constexpr int kMaskBytes = kSoftmaxWarps * 32 * kMaskPitch;
constexpr int kScatterPitch = 136;        // bytes per staged output row (64 halfs + 8 bytes against bank conflicts)
constexpr int kScatterBytes = kBQ * kScatterPitch;
constexpr int kPolyPairs = 2;             // of 16 pairs of exponentials, how many go to the FMA pipe

struct TcParams {
    half* Z;
    const half* mask;
    const int* cu_seqlens;
    const int* valid_lens;
    const int* qk_head_ptr;
    const int* v_head_ptr;
    const int* v_col_id;
    int z_pitch, mask_ld, batch, uniform_len, nhead;
    float scale_log2;
    bool take_over;   // CTAs ask for items that have not started
    bool mask_two;    // two places for masks: where a CTA has an SM to itself
    bool mask_rows;   // equal lengths, and every row of the mask starts on a 16-byte boundary behind the one before: it comes by TMA
    int* err;
};

// A work item as the loading warp hands it to the others.
struct Item {
    int tok0, q0, len, valid, head;
    int nkb;               // key blocks; < 0: no more items
    int v_x, v_off, v_n, v_base;   // pruned V: first column of the copied box, of the head's window in it, width, index of its first column id
    int qk_x, qk_steps;    // first column of the Q and K boxes, 16-wide steps of Q K^T
    int v_add;             // second part of a wide window: only its own columns are written
};

enum Form { kDense = 0, kScatterV = 1, kCompact = 2 };

template <bool kMask, int kForm>
struct Cfg {
    static constexpr bool kPruneV = kForm == kScatterV;
    // The operator with compact V replaced a kernel that takes every exponential on the special-function unit, relative to the
    // row's true maximum (the largest P is then 1, but for the fp32 rounding of that maximum); it keeps that, as its results would be
    // further from exact ones otherwise (up to 1.12 times with a mask and 1000 tokens). The other forms replaced packed fp16 exponentials, three times as far off.
    static constexpr int kPolyPairs = kPruneV ? 0 : et::kPolyPairs;
    static constexpr float kRescaleStep = kPruneV ? 0.f : et::kRescaleStep;
    static constexpr int kQS = (kMask || kPruneV) ? 1 : 2;
    static constexpr int kKS = 2;
    static constexpr int kVS = (kMask || kPruneV) ? 1 : 2;
    static constexpr int kMaskAt = (kQS + kKS + kVS) * kTile;
    static constexpr int kScatterAt = kMaskAt + (kMask ? kMaskBytes : 0);
    static constexpr int kBytes = kScatterAt + (kPruneV ? kScatterBytes : 0);
    template <bool kSorted>
    __host__ __device__ static constexpr int second_mask_at();   // what a second mask takes begins there
};

struct TcShared {
    uint4 clc;                            // answer of the cluster launch control
    uint64_t clc_full;
    uint64_t q_full[2], q_empty[2], k_full[2], k_empty[2], v_full[2], v_empty[2];
    uint64_t s_full, s_free, p_full, pv_done;
    uint64_t m_full[2], m_empty[2];       // kMask: blocks' masks
    uint64_t item_full[kItemRing], item_empty[kItemRing];
    Item item[kItemRing];
    uint32_t tmem_base;
};
// A ragged batch in order of length: the sequences, and how many query blocks lie before each.
struct SeqTable {
    int tok0[kMaxSorted], len[kMaxSorted], valid[kMaxSorted], before[kMaxSorted + 1];
    int class_at[kLenClasses + 1];
    int given_tok0[kMaxSorted], given_len[kMaxSorted], given_valid[kMaxSorted];   // in the caller's order
};

template <bool kMask, int kForm>
template <bool kSorted>
__host__ __device__ constexpr int Cfg<kMask, kForm>::second_mask_at() {
    return (kBytes + (int)sizeof(TcShared) + (kSorted ? (int)sizeof(SeqTable) : 0) + 1023) / 1024 * 1024;
}

__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const float (&v)[32]) {
    const uint32_t(&r)[32] = reinterpret_cast<const uint32_t(&)[32]>(v);
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,"
        "%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
        "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]),
        "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
// -infinity in columns [from, to) of a warp's lanes (whole warp).
__device__ __forceinline__ void tmem_fill_neg_inf(uint32_t taddr, int from, int to) {
    const uint32_t v = 0xff800000u;
    for (; to - from >= 16; from += 16)
        asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1};" ::"r"(taddr + from), "r"(v) : "memory");
    if ((to - from) & 8) {
        asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1};" ::"r"(taddr + from), "r"(v) : "memory");
        from += 8;
    }
    if ((to - from) & 4) {
        asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%1,%1,%1};" ::"r"(taddr + from), "r"(v) : "memory");
        from += 4;
    }
    if ((to - from) & 2) {
        asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1,%1};" ::"r"(taddr + from), "r"(v) : "memory");
        from += 2;
    }
    if ((to - from) & 1) asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};" ::"r"(taddr + from), "r"(v) : "memory");
    tmem_st_wait();
}
__device__ __forceinline__ uint32_t pack2(float a, float b) {
    half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
}
// 2^x for two values on the FMA and ALU pipes, x <= 127: x = n + f with n the nearest whole number (adding 1.5 * 2^23 leaves
// n in the low bits of the sum) and |f| <= 1/2; 2^f by the cubic that interpolates it at the Chebyshev nodes of [-1/2, 1/2]
// (largest relative error 1.0e-4, below half a unit of the fp16 that the result is rounded to); n goes into the exponent.
// Not a number stays so: the maximum keeps it, and as the arithmetic on the exponent would make a number of it, x * 0 is added.
__device__ __forceinline__ float2 ex2_poly2(float2 x) {
    x.x = max_nan(x.x, -126.f);
    x.y = max_nan(x.y, -126.f);
    const float2 big = make_float2(12582912.f, 12582912.f), nbig = make_float2(-12582912.f, -12582912.f);
    const float2 t = add2(x, big);
    const float2 n = add2(t, nbig);
    const float2 f = add2(x, make_float2(-n.x, -n.y));
    float2 r = fma2(f, make_float2(0.0558382832f, 0.0558382832f), make_float2(0.242639482f, 0.242639482f));
    r = fma2(r, f, make_float2(0.693136752f, 0.693136752f));
    r = fma2(r, f, make_float2(0.999924541f, 0.999924541f));
    float2 y;
    y.x = __int_as_float(__float_as_int(r.x) + (__float_as_int(t.x) << 23));
    y.y = __int_as_float(__float_as_int(r.y) + (__float_as_int(t.y) << 23));
    return fma2(x, make_float2(0.f, 0.f), y);
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src, int bytes) {   // bytes < 16: the rest is zero-filled
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes) : "memory");
}

// Asks for a CTA of the grid that has not started; the answer (16 bytes) completes `bar`. Documented as undefined after an
// answer that there is none: the caller stops there.
__device__ __forceinline__ void clc_try_cancel(uint4* answer, uint64_t* bar) {
    asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(
                     smem_u32(answer)),
                 "r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ bool clc_query(const uint4* answer, int& x) {
    uint32_t ok, cx;
    asm volatile(
        "{\n.reg .b128 h;\n.reg .pred p;\nld.shared.b128 h, [%2];\n"
        "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, h;\nselp.u32 %0, 1, 0, p;\nmov.u32 %1, 0;\n"
        "@p clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %1, h;\n}"
        : "=r"(ok), "=r"(cx)
        : "r"(smem_u32(answer))
        : "memory");
    x = (int)cx;
    return ok != 0;
}

// Sorts a ragged batch by key blocks, the longest first (whole warp; sequences of one class keep their order): what is left when CTAs
// run out of items are then short ones, and an item is found without reading memory. In the caller's order, with two rounds of loads per
// item, the CTAs of 64 sequences of 32..512 tokens, 12 heads, finished between 43 and 52.5 us, and 256 x 128 tokens waited for items:
// 51.7 -> 49.4 and 64 -> 46 us with operands in L2 (55.7 -> 53.9 from memory). It takes ~1 us before the first item, so only batches that outlast one wave of CTAs are sorted (16 x 128
// tokens would take 7.7 us instead of 6.1).
__device__ __forceinline__ void sort_sequences(const TcParams& p, SeqTable* t, int lane) {
    if (lane <= kLenClasses) t->class_at[lane] = 0;
    __syncwarp();
    const unsigned below = (1u << lane) - 1u;
    for (int pass = 0; pass < 2; ++pass) {   // count, place
        for (int base = 0; base < p.batch; base += 32) {
            const int i = base + lane;
            const bool in = i < p.batch;
            int tok0 = 0, len = 0, valid = 0;
            if (in && pass == 0) {
                tok0 = p.cu_seqlens[i];
                len = p.cu_seqlens[i + 1] - tok0;
                valid = p.valid_lens ? max(0, min(p.valid_lens[i], len)) : len;
                t->given_tok0[i] = tok0;
                t->given_len[i] = len;
                t->given_valid[i] = valid;
            } else if (in) {
                tok0 = t->given_tok0[i];
                len = t->given_len[i];
                valid = t->given_valid[i];
            }
            const int c = in ? 8 - min((valid + kBK - 1) / kBK, 8) : kLenClasses;
            const unsigned same = __match_any_sync(0xffffffffu, c);
            const int at = t->class_at[c];
            __syncwarp();
            if ((same & below) == 0) t->class_at[c] = at + __popc(same);
            __syncwarp();
            if (pass == 1 && in) {
                const int pos = at + __popc(same & below);
                t->tok0[pos] = tok0;
                t->len[pos] = len;
                t->valid[pos] = valid;
            }
        }
        if (pass == 0) {   // counts -> where each class starts
            const int n = lane < kLenClasses ? t->class_at[lane] : 0;
            int incl = n;
#pragma unroll
            for (int o = 1; o < 16; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += v;
            }
            if (lane < kLenClasses) t->class_at[lane] = incl - n;
            __syncwarp();
        }
    }
    __syncwarp();
    int before = 0;
    for (int base = 0; base < p.batch; base += 32) {
        const int i = base + lane;
        int incl = i < p.batch ? (t->len[i] + kBQ - 1) / kBQ : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        if (i < p.batch) t->before[i + 1] = before + incl;
        before += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) t->before[0] = 0;
    __syncwarp();
}

// Which queries block `blk` of head `h` is (whole warp). nkb = -1: the block lies beyond the batch (the grid of a ragged batch has
// slack). A ragged batch that is not sorted is searched in memory: 32 sequences per round, each lane takes one, a prefix sum of their
// query-block counts locates the block.
template <bool kSorted>
__device__ __forceinline__ Item find_item(const TcParams& p, const SeqTable* t, int blk, int h, int lane) {
    Item it;
    it.tok0 = it.q0 = it.len = it.valid = 0;
    it.head = h;
    it.qk_x = h * kHD; it.qk_steps = kHD / 16;
    it.v_x = h * kHD; it.v_off = 0; it.v_n = kHD; it.v_base = 0; it.v_add = 0;
    int b = -1;
    if constexpr (kSorted) {
        for (int base = 0; base < p.batch; base += 32) {
            const unsigned hit = __ballot_sync(0xffffffffu, base + lane < p.batch && blk < t->before[min(base + lane, kMaxSorted - 1) + 1]);
            if (!hit) continue;
            b = base + __ffs(hit) - 1;
            it.tok0 = t->tok0[b];
            it.len = t->len[b];
            it.valid = t->valid[b];
            it.q0 = (blk - t->before[b]) * kBQ;
            break;
        }
    } else if (p.cu_seqlens) {
        for (int base = 0; base < p.batch && b < 0; base += 32) {
            const int i = base + lane;
            const int t0 = i < p.batch ? p.cu_seqlens[i] : 0;
            const int Li = i < p.batch ? p.cu_seqlens[i + 1] - t0 : 0;
            const int nbi = (Li + kBQ - 1) / kBQ;
            int incl = nbi;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += v;
            }
            const unsigned hit = __ballot_sync(0xffffffffu, blk < incl);
            if (hit) {
                const int src = __ffs(hit) - 1;
                const int excl = __shfl_sync(0xffffffffu, incl - nbi, src);
                b = base + src;
                it.tok0 = __shfl_sync(0xffffffffu, t0, src);
                it.len = __shfl_sync(0xffffffffu, Li, src);
                it.q0 = (blk - excl) * kBQ;
            } else {
                blk -= __shfl_sync(0xffffffffu, incl, 31);
            }
        }
    } else {
        const int nb = (p.uniform_len + kBQ - 1) / kBQ;
        if (blk < nb * p.batch) { b = blk / nb; it.tok0 = b * p.uniform_len; it.q0 = (blk % nb) * kBQ; it.len = p.uniform_len; }
    }
    it.nkb = -1;
    if (b >= 0) {
        if (!kSorted) it.valid = p.valid_lens ? min(p.valid_lens[b], it.len) : it.len;
        it.nkb = it.valid > 0 ? (it.valid + kBK - 1) / kBK : 0;
    }
    return it;
}

// kSorted: a ragged batch of at most kMaxSorted sequences, taken longest first.
template <bool kMask, int kForm, bool kSorted>
__global__ void __launch_bounds__(kThreads, kCtasPerSm) attention_tc_kernel(const __grid_constant__ CUtensorMap tmQ,
                                                                            const __grid_constant__ CUtensorMap tmK,
                                                                            const __grid_constant__ CUtensorMap tmV,
                                                                            const __grid_constant__ CUtensorMap tmM,
                                                                            const __grid_constant__ TcParams p) {
    using C = Cfg<kMask, kForm>;
    constexpr bool kPruneV = kForm == kScatterV;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* const sQ = smem;
    uint8_t* const sK = sQ + C::kQS * kTile;
    uint8_t* const sV = sK + C::kKS * kTile;
    TcShared* const sh = reinterpret_cast<TcShared*>(smem + C::kBytes);
    SeqTable* const table = reinterpret_cast<SeqTable*>(sh + 1);   // kSorted
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    pdl_launch_dependents();
    // The place of block g's mask, and how often it has been used before. The second place lies behind everything else.
    auto mask_place = [&](uint32_t g) {
        return smem + (p.mask_two && (g & 1u) ? C::template second_mask_at<kSorted>() : C::kMaskAt);
    };
    auto mask_slot = [&](uint32_t g) { return p.mask_two ? g & 1u : 0u; };
    auto mask_turn = [&](uint32_t g) { return p.mask_two ? g >> 1 : g; };

    if (warp == kSoftmaxWarps) {
        if (lane == 0) {
            mbar_init(&sh->clc_full, 1);
            for (int i = 0; i < 2; ++i) {
                mbar_init(&sh->q_full[i], 1); mbar_init(&sh->q_empty[i], 1);
                mbar_init(&sh->k_full[i], 1); mbar_init(&sh->k_empty[i], 1);
                mbar_init(&sh->v_full[i], 1); mbar_init(&sh->v_empty[i], 1);
            }
            mbar_init(&sh->s_full, 1);
            mbar_init(&sh->s_free, kSoftmaxWarps);
            mbar_init(&sh->p_full, kSoftmaxWarps);
            mbar_init(&sh->pv_done, 1);
            if constexpr (kMask) {
                for (int i = 0; i < 2; ++i) {
                    mbar_init(&sh->m_full[i], p.mask_rows ? 1 : 32 * kMaskWarps);
                    mbar_init(&sh->m_empty[i], kSoftmaxWarps);
                }
                if (p.mask_rows) prefetch_tmap(&tmM);
            }
            for (int i = 0; i < kItemRing; ++i) {
                mbar_init(&sh->item_full[i], 1);
                mbar_init(&sh->item_empty[i], kSoftmaxWarps + 1 + (kMask && !p.mask_rows ? kMaskWarps : 0));
            }
            fence_mbar_init();
            prefetch_tmap(&tmQ);
            prefetch_tmap(&tmK);
            prefetch_tmap(&tmV);
        }
    } else if (warp == kSoftmaxWarps + 1) {
        tmem_alloc(&sh->tmem_base, kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh->tmem_base;
    if (warp == kSoftmaxWarps) {
        // ---- items and loads (all lanes stay together; lane 0 issues)
        pdl_wait();   // lengths and activations come from the preceding kernels
        if constexpr (kSorted) sort_sequences(p, table, lane);
        int id = blockIdx.x;   // heads fastest: what a ragged batch has too many lies at the end of the grid
        int ni = 0, nq = 0, nk = 0, nv = 0;   // items handed out, tiles requested
        uint32_t clc_phase = 0;
        bool ok = true;
        for (;;) {
            if (lane == 0 && p.take_over) {
                mbar_expect_tx(&sh->clc_full, 16);
                clc_try_cancel(&sh->clc, &sh->clc_full);
            }
            const int by = id % p.nhead;
            Item it = find_item<kSorted>(p, table, id / p.nhead, by, lane);
            if constexpr (kForm == kCompact) {
                if (p.qk_head_ptr) {
                    it.qk_x = p.qk_head_ptr[by];
                    it.qk_steps = (p.qk_head_ptr[by + 1] - it.qk_x) >> 4;
                }
                it.v_x = p.v_head_ptr[by];
                it.v_n = p.v_head_ptr[by + 1] - it.v_x;
            }
            int vx0 = 0, vw = 0;
            if constexpr (kPruneV) {
                vx0 = p.v_head_ptr[by];
                vw = p.v_head_ptr[by + 1] - vx0;
            }
            for (int part = 0; part < (kPruneV ? 2 : 1) && it.nkb >= 0 && ok; ++part) {
                if constexpr (kPruneV) {
                    // the head's compact columns start anywhere; the copied box of 64 starts at a multiple of 8. A window
                    // that does not fit one box is done in two passes (the second starts at a multiple of 8 and holds at most 7 columns).
                    const int c0 = part == 0 ? 0 : kHD - (vx0 & 7);   // columns of the window done by the first pass
                    if (part > 0 && c0 >= vw) break;
                    it.v_x = (vx0 + c0) & ~7;
                    it.v_off = (vx0 + c0) & 7;
                    it.v_n = min(vw - c0, kHD - it.v_off);
                    it.v_base = vx0 + c0;
                    it.v_add = part;
                }
                const int slot = ni % kItemRing;
                if (!(ok = mbar_wait(&sh->item_empty[slot], ((uint32_t)(ni / kItemRing) & 1u) ^ 1u))) break;
                if (lane == 0) {
                    sh->item[slot] = it;
                    mbar_arrive(&sh->item_full[slot]);
                }
                __syncwarp();
                ++ni;
                if (it.nkb == 0) continue;
                const int qs = nq % C::kQS;
                if (!(ok = mbar_wait(&sh->q_empty[qs], ((uint32_t)(nq / C::kQS) & 1u) ^ 1u))) break;
                if (lane == 0) {
                    mbar_expect_tx(&sh->q_full[qs], kTile);
                    tma_load_2d(sQ + qs * kTile, &tmQ, it.qk_x, it.tok0 + it.q0, &sh->q_full[qs]);
                }
                ++nq;
                // K_0, then K_{j+1} ahead of V_j: the next Q K^T needs its block before this one's P V does. The mask of a block follows:
                // its place is free when the previous block's has been added.
                for (int j = -1; j < it.nkb && ok; ++j) {
                    if (j + 1 < it.nkb) {
                        const int ks = nk & 1;
                        if (!(ok = mbar_wait(&sh->k_empty[ks], ((uint32_t)(nk >> 1) & 1u) ^ 1u))) break;
                        if (lane == 0) {
                            mbar_expect_tx(&sh->k_full[ks], kTile);
                            tma_load_2d(sK + ks * kTile, &tmK, it.qk_x, it.tok0 + (j + 1) * kBK, &sh->k_full[ks]);
                        }
                        ++nk;
                    }
                    if (j >= 0) {
                        const int vs = nv % C::kVS;
                        if (!(ok = mbar_wait(&sh->v_empty[vs], ((uint32_t)(nv / C::kVS) & 1u) ^ 1u))) break;
                        if (lane == 0) {
                            mbar_expect_tx(&sh->v_full[vs], kTile);
                            tma_load_2d(sV + vs * kTile, &tmV, it.v_x, it.tok0 + j * kBK, &sh->v_full[vs]);
                        }
                        ++nv;
                    }
                    if (kMask && j + 1 < it.nkb && p.mask_rows) {   // block number nk - 1
                        const uint32_t g = (uint32_t)nk - 1u, ms = mask_slot(g);
                        if (!(ok = mbar_wait(&sh->m_empty[ms], (mask_turn(g) & 1u) ^ 1u))) break;
                        if (lane == 0) {
                            mbar_expect_tx(&sh->m_full[ms], 2 * kTile);
                            tma_load_2d(mask_place(g), &tmM, (j + 1) * kBK, it.q0, &sh->m_full[ms]);
                            tma_load_2d(mask_place(g) + kTile, &tmM, (j + 1) * kBK + 64, it.q0, &sh->m_full[ms]);
                        }
                    }
                }
            }
            if (!p.take_over) break;
            // the answer is awaited even on the way out: nothing may be in flight towards shared memory when the CTA leaves
            const bool answered = mbar_wait(&sh->clc_full, clc_phase);
            clc_phase ^= 1u;
            ok = ok && answered;
            if (!ok) break;
            const bool more = clc_query(&sh->clc, id);
            fence_proxy_async_smem();   // the answer has been read before the next one may be written
            __syncwarp();
            if (!more) break;
        }
        if (ok) {
            const int slot = ni % kItemRing;
            ok = mbar_wait(&sh->item_empty[slot], ((uint32_t)(ni / kItemRing) & 1u) ^ 1u);
            if (ok && lane == 0) {
                sh->item[slot].nkb = -1;
                mbar_arrive(&sh->item_full[slot]);
            }
        }
        if (!ok) {
            if (lane == 0) atomicExch(p.err, 21);
            // copies still in flight land before the CTA leaves (bounded)
            for (int i = max(nq - C::kQS, 0); i < nq; ++i) mbar_wait(&sh->q_full[i % C::kQS], (uint32_t)(i / C::kQS) & 1u);
            for (int i = max(nk - 2, 0); i < nk; ++i) mbar_wait(&sh->k_full[i & 1], (uint32_t)(i >> 1) & 1u);
            for (int i = max(nv - C::kVS, 0); i < nv; ++i) mbar_wait(&sh->v_full[i % C::kVS], (uint32_t)(i / C::kVS) & 1u);
            if (kMask && p.mask_rows)
                for (int g = max(nk - 2, 0); g < nk; ++g) mbar_wait(&sh->m_full[mask_slot(g)], mask_turn(g) & 1u);
        }
        __syncwarp();
    } else if (kMask && warp >= kSoftmaxWarps + 2) {
        // ---- masks that do not come by TMA: the seventeen granules that a row of a block touches, asynchronously
        if (!p.mask_rows) {
            pdl_wait();
            const int t = tid - 32 * (kSoftmaxWarps + 2);
            uint32_t g = 0;
            bool ok = true;
            for (int ni = 0;; ++ni) {
                const int slot = ni % kItemRing;
                ok = mbar_wait(&sh->item_full[slot], (uint32_t)(ni / kItemRing) & 1u);
                if (!ok) break;
                const int nkb = sh->item[slot].nkb, q0 = sh->item[slot].q0, len = sh->item[slot].len;
                __syncwarp();
                if (elect_one()) mbar_arrive(&sh->item_empty[slot]);
                __syncwarp();
                if (nkb < 0) break;
                const uint8_t* const mend = reinterpret_cast<const uint8_t*>(p.mask + (size_t)(len - 1) * p.mask_ld + len);
                for (int j = 0; j < nkb; ++j, ++g) {
                    ok = mbar_wait(&sh->m_empty[mask_slot(g)], (mask_turn(g) & 1u) ^ 1u);
                    if (!ok) break;
                    uint8_t* const place = mask_place(g);
                    const uint8_t* const m0 = reinterpret_cast<const uint8_t*>(p.mask + (size_t)q0 * p.mask_ld + j * kBK);
                    const int rows = min(kBQ, len - q0);   // (what is not copied belongs to rows that are not stored, or to keys beyond the length)
                    auto granule = [&](const uint8_t* row, int r, int c) {
                        const uint8_t* src = reinterpret_cast<const uint8_t*>(reinterpret_cast<uintptr_t>(row) & ~(uintptr_t)15) + c * 16;
                        const long left = (long)(mend - src);
                        if (left > 0) cp_async16(place + r * kMaskPitch + c * 16, src, left >= 16 ? 16 : (int)left);
                    };
                    // sixteen granules of a row by sixteen threads, then the seventeenth ones
                    const uint8_t* row = m0 + (size_t)(t >> 4) * p.mask_ld * 2;
#pragma unroll 4
                    for (int r = t >> 4; r < rows; r += kMaskWarps * 2, row += (size_t)p.mask_ld * (kMaskWarps * 4)) granule(row, r, t & 15);
                    for (int r = t; r < rows; r += 32 * kMaskWarps) granule(m0 + (size_t)r * p.mask_ld * 2, r, 16);
                    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&sh->m_full[mask_slot(g)])) : "memory");
                }
                if (!ok) break;
            }
            asm volatile("cp.async.wait_all;" ::: "memory");
            if (!ok && lane == 0) atomicExch(p.err, 23);
            __syncwarp();
        }
    } else if (warp == kSoftmaxWarps + 1) {
        // ---- UMMAs: the warp stays converged (every lane waits), one elected lane issues. Blocks are numbered through
        // across items: Q K^T of block g + 1 is issued as soon as the scores of block g have been read, ahead of P V of g.
        const uint32_t idesc_qk = make_idesc_f16(128, kBK), idesc_qk_half = make_idesc_f16(128, kBK / 2);
        uint32_t idesc_pv = make_idesc_f16(128, kHD, false, true);   // V is an MN-major B operand
        uint32_t idesc_pv_next = idesc_pv;   // of the item whose Q K^T is being issued
        int steps = kHD / 16;
        int ni = 0, nq = 0;
        uint32_t g = 0;
        bool ok = true, end = false;
        int nkb = 0, valid = 0;      // current item
        // takes the next item that has blocks (or the end); the items' slots go back at once: everything needed is kept here
        auto next_item = [&]() -> bool {
            for (;;) {
                const int slot = ni % kItemRing;
                if (!mbar_wait(&sh->item_full[slot], (uint32_t)(ni / kItemRing) & 1u)) return false;
                nkb = sh->item[slot].nkb;
                valid = sh->item[slot].valid;
                if constexpr (kForm == kCompact) {
                    steps = sh->item[slot].qk_steps;
                    idesc_pv_next = make_idesc_f16(128, sh->item[slot].v_n, false, true);
                }
                __syncwarp();
                if (elect_one()) mbar_arrive(&sh->item_empty[slot]);
                __syncwarp();
                ++ni;
                if (nkb < 0) { end = true; return true; }
                if (nkb > 0) return true;
            }
        };
        // S = Q K_j^T, block number gg; `last`: Q is not needed afterwards
        auto issue_qk = [&](uint32_t gg, int qs, bool half, bool last) {
            tc_fence_after();
            if (elect_one()) {
                const uint32_t qa = smem_u32(sQ + qs * kTile), ka = smem_u32(sK + (gg & 1) * kTile);
#pragma unroll
                for (int ks = 0; ks < 4; ++ks) {
                    if (kForm == kCompact && ks >= steps) break;
                    umma_f16(tmem + kSCol, make_smem_desc(qa + ks * 32, 16, 1024, 2), make_smem_desc(ka + ks * 32, 16, 1024, 2),
                             half ? idesc_qk_half : idesc_qk, ks > 0);
                }
                umma_commit(&sh->s_full);
                umma_commit(&sh->k_empty[gg & 1]);
                if (last) umma_commit(&sh->q_empty[qs]);
            }
            __syncwarp();
        };
        auto is_half = [&](int j) { return valid - j * kBK <= kBK / 2; };

        ok = next_item();
        if (ok && !end) {
            const int qs = nq % C::kQS;
            ok = mbar_wait(&sh->q_full[qs], (uint32_t)(nq / C::kQS) & 1u) && mbar_wait(&sh->k_full[0], 0);
            if (ok) issue_qk(0, qs, is_half(0), nkb == 1);
            ++nq;
        }
        int j = 0;
        while (ok && !end) {
            const bool half = is_half(j);
            const bool first = j == 0;
            if (first) idesc_pv = idesc_pv_next;
            bool issued = false;
            const uint32_t kb1 = (g + 1) & 1, kp1 = ((g + 1) >> 1) & 1;
            if (j + 1 < nkb) {
                ok = mbar_wait(&sh->s_free, g & 1) && mbar_wait(&sh->k_full[kb1], kp1);
                if (!ok) break;
                issue_qk(g + 1, (nq - 1) % C::kQS, is_half(j + 1), j + 2 == nkb);
                issued = true;
            } else if (mbar_poll_warp(&sh->item_full[ni % kItemRing], (uint32_t)(ni / kItemRing) & 1u) &&
                       sh->item[ni % kItemRing].nkb > 0) {
                // the next item's first block, if its operands are there already: P V of this block does not wait for them
                const int qs = nq % C::kQS;
                if (C::kQS > 1 && mbar_poll_warp(&sh->q_full[qs], (uint32_t)(nq / C::kQS) & 1u) && mbar_poll_warp(&sh->k_full[kb1], kp1)) {
                    ok = mbar_wait(&sh->s_free, g & 1) && next_item();
                    if (!ok) break;
                    issue_qk(g + 1, qs, is_half(0), nkb == 1);
                    ++nq;
                    j = -1;
                    issued = true;
                }
            }
            // O += P V of block g
            const int vs = g % C::kVS;
            ok = mbar_wait(&sh->p_full, g & 1) && mbar_wait(&sh->v_full[vs], (uint32_t)(g / C::kVS) & 1u);
            if (!ok) break;
            tc_fence_after();
            if (elect_one()) {
                const uint32_t va = smem_u32(sV + vs * kTile);
                const int steps = half ? kBK / 32 : kBK / 16;
                for (int ks = 0; ks < steps; ++ks)   // P of keys 16ks..16ks+15: 8 packed columns
                    umma_f16_ts(tmem + kOCol, tmem + kPCol + (uint32_t)(ks * 8), make_smem_desc(va + ks * 2048, 0, 1024, 2), idesc_pv,
                                (!first || ks > 0) ? 1u : 0u);
                umma_commit(&sh->pv_done);
                umma_commit(&sh->v_empty[vs]);
            }
            __syncwarp();
            if (!issued) {
                ok = next_item();
                if (!ok || end) break;
                const int qs = nq % C::kQS;
                ok = mbar_wait(&sh->q_full[qs], (uint32_t)(nq / C::kQS) & 1u) && mbar_wait(&sh->k_full[kb1], kp1) &&
                     mbar_wait(&sh->s_free, g & 1);
                if (!ok) break;
                issue_qk(g + 1, qs, is_half(0), nkb == 1);
                ++nq;
                j = -1;
            }
            ++j;
            ++g;
        }
        if (!ok && lane == 0) atomicExch(p.err, 21);
        __syncwarp();
    } else if (warp < kSoftmaxWarps) {
        // ---- softmax: one thread per query row (TMEM lane)
        pdl_wait();
        const int row = warp * 32 + lane;
        const uint32_t lane_base = (uint32_t)(warp * 32) << 16;
        const uint32_t s_addr = tmem + lane_base + kSCol, p_addr = tmem + lane_base + kPCol, o_addr = tmem + lane_base + kOCol;
        const bool wide = (p.z_pitch & 15) == 0 && (reinterpret_cast<uintptr_t>(p.Z) & 31) == 0;
        uint32_t g = 0;
        bool ok = true;
        int done_slot = -1;     // item whose P V is on its way and whose rows are still to be written
        float done_sum = 0.f;   // its row sum
        // Output columns of the window's features `lane` and `lane` + 32, of this item and of the one still to be written: read
        // when the item is taken up (one by one in the epilogue they cost more than everything else of a short item).
        int cols[2] = {0, 0}, done_cols[2] = {0, 0};
        auto release = [&](int slot) {
            __syncwarp();
            if (elect_one()) mbar_arrive(&sh->item_empty[slot]);
            __syncwarp();
        };
        // O / row sum -> fp16 -> global. Called when the item's last P V has completed: inside the
        // next item's first block, whose scores and exponentials cover the wait.
        auto finish = [&]() {
            const Item& it = sh->item[done_slot];
            const float inv = done_sum > 0.f ? 1.f / done_sum : 0.f;
            const int qr = it.q0 + row;
            const bool in = qr < it.len;
            half* const zrow = p.Z + (size_t)(it.tok0 + qr) * p.z_pitch + (kForm == kCompact ? it.v_x : it.head * kHD);
            if constexpr (kPruneV) {
                // a row is put together in shared memory (zeros where V was pruned) and written whole
                half* const st = reinterpret_cast<half*>(smem + C::kScatterAt + row * kScatterPitch);
                if (!it.v_add) {
#pragma unroll
                    for (int i = 0; i < 16; ++i) reinterpret_cast<uint2*>(st)[i] = make_uint2(0u, 0u);
                }
#pragma unroll 1
                for (int c = 0; c < 4; ++c) {
                    uint32_t r[16];
                    tmem_ld16(o_addr + c * 16, r);
                    tmem_ld_wait(r);
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const int k = c * 16 + i - it.v_off;
                        if (k >= 0 && k < it.v_n) {   // the same for the whole warp
                            const int col = __shfl_sync(0xffffffffu, k < 32 ? done_cols[0] : done_cols[1], k & 31) - it.head * kHD;
                            const half z = __float2half_rn(__uint_as_float(r[i]) * inv);
                            if (!it.v_add) st[col] = z;
                            else if (in) zrow[col] = z;
                        }
                    }
                }
                if (!it.v_add && in) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const uint2* s2 = reinterpret_cast<const uint2*>(st) + 2 * i;
                        *reinterpret_cast<uint4*>(zrow + i * 8) = make_uint4(s2[0].x, s2[0].y, s2[1].x, s2[1].y);
                    }
                }
            } else {
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    if (kForm == kCompact && 16 * c >= it.v_n) break;   // the same for the whole CTA
                    uint32_t r[16];
                    tmem_ld16(o_addr + c * 16, r);
                    tmem_ld_wait(r);
                    if (in) {
                        uint32_t ow[8];
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            ow[i] = pack2(__uint_as_float(r[2 * i]) * inv, __uint_as_float(r[2 * i + 1]) * inv);
                        half* const z = zrow + c * 16;
                        if (wide) {
                            asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(z), "r"(ow[0]), "r"(ow[1]), "r"(ow[2]),
                                         "r"(ow[3]), "r"(ow[4]), "r"(ow[5]), "r"(ow[6]), "r"(ow[7])
                                         : "memory");
                        } else {
                            *reinterpret_cast<uint4*>(z) = make_uint4(ow[0], ow[1], ow[2], ow[3]);
                            *reinterpret_cast<uint4*>(z + 8) = make_uint4(ow[4], ow[5], ow[6], ow[7]);
                        }
                    }
                }
            }
            release(done_slot);
            done_slot = -1;
        };
        for (int ni = 0; ok; ++ni) {
            const int slot = ni % kItemRing;
            ok = mbar_wait(&sh->item_full[slot], (uint32_t)(ni / kItemRing) & 1u);
            if (!ok) break;
            const Item& it = sh->item[slot];   // stays in shared memory
            const int nkb = it.nkb;
            if (nkb <= 0) {
                if (done_slot >= 0) {   // (the ring could run out of slots if an item waited behind empty ones)
                    ok = mbar_wait(&sh->pv_done, (g - 1) & 1);
                    if (!ok) break;
                    tc_fence_after();
                    finish();
                }
                if (nkb < 0) break;
                const int qr = it.q0 + row;   // no valid key: the output rows are zero
                if (qr < it.len) {
                    uint4* z = reinterpret_cast<uint4*>(p.Z + (size_t)(it.tok0 + qr) * p.z_pitch + (kForm == kCompact ? it.v_x : it.head * kHD));
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        if (kForm != kCompact || 8 * i < it.v_n) z[i] = make_uint4(0, 0, 0, 0);
                }
                release(slot);
                continue;
            }
            const int valid = it.valid;
            if constexpr (kPruneV) {
#pragma unroll
                for (int i = 0; i < 2; ++i) cols[i] = lane + 32 * i < it.v_n ? __ldg(p.v_col_id + it.v_base + lane + 32 * i) : 0;
            }
            float m_run = -INFINITY;
            float2 l2 = make_float2(0.f, 0.f);
            for (int j = 0; j < nkb; ++j, ++g) {
                const int left = valid - j * kBK;          // valid keys from here on
                const bool full = left > kBK / 2;          // otherwise half a block: two 32-column chunks instead of four
                ok = mbar_wait(&sh->s_full, g & 1);
                if (!ok) break;
                tc_fence_after();
                const float sc = p.scale_log2;
                const int chunks = full ? 4 : 2;
                if (!kMask && left < chunks * 32) tmem_fill_neg_inf(s_addr, left, chunks * 32);   // keys beyond the valid length
                if constexpr (kMask) {
                    ok = mbar_wait(&sh->m_full[mask_slot(g)], mask_turn(g) & 1u);
                    if (!ok) break;
                }
                // the maximum, half a block at a time; masked scores go back to where they came from
                float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll 1
                for (int c = 0; c < chunks; c += 2) {
                    float v[2][32];
                    tmem_ld32(s_addr + c * 32, reinterpret_cast<uint32_t(&)[32]>(v[0]));
                    tmem_ld32(s_addr + c * 32 + 32, reinterpret_cast<uint32_t(&)[32]>(v[1]));
                    tmem_ld_wait(v[0], v[1]);
                    if constexpr (kMask) {
                        // scale x score + mask = scale x (score + mask x 8): eight is 1 / scale, and the product with it exact
                        auto add_mask = [&](float& score, uint32_t two, bool high) {
                            asm("{\n.reg .b16 l, h, e;\nmov.b32 {l, h}, %1;\nmov.b16 e, 0x4800;\nfma.rn.f32.f16 %0, l, e, %0;\n}" : "+f"(score) : "r"(high ? two >> 16 : two));
                        };
                        if (p.mask_rows) {
                            const uint8_t* const mr = mask_place(g) + (c >> 1) * kTile + row * 128;
#pragma unroll
                            for (int e = 0; e < 8; ++e) {
                                const uint4 m4 = *reinterpret_cast<const uint4*>(mr + ((e ^ (row & 7)) << 4));
                                const uint32_t w[4] = {m4.x, m4.y, m4.z, m4.w};
#pragma unroll
                                for (int i = 0; i < 4; ++i) {
                                    add_mask(v[e >> 2][(e & 3) * 8 + 2 * i], w[i], false);
                                    add_mask(v[e >> 2][(e & 3) * 8 + 2 * i + 1], w[i], true);
                                }
                            }
                        } else {
                            const int q = min(it.q0 + row, it.len - 1);
                            const int shift = (int)((reinterpret_cast<uintptr_t>(p.mask + (size_t)q * p.mask_ld + j * kBK) & 15) >> 1);
                            const uint8_t* gr = mask_place(g) + row * kMaskPitch + c * 64;
                            uint4 cur = *reinterpret_cast<const uint4*>(gr);
#pragma unroll
                            for (int e = 0; e < 8; ++e) {
                                const uint4 nxt = *reinterpret_cast<const uint4*>(gr + (e + 1) * 16);
                                uint32_t w[8] = {cur.x, cur.y, cur.z, cur.w, nxt.x, nxt.y, nxt.z, nxt.w};
                                if (shift & 4)
#pragma unroll
                                    for (int i = 0; i < 6; ++i) w[i] = w[i + 2];
                                if (shift & 2)
#pragma unroll
                                    for (int i = 0; i < 5; ++i) w[i] = w[i + 1];
#pragma unroll
                                for (int i = 0; i < 4; ++i) {
                                    const uint32_t mv = (shift & 1) ? __funnelshift_r(w[i], w[i + 1], 16) : w[i];
                                    add_mask(v[e >> 2][(e & 3) * 8 + 2 * i], mv, false);
                                    add_mask(v[e >> 2][(e & 3) * 8 + 2 * i + 1], mv, true);
                                }
                                cur = nxt;
                            }
                        }
                        if (left < (c + 2) * 32) {   // keys beyond the valid length, whatever their mask is
#pragma unroll
                            for (int i = 0; i < 64; ++i)
                                if (c * 32 + i >= left) v[i >> 5][i & 31] = -INFINITY;
                        }
                        tmem_st32(s_addr + c * 32, v[0]);
                        tmem_st32(s_addr + c * 32 + 32, v[1]);
                    }
#pragma unroll
                    for (int i = 0; i < 32; ++i) mx[i & 3] = max3(mx[i & 3], v[i >> 4][2 * (i & 15)], v[i >> 4][2 * (i & 15) + 1]);
                }
                if constexpr (kMask) {
                    tmem_st_wait();
                    __syncwarp();
                    if (elect_one()) mbar_arrive(&sh->m_empty[mask_slot(g)]);
                    __syncwarp();
                }
                const float bmax = fmaxf(max3(mx[0], mx[1], mx[2]), mx[3]) * sc;   // the scale is positive: scale the maximum once
                // The reference point moves only when the row maximum has grown by more than 2^8 (P could leave the fp16
                // range; with each growth where kRescaleStep is 0); the final division by the row sum makes the result independent of it.
                const bool grow = bmax > m_run + C::kRescaleStep;   // also true for the first finite score of a row
                const bool any = __any_sync(0xffffffffu, grow);
                float alpha = 1.f;
                if (grow) {
                    alpha = m_run == -INFINITY ? 0.f : ex2_fast(m_run - bmax);
                    m_run = bmax;
                    l2.x *= alpha;
                    l2.y *= alpha;
                }
                const float nshift = (m_run == -INFINITY) ? 0.f : -m_run;
                const float2 sc2 = make_float2(sc, sc), sh2 = make_float2(nshift, nshift);
                // P and O may be written once P V of the previous block has completed
                if (g > 0) {
                    ok = mbar_wait(&sh->pv_done, (g - 1) & 1);
                    if (!ok) break;
                    tc_fence_after();
                }
                if (j == 0) {
                    if (done_slot >= 0) finish();
                } else if (any) {
#pragma unroll 1
                    for (int c = 0; c < 4; ++c) {
                        uint32_t o[16];
                        tmem_ld16(o_addr + c * 16, o);
                        tmem_ld_wait(o);
#pragma unroll
                        for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                        tmem_st16(o_addr + c * 16, o);
                    }
                }
                // exponentials of 32 scores, while the next 32 are fetched
                auto chunk = [&](const float (&v)[32], int c) {
                    uint32_t pk[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        float2 e = fma2(make_float2(v[2 * i], v[2 * i + 1]), sc2, sh2);
                        // spread over the chunk so that both pipes stay busy
                        if ((i * C::kPolyPairs) / 16 != ((i + 1) * C::kPolyPairs) / 16) {
                            e = ex2_poly2(e);
                        } else {
                            e.x = ex2_fast(e.x);
                            e.y = ex2_fast(e.y);
                        }
                        l2 = add2(l2, e);
                        pk[i] = pack2(e.x, e.y);
                    }
                    tmem_st16(p_addr + c * 16, pk);
                };
                {
                    float v[32], w[32];
                    tmem_ld32(s_addr, reinterpret_cast<uint32_t(&)[32]>(v));
                    tmem_ld_wait(v);
                    int c = 0;
#pragma unroll 1
                    for (;; c += 2) {
                        tmem_ld32(s_addr + c * 32 + 32, reinterpret_cast<uint32_t(&)[32]>(w));
                        chunk(v, c);
                        tmem_ld_wait(w);
                        if (c + 2 == chunks) break;
                        tmem_ld32(s_addr + c * 32 + 64, reinterpret_cast<uint32_t(&)[32]>(v));
                        chunk(w, c + 1);
                        tmem_ld_wait(v);
                    }
                    tc_fence_before();   // the next block's scores may be written
                    __syncwarp();
                    if (elect_one()) mbar_arrive(&sh->s_free);
                    __syncwarp();
                    chunk(w, c + 1);
                }
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (elect_one()) mbar_arrive(&sh->p_full);
                __syncwarp();
            }
            if (!ok) break;
            done_slot = slot;
            done_sum = l2.x + l2.y;
            if constexpr (kPruneV) {
                done_cols[0] = cols[0];
                done_cols[1] = cols[1];
            }
        }
        if (!ok && lane == 0) atomicExch(p.err, 22);
        __syncwarp();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == kSoftmaxWarps + 1) tmem_dealloc(tmem, kTmemCols);
}

bool g_scores_fp32 = false;   // kept for et_attention_scores_fp32: Q K^T accumulates in fp32 either way

// Error word of the kernel's bounded waits: a device variable of the library image (one copy per device that
// loads the library, zero at load), so that no launch ever allocates. The kernel writes it only when a wait
// gives up. In host code the symbol is a handle, not an address: the address is looked up once per device.
__device__ int g_attn_err_word;
constexpr int kMaxDevices = 64;
std::mutex g_err_mu;
int* g_err_ptr[kMaxDevices] = {nullptr};

int attn_err_address(int** out) {
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_status(e, "attention: cudaGetDevice");
    if (dev < 0 || dev >= kMaxDevices) return fail(ET_ERR_UNSUPPORTED, "attention: device ordinal above 63");
    std::lock_guard<std::mutex> lk(g_err_mu);
    if (!g_err_ptr[dev]) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_attn_err_word);
        if (e != cudaSuccess) return cuda_status(e, "attention: cudaGetSymbolAddress");
        g_err_ptr[dev] = static_cast<int*>(p);
    }
    *out = g_err_ptr[dev];
    return ET_OK;
}

template <bool kMask, int kForm, bool kSorted>
cudaError_t opt_in() {
    return cudaFuncSetAttribute(attention_tc_kernel<kMask, kForm, kSorted>, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448);
}
template <bool kMask, int kForm, bool kSorted = false>
cudaError_t launch(dim3 grid, cudaStream_t st, const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tm, const TcParams& p) {
    using C = Cfg<kMask, kForm>;
    const size_t smem = (p.mask_two ? (size_t)C::template second_mask_at<kSorted>() + kMaskBytes : C::kBytes + sizeof(TcShared) + (kSorted ? sizeof(SeqTable) : 0)) + 1024;
    return launch_pdl(attention_tc_kernel<kMask, kForm, kSorted>, grid, dim3(kThreads), smem, st, tq, tk, tv, tm, p);
}

}  // namespace

// Looks up the error word's address on the current device (encoder constructors call this so that the first
// launch, possibly inside a caller's stream capture, has nothing left to set up).
int attention_prepare_device() {
    int* p = nullptr;
    return attn_err_address(&p);
}

// Returns ET_ERR_UNSUPPORTED (without touching anything) when the case is outside the kernel's range, so the caller can use
// the general kernel instead.
//   v_head_ptr and v_col_id: V is compact ([tokens x v_cols]), results are scattered to their original columns.
//   v_head_ptr without v_col_id: V (and Q and K where qk_head_ptr is given) are compact, each head's columns start at a multiple
//   of 16 and number 16 to 64, a multiple of 16; the result is [tokens x v_cols] in V's layout.
int attention_tc_launch(half* Z, const half* Q, const half* K, const half* V, int q_pitch, int v_pitch, int qk_cols, int v_cols,
                        const int* qk_head_ptr, const int* v_head_ptr, const int* v_col_id, const half* mask, int mask_ld,
                        const int* cu_seqlens, const int* valid_lens, int batch, int uniform_len, int total_tokens, int max_len,
                        int d_model, int nhead, cudaStream_t st) {
    const bool compact = v_head_ptr && !v_col_id;
    if (qk_head_ptr && !compact) return ET_ERR_UNSUPPORTED;
    if (d_model / nhead != kHD || d_model % nhead) return ET_ERR_UNSUPPORTED;
    if (max_len <= 0) return ET_ERR_UNSUPPORTED;   // longest sequence unknown: the caller uses the general kernel
    // TMA: operands and pitches in whole 16-byte units; the mask's granules are read from a 16-byte aligned start
    if ((q_pitch & 7) || (v_pitch & 7) || (d_model & 7) || !aligned16(Q) || !aligned16(K) || !aligned16(V) || !aligned16(Z) ||
        (mask && !aligned16(mask)))
        return ET_ERR_UNSUPPORTED;
    if (batch <= 0 || total_tokens <= 0) return ET_OK;
    int* err_word = nullptr;
    {
        const int rc = attn_err_address(&err_word);
        if (rc) return rc;
    }
    CUtensorMap tq, tk, tv;
    const uint64_t rows = (uint64_t)total_tokens;
    // the column extent covers all heads of the operand; Q/K/V may be slices of one fused buffer
    if (!make_tmap_2d_f16(&tq, Q, rows, (uint64_t)qk_cols, (uint64_t)q_pitch, kBQ, kHD, 128) ||
        !make_tmap_2d_f16(&tk, K, rows, (uint64_t)qk_cols, (uint64_t)q_pitch, kBK, kHD, 128) ||
        !make_tmap_2d_f16(&tv, V, rows, (uint64_t)v_cols, (uint64_t)v_pitch, kBK, kHD, 128))
        return fail(ET_ERR_CUDA, "attention: cuTensorMapEncodeTiled failed");
    TcParams p;
    p.Z = Z; p.mask = mask; p.cu_seqlens = cu_seqlens; p.valid_lens = valid_lens;
    p.qk_head_ptr = qk_head_ptr; p.v_head_ptr = v_head_ptr; p.v_col_id = v_col_id;
    p.z_pitch = compact ? v_cols : d_model; p.mask_ld = mask_ld; p.batch = batch; p.uniform_len = uniform_len;
    p.scale_log2 = kLog2e / sqrtf((float)kHD);
    p.err = err_word;
    // (Of a ragged batch max_len may be more than the mask has rows: only the kernel knows how far it may read. Rows that overlap,
    // as those of a mask that depends on key - query alone may, are no matrix for a tensor map.)
    p.mask_rows = mask && !cu_seqlens && mask_ld % 8 == 0 && mask_ld >= uniform_len;
    CUtensorMap tm = tq;
    if (p.mask_rows && !make_tmap_2d_f16(&tm, mask, (uint64_t)uniform_len, (uint64_t)uniform_len, (uint64_t)mask_ld, kBQ, 64, 128))
        return fail(ET_ERR_CUDA, "attention: cuTensorMapEncodeTiled failed");
    static PerDeviceOnce once;
    const cudaError_t attr_err = once.run([] {
        cudaError_t e = opt_in<false, kDense, false>();
        if (e == cudaSuccess) e = opt_in<true, kDense, false>();
        if (e == cudaSuccess) e = opt_in<false, kDense, true>();
        if (e == cudaSuccess) e = opt_in<true, kDense, true>();
        if (e == cudaSuccess) e = opt_in<false, kScatterV, false>();
        if (e == cudaSuccess) e = opt_in<true, kScatterV, false>();
        if (e == cudaSuccess) e = opt_in<false, kCompact, false>();
        if (e == cudaSuccess) e = opt_in<true, kCompact, false>();
        if (e == cudaSuccess) e = opt_in<false, kCompact, true>();
        if (e == cudaSuccess) e = opt_in<true, kCompact, true>();
        return e;
    });
    if (attr_err != cudaSuccess) return cuda_status(attr_err, "attention: shared memory opt-in");
    const int nblk = cu_seqlens ? (total_tokens + kBQ - 1) / kBQ + batch : batch * ((uniform_len + kBQ - 1) / kBQ);
    const dim3 grid(nblk * nhead);
    p.nhead = nhead;
    // CTAs that all fit are left to the hardware: one that starts early would take an item for which a place is still free. (Of a
    // ragged batch only the tokens are known here: at least this many blocks. 4 x 512 tokens, 16 heads: 18.2 -> 11.3 us.)
    const long items = cu_seqlens ? (total_tokens + kBQ - 1) / kBQ : nblk;
    p.take_over = items * nhead > (long)kCtasPerSm * sm_count();
    p.mask_two = mask && items * nhead <= sm_count() && !cu_seqlens;
    // (The form that scatters V is never ragged: the operator takes one sequence.)
    const bool sorted = p.take_over && cu_seqlens && batch <= kMaxSorted;
    const auto run = compact      ? (sorted ? (mask ? launch<true, kCompact, true> : launch<false, kCompact, true>)
                                            : (mask ? launch<true, kCompact> : launch<false, kCompact>))
                     : v_head_ptr ? (mask ? launch<true, kScatterV> : launch<false, kScatterV>)
                     : sorted     ? (mask ? launch<true, kDense, true> : launch<false, kDense, true>)
                                  : (mask ? launch<true, kDense> : launch<false, kDense>);
    const cudaError_t e = run(grid, st, tq, tk, tv, tm, p);
    return cuda_status(e, "attention (tcgen05) launch");
}

void attention_tc_set_scores_fp32(int on) { g_scores_fp32 = on != 0; }
int attention_tc_scores_fp32() { return g_scores_fp32 ? 1 : 0; }

// Reads and clears the current device's error word of the tcgen05 attention kernel (synchronises).
// 0 = no wait gave up since the last read.
int attention_tc_error(int* code) {
    *code = 0;
    int* word = nullptr;
    int rc = attn_err_address(&word);
    if (rc) return rc;
    cudaError_t e = cudaMemcpy(code, word, sizeof(int), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return cuda_status(e, "attention error read");
    if (*code) {
        e = cudaMemset(word, 0, sizeof(int));
        if (e != cudaSuccess) return cuda_status(e, "attention error clear");
    }
    return ET_OK;
}

}  // namespace et
