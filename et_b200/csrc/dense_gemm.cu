// Dense linear  Y[T x N] = X[T x K] . W^T + bias  (optional tanh-GELU) on tcgen05: what a tile-pruned or row-pruned weight
// becomes when the multiplications with its zero tiles cost less than skipping them (the rule is in tile_gemm.cu).
// Replaces, for those weights, kernels/linear.cu:5-34 (row-pruned) and :54-167 (tile-pruned) of the reference.
//
// Two kernels. Both keep X and W in panels of 64 K elements, 128-byte-swizzled in shared memory (one TMA copy each), one or two
// panels to a stage, and accumulate in fp32 in tensor memory with both UMMA operands from shared memory. A stage costs the
// issuing warp ~400 clocks beside its UMMAs (a wait that finds its barrier complete, fences, commits), hence two panels where
// a panel's UMMAs are short; wide tiles take one, for more stages.
//
// dense_kernel, many tiles: persistent pairs of CTAs (cta_group::2, UMMAs 256 x BN x 16): each CTA of a pair copies its own 128
// tokens and half of the weight's rows, so that a 256 x 256 tile needs 32 KB per CTA and 512 clocks of UMMA time. What bounds a
// dense linear otherwise is the way from L2: with one CTA per 128 x 256 tile an SM asks for 94 bytes per clock and gets ~58
// (measured, all SMs busy). Four warps copy, one (of the pair's first CTA) issues, eight convert and store; two accumulators,
// so that a tile is stored while the next one is multiplied. 16384 x 4096 x 1024: tensor pipe 90 % busy.
//
// dense_split_kernel, few tiles (small batches): the K range is split over a thread-block cluster. Each CTA accumulates its
// share and finishes 1/cluster of the tile's columns: it sends the other CTAs the fp32 parts of theirs (asynchronous stores to
// distributed shared memory that count towards a barrier of the receiver), and when its own bytes have arrived adds them to its part, in rank order
// (no atomics: results do not depend on timing). With parts left in place and rows of the others' loaded 128 x 3072 -> 768 took 8.5 us (5.7 now),
// 4096 -> 1024 10.6 (6.3), 256 x 3072 -> 768 12.0 (7.0); with stores and a barrier of the cluster 6.3, 7.3 and 7.8. 128 x 768 -> 768 in the tile
// kernel 5.1 us, here 3.9.
// (A K share per pair of CTAs with tiles of 256 tokens: 1024 x 3072 -> 768 12.4 against 12.1 us, 2048 16.8 against 13.9.)
//
// The weight does not depend on the preceding kernel: its first copies are requested before griddepcontrol.wait. In both kernels the activations of the
// first stages are requested by warps that have nothing else to do yet, right behind that wait.
// Every mbarrier wait is bounded; a role that gives up records a code, and all threads reach the common exit (and the
// cluster barriers) whatever happened.
#include <algorithm>
#include "common.h"
#include "dense_gemm.h"
#include "epilogue.cuh"
#include "ptx.cuh"
#include "tmap.h"

namespace et {

namespace {

constexpr int kBM = 128;                  // tokens per CTA
constexpr int kBK = 64;                   // K elements per panel: one 128-byte-swizzled row
constexpr int kAPanel = kBM * kBK * 2;    // 16 KB
constexpr int kEpiWarps = 8;
constexpr int kUnitCols = 32;             // columns per epilogue store
constexpr int kUnitBytes = 32 * kUnitCols * 2;
constexpr int kMaxStages = 8;
// Copying warps take the stages in turn. A stage must always fall to the same warp: a parity wait is only safe for a waiter
// that has seen the barrier's previous phase, so the number of warps at work divides the number of stages (copy_warps).
constexpr int kCopyWarps = 4;
constexpr int kFirstEpi = kCopyWarps + 1;
constexpr int kThreads = 32 * (kFirstEpi + kEpiWarps);
constexpr int kSmemMax = 232448;
constexpr int kMaxBN = 256;

struct DenseParams {
    const half* bias;
    bool bias_given;        // the caller's, not the weight's own: the preceding kernel may still be writing it
    half* Y;
    int T, N, K, k_panels, tiles_n, tiles, bn, stages, panels;   // panels: per stage; the last stage of a K range may hold fewer
    int* err;
    const half* X;
    const half* W;
    const uint32_t* kept;   // kPruned: one bit per 16 x 16 tile, rows of whole words
};

__host__ __device__ constexpr int copy_warps(int stages) {
    return stages % 4 == 0 ? 4 : stages % 3 == 0 ? 3 : stages % 2 == 0 ? 2 : 1;
}
// The largest ring of at most n stages that several warps can share.
inline int ring_stages(int n) { return n >= 8 ? 8 : n == 7 ? 6 : n == 5 ? 4 : n; }

struct DenseShared {
    uint64_t full[kMaxStages], empty[kMaxStages];
    uint64_t acc_full[2], acc_empty[2];
    uint64_t received;   // split K: the other CTAs' parts of this CTA's columns
    uint32_t tmem_base;
    __align__(16) half bias[2][kMaxBN];
};

// Columns to allocate for `n` (a power of two, at least 32).
__device__ __forceinline__ uint32_t tmem_cols(int n) {
    uint32_t c = 32;
    while ((int)c < n) c <<= 1;
    return c;
}
__device__ __forceinline__ void epi_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(32 * kEpiWarps) : "memory"); }
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The address of the same shared-memory object in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t in_cta(const void* p, uint32_t rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
    return a;
}
// A copy into this CTA's shared memory that reports to a barrier of either CTA of the pair (cluster address).
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const void* tmap, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            smem_u32(dst)),
        "l"(tmap), "r"(x), "r"(y), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void umma_f16_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.u32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// Arrives on the barrier at this address in both CTAs of the pair once every UMMA issued so far has completed.
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
                 "h"((uint16_t)3)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}

// A pruned tile takes no part in the product, but 0 x infinity does here. Results that are not finite are therefore computed
// again from the kept tiles alone (one that really leaves the fp16 range comes out the same). Finding them costs one operation
// per two results (3072 -> 768 at 75 %, 128 tokens 8.86 -> 8.98 us, at 50 %, 4096 tokens 18.8 -> 19.3), in kernels of their own
// (kPruned) that weights without pruned tiles do not take.
struct NotFinite {   // zeros, until a value came that is not finite
    half2 s[4];
    __device__ __forceinline__ NotFinite() {
#pragma unroll
        for (int i = 0; i < 4; ++i) s[i] = __float2half2_rn(0.f);
    }
    __device__ __forceinline__ void note(const uint4& v) {
        const half2* h = reinterpret_cast<const half2*>(&v);
#pragma unroll
        for (int i = 0; i < 4; ++i) s[i] = __hfma2(h[i], __float2half2_rn(0.f), s[i]);
    }
    __device__ __forceinline__ bool any() const {
        const half2 t = __hadd2(__hadd2(s[0], s[1]), __hadd2(s[2], s[3]));
        return !(__low2float(t) + __high2float(t) == 0.f);
    }
};

// Those of the kCols results of `row` from column n0 on (all of one block-row) that are not finite, in place.
template <bool kGelu, int kCols = 8>
__device__ __forceinline__ void recompute_segment(const DenseParams& p, int row, int n0) {
    half* const y = p.Y + (size_t)row * p.N + n0;
    __align__(16) half h[kCols];
    bool odd = false;
#pragma unroll
    for (int c = 0; c < kCols; c += 4) {
        *reinterpret_cast<uint2*>(h + c) = __ldcg(reinterpret_cast<const uint2*>(y + c));
#pragma unroll
        for (int i = c; i < c + 4; ++i) odd = odd || (__half_as_ushort(h[i]) & 0x7c00u) == 0x7c00u;
    }
    if (!odd) return;
    const uint32_t* kept = p.kept + (size_t)(n0 / 16) * ((p.K / 16 + 31) / 32);
    float acc[kCols] = {};
    for (int t = 0; t < p.K / 16; ++t) {
        if (!((kept[t >> 5] >> (t & 31)) & 1u)) continue;
        const uint4* xs = reinterpret_cast<const uint4*>(p.X + (size_t)row * p.K + 16 * t);
        const uint4 x2[2] = {__ldcg(xs), __ldcg(xs + 1)};
        const half* x = reinterpret_cast<const half*>(x2);
#pragma unroll
        for (int c = 0; c < kCols; ++c) {
            const uint4* ws = reinterpret_cast<const uint4*>(p.W + (size_t)(n0 + c) * p.K + 16 * t);
            const uint4 w2[2] = {__ldg(ws), __ldg(ws + 1)};
            const half* w = reinterpret_cast<const half*>(w2);
#pragma unroll
            for (int k = 0; k < 16; ++k) acc[c] = fmaf(__half2float(x[k]), __half2float(w[k]), acc[c]);
        }
    }
#pragma unroll
    for (int c = 0; c < kCols; ++c) {
        if ((__half_as_ushort(h[c]) & 0x7c00u) != 0x7c00u) continue;
        const half v = __float2half_rn(acc[c] + __half2float(p.bias[n0 + c]));
        h[c] = kGelu ? __low2half(gelu_tanh_h2(__half2half2(v))) : v;
    }
#pragma unroll
    for (int c = 0; c < kCols; c += 4) *reinterpret_cast<uint2*>(y + c) = *reinterpret_cast<const uint2*>(h + c);
}

template <bool kGelu, bool kPruned>
__global__ void __launch_bounds__(kThreads, 1) dense_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW,
                                                            const __grid_constant__ CUtensorMap tmY, const __grid_constant__ DenseParams p) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int S = p.stages, bn = p.bn;
    const int b_panel = bn * kBK;   // bytes: half of the tile's features
    const int stage_bytes = p.panels * (kAPanel + b_panel);
    const int k_stages = (p.k_panels + p.panels - 1) / p.panels;
    uint8_t* const epi = smem + (size_t)S * stage_bytes;
    DenseShared* const sh = reinterpret_cast<DenseShared*>(epi + kEpiWarps * kUnitBytes);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = cluster_rank();
    const int pair = (int)blockIdx.x >> 1, G = (int)gridDim.x >> 1;
    const int my_tiles = (p.tiles - pair + G - 1) / G;
    if (tid == 0) {
        for (int i = 0; i < S; ++i) { mbar_init(&sh->full[i], 1); mbar_init(&sh->empty[i], 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(&sh->acc_full[i], 1); mbar_init(&sh->acc_empty[i], 2 * kEpiWarps); }
        fence_mbar_init();
        prefetch_tmap(&tmX);
        prefetch_tmap(&tmW);
    }
    if (warp == kCopyWarps) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh->tmem_base)), "r"(tmem_cols(2 * bn))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();   // the other CTA's barriers exist
    tc_fence_after();
    const uint32_t tmem = sh->tmem_base;

    // Of the first tile's first stages the weight's panels are requested before the wait for the preceding kernel, the activations behind it by
    // the epilogue's warps, which have nothing to do yet (one warp for both, behind its wait for an empty stage: 128 x 768 -> 2304 6.85
    // instead of 6.3 us, 1100 x 3072 -> 768 12.2 instead of 11.4, 32768 x 768 -> 2304 the same).
    const int ahead = min(S, k_stages);
    auto load_x = [&](int s, int kc, int tile) {
        const int np = min(p.panels, p.k_panels - kc * p.panels);
        const uint32_t bar = in_cta(&sh->full[s], 0);
        for (int i = 0; i < np; ++i)
            tma_load_2d_pair(smem + (size_t)s * stage_bytes + i * kAPanel, &tmX, (kc * p.panels + i) * kBK,
                             (tile / p.tiles_n) * (2 * kBM) + (int)rank * kBM, bar);
    };
    if (warp < kCopyWarps) {
        // ---- copies, stages in turn; both CTAs' report to the first one's barriers
        bool ok = true;
        const int cw = copy_warps(S);
        auto load_w = [&](int s, int kc, int tile) {
            const int np = min(p.panels, p.k_panels - kc * p.panels);
            const uint32_t bar = in_cta(&sh->full[s], 0);
            if (rank == 0) mbar_expect_tx(&sh->full[s], 2 * np * (kAPanel + b_panel));
            for (int i = 0; i < np; ++i)
                tma_load_2d_pair(smem + (size_t)s * stage_bytes + p.panels * kAPanel + i * b_panel, &tmW, (kc * p.panels + i) * kBK,
                                 (tile % p.tiles_n) * bn + (int)rank * (bn / 2), bar);
        };
        if (warp < cw && lane == 0)
            for (int i = warp; i < ahead; i += cw) load_w(i, i, pair);
        __syncwarp();
        pdl_wait();
        int tl = 0, kc = warp, s = warp;
        uint32_t ph = 1;
        for (int c = warp; warp < cw && c < my_tiles * k_stages; c += cw) {
            while (kc >= k_stages) { kc -= k_stages; ++tl; }
            if (s >= S) { s -= S; ph ^= 1u; }
            const int tile = pair + tl * G;
            if (c >= ahead) {
                ok = c < S || mbar_wait(&sh->empty[s], ph);
                if (!ok) break;
                if (lane == 0) { load_w(s, kc, tile); load_x(s, kc, tile); }
                __syncwarp();
            }
            kc += cw;
            s += cw;
        }
        // (On the normal way out every copy has been consumed: the accumulators of the last tile are complete. A wait that gives
        // up has lasted far longer than any copy.)
        if (!ok && lane == 0) atomicExch(p.err, 31);
    } else if (warp == kCopyWarps && rank == 0) {
        // ---- UMMAs of the pair
        const uint32_t idesc = make_idesc_f16(2 * kBM, bn);
        const uint64_t a0 = make_smem_desc(smem_u32(smem), 16, 1024, 2);
        const uint64_t b0 = make_smem_desc(smem_u32(smem) + p.panels * kAPanel, 16, 1024, 2);
        if (elect_one()) {   // one lane is the role
            const uint32_t full0 = smem_u32(&sh->full[0]);
            bool ok = true;
            int s = 0;
            uint32_t ph = 0;
            uint64_t a = a0, b = b0;
            const uint32_t step = (uint32_t)stage_bytes >> 4;   // descriptors count 16-byte units
            for (int tl = 0; tl < my_tiles && ok; ++tl) {
                const int buf = tl & 1;
                ok = mbar_wait(&sh->acc_empty[buf], ((uint32_t)(tl >> 1) & 1u) ^ 1u);
                if (!ok) break;
                tc_fence_after();
                const uint32_t d = tmem + buf * bn;
                uint32_t accumulate = 0;
                for (int left = p.k_panels; left > 0; left -= p.panels) {
                    if (!mbar_wait_at(full0 + s * 8, ph)) { ok = false; break; }
                    tc_fence_after();
                    const int np = min(p.panels, left);
                    for (int i = 0; i < np; ++i)
#pragma unroll
                        for (int ks = 0; ks < 4; ++ks) {
                            umma_f16_pair(d, a + (i * kAPanel >> 4) + ks * 2, b + (i * b_panel >> 4) + ks * 2, idesc, accumulate);
                            accumulate = 1;
                        }
                    umma_commit_pair(&sh->empty[s]);
                    a += step;
                    b += step;
                    if (++s == S) { s = 0; ph ^= 1u; a = a0; b = b0; }
                }
                if (ok) umma_commit_pair(&sh->acc_full[buf]);
            }
            if (!ok) atomicExch(p.err, 32);
        }
        __syncwarp();
    } else if (warp >= kFirstEpi) {
        // ---- convert and store this CTA's 128 tokens: two warps per 32 rows take the tile's 32-column units in turn
        const int w = warp - kFirstEpi, q = warp & 3, h = w >> 2;
        static_assert(kEpiWarps >= kMaxStages, "a warp for the activations of each first stage");
        if (w < ahead) {
            pdl_wait();
            if (lane == 0) load_x(w, w, pair);
            __syncwarp();
        }
        const uint32_t lane_base = (uint32_t)(q * 32) << 16;
        uint8_t* const buf = epi + (size_t)w * kUnitBytes;
        const uint32_t to = smem_u32(buf) + lane * 64, swizzle = (lane >> 1) & 3;   // row `lane`: four 16-byte chunks under the 64-byte swizzle
        const int units = bn / kUnitCols;
        bool ok = true;
        if (p.bias_given) pdl_wait();
        for (int tl = 0; tl < my_tiles; ++tl) {
            const int tile = pair + tl * G;
            const int m0 = (tile / p.tiles_n) * (2 * kBM) + (int)rank * kBM + q * 32, n0 = (tile % p.tiles_n) * bn;
            const int a = tl & 1;
            const uint32_t bias_at = smem_u32(sh->bias[a]);
            for (int i = tid - 32 * kFirstEpi; i < bn; i += 32 * kEpiWarps)
                sh->bias[a][i] = n0 + i < p.N ? p.bias[n0 + i] : __float2half(0.f);
            epi_barrier();
            if (ok) ok = mbar_wait(&sh->acc_full[a], (uint32_t)(tl >> 1) & 1u);
            if (!ok) continue;   // the barrier above needs every warp
            tc_fence_after();
            if (tl + 1 == my_tiles) pdl_launch_dependents();
            auto accumulator_read = [&]() {
                tc_fence_before();
                __syncwarp();
                if (elect_one()) mbar_arrive_cluster(in_cta(&sh->acc_empty[a], 0));
                __syncwarp();
            };
            NotFinite odd;
            for (int u = h; u < units; u += kEpiWarps / 4) {
                uint32_t acc[32];
                tmem_ld32(tmem + a * bn + lane_base + u * kUnitCols, acc);
                tmem_ld_wait(acc);
                if (u + kEpiWarps / 4 >= units) accumulator_read();   // this warp's share: it may be overwritten
                uint4 ov[4];
                uint4 bv[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) bv[c] = lds128(bias_at + u * kUnitCols * 2 + c * 16);
                epi_convert_regs<kGelu>(acc, bv, ov);
                tma_store_wait_read();   // the buffer's previous store has read it
                __syncwarp();
#pragma unroll
                for (int c = 0; c < 4; ++c) sts128(to + ((c ^ swizzle) << 4), ov[c]);
                if constexpr (kPruned) {
#pragma unroll
                    for (int c = 0; c < 4; ++c) odd.note(ov[c]);
                }
                fence_proxy_async_smem();
                __syncwarp();
                if (n0 + u * kUnitCols < p.N && m0 < p.T && elect_one()) {
                    tma_store_2d(&tmY, buf, n0 + u * kUnitCols, m0);
                    tma_store_commit();
                }
                __syncwarp();
            }
            if (h >= units) accumulator_read();
            if (kPruned && __any_sync(0xffffffffu, odd.any())) {
                tma_store_wait();   // the results are in memory
                __syncwarp();
                fence_proxy_async_global();
                for (int u = h; u < units && odd.any() && m0 + lane < p.T; u += kEpiWarps / 4)
                    for (int c = n0 + u * kUnitCols; c < min(n0 + (u + 1) * kUnitCols, p.N); c += 8) recompute_segment<kGelu>(p, m0 + lane, c);
                __syncwarp();
            }
        }
        if (!ok && lane == 0) atomicExch(p.err, 33);
        tma_store_wait_read();
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    cluster_sync();   // nobody still reads this CTA's shared memory or signals its barriers
    tc_fence_after();
    if (warp == kCopyWarps) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tmem_cols(2 * bn)) : "memory");
}

// ------------------------------------------------------------------------------------------ K split over a cluster
constexpr int kSplitThreads = 256;

// Four words to the address `addr` of CTA `rank` of the cluster, which count towards the bytes that its barrier at `bar` waits for.
__device__ __forceinline__ void st_async_cluster(uint32_t addr, uint32_t bar, uint32_t rank, const uint32_t* v) {
    asm volatile("{\n.reg .b32 a, b;\nmapa.shared::cluster.u32 a, %0, %2;\nmapa.shared::cluster.u32 b, %1, %2;\n"
                 "st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [a], {%3,%4,%5,%6}, [b];\n}" ::"r"(addr), "r"(bar), "r"(rank),
                 "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3])
                 : "memory");
}
// A bounded wait like mbar_wait, for what other CTAs of the cluster have written.
__device__ __forceinline__ bool mbar_wait_cluster(uint32_t bar, uint32_t parity) {
#pragma unroll 1
    for (uint32_t i = 0; i < kMbarSpinLimit; ++i) {
        uint32_t ok;
        asm volatile("{\n.reg .pred P;\nmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 P, [%1], %2;\nselp.u32 %0, 1, 0, P;\n}"
                     : "=r"(ok)
                     : "r"(bar), "r"(parity)
                     : "memory");
        if (ok) return true;
    }
    return false;
}

// Bound by a chain of latencies: of the ~7500 clocks from launch to launch of 128 x 768 -> 768 (3.9 us), ~2700 lie between the end of the
// kernel before and the return of griddepcontrol.wait, 1300-1400 between the request of the activations and the first UMMA, 1200 to the
// last panel's UMMAs, 700 are the sends of accumulators, 600 their way, 1000 the sums and stores. So nothing waits that need not: the first stages' weight is requested
// before the other warps know the barriers, the activations by warps of their own without a look at empty stages, and each CTA
// waits for the bytes of its own columns instead of a barrier of the cluster behind all sends (1450 clocks). Before: 4.2 us, 3072 -> 768 6.3 (5.6 now),
// 4096 -> 1024 7.3 (6.3), 256 x 1024 -> 1024 6.3 (5.5).
template <bool kGelu, bool kPruned>
__global__ void __launch_bounds__(kSplitThreads, 1) dense_split_kernel(const __grid_constant__ CUtensorMap tmX,
                                                                       const __grid_constant__ CUtensorMap tmW,
                                                                       const __grid_constant__ DenseParams p, int split) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int S = p.stages, bn = p.bn;
    const int b_panel = bn * kBK * 2;
    const int stage_bytes = p.panels * (kAPanel + b_panel);
    // What the other shares send of this CTA's columns: [share][four columns][row], this CTA's own share left out.
    const int own_cols = bn / split;
    float4* const recv = reinterpret_cast<float4*>(smem + (size_t)S * stage_bytes);
    DenseShared* const sh = reinterpret_cast<DenseShared*>(recv + (size_t)(split - 1) * (own_cols / 4) * kBM);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = (int)cluster_rank();
    const int tile = (int)blockIdx.x / split;
    const int m0 = (tile / p.tiles_n) * kBM, n0 = (tile % p.tiles_n) * bn;
    const int kp0 = rank * p.k_panels / split, kp1 = (rank + 1) * p.k_panels / split;   // this CTA's panels
    const int kn = (kp1 - kp0 + p.panels - 1) / p.panels;                               // in stages
    const int cw = copy_warps(S), first = min(S, kn);
    auto expect = [&](int s, int kc) { mbar_expect_tx(&sh->full[s], min(p.panels, kp1 - kp0 - kc * p.panels) * (kAPanel + b_panel)); };
    auto load_w = [&](int s, int kc) {
        const int k0 = kp0 + kc * p.panels, np = min(p.panels, kp1 - k0);
        for (int i = 0; i < np; ++i)
            tma_load_2d(smem + (size_t)s * stage_bytes + p.panels * kAPanel + i * b_panel, &tmW, (k0 + i) * kBK, n0, &sh->full[s]);
    };
    auto load_x = [&](int s, int kc) {
        const int k0 = kp0 + kc * p.panels, np = min(p.panels, kp1 - k0);
        for (int i = 0; i < np; ++i) tma_load_2d(smem + (size_t)s * stage_bytes + i * kAPanel, &tmX, (k0 + i) * kBK, m0, &sh->full[s]);
    };
    // The first stages: the weight's panels, which do not depend on the preceding kernel, by the warp that makes the barriers, as soon as
    // they exist; the activations by three others, which wait for the preceding kernel meanwhile.
    if (warp == 0) {
        if (lane == 0) {
            for (int i = 0; i < S; ++i) { mbar_init(&sh->full[i], 1); mbar_init(&sh->empty[i], 1); }
            mbar_init(&sh->acc_full[0], 1);
            mbar_init(&sh->received, 1);
            fence_mbar_init();
            for (int i = 0; i < first; ++i) expect(i, i);
            mbar_expect_tx(&sh->received, (uint32_t)((split - 1) * own_cols * kBM * 4));
        }
        __syncwarp();
        asm volatile("bar.arrive 2, %0;" ::"n"(kSplitThreads) : "memory");
        if (lane == 0)
            for (int i = 0; i < first; ++i) load_w(i, i);
        __syncwarp();
        asm volatile("bar.sync 3, 64;" ::: "memory");   // tensor memory has been allocated
    } else {
        if (warp == kCopyWarps) {
            tmem_alloc(&sh->tmem_base, tmem_cols(bn));
            tmem_relinquish();
        }
        tc_fence_before();
        asm volatile("bar.sync 2, %0;" ::"n"(kSplitThreads) : "memory");
        if (warp == kCopyWarps) asm volatile("bar.arrive 3, 64;" ::: "memory");
    }
    tc_fence_after();
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");   // this CTA runs: its memory may be written to
    pdl_wait();
    bool ok = true;
    if (warp < cw) {
        int s = warp;
        uint32_t ph = 0;
        for (int i = warp + S; i < kn; i += cw) {
            ok = mbar_wait(&sh->empty[s], ph);
            if (!ok) break;
            if (lane == 0) { expect(s, i); load_w(s, i); load_x(s, i); }
            __syncwarp();
            s += cw;
            if (s >= S) { s -= S; ph ^= 1u; }
        }
    } else if (warp == kCopyWarps) {
        const uint32_t tmem = lds32(smem_u32(&sh->tmem_base)), full = smem_u32(&sh->full[0]), empty = smem_u32(&sh->empty[0]);
        const uint32_t idesc = make_idesc_f16(kBM, bn);
        const uint64_t a0 = make_smem_desc(smem_u32(smem), 16, 1024, 2);
        const uint64_t b0 = make_smem_desc(smem_u32(smem) + p.panels * kAPanel, 16, 1024, 2);
        if (elect_one()) {
            int s = 0;
            uint32_t ph = 0;
            for (int i = 0; i < kn; ++i) {
                ok = mbar_wait_at(full + s * 8, ph);
                if (!ok) break;
                tc_fence_after();
                const uint64_t at = (uint64_t)(s * stage_bytes) >> 4;   // descriptors count 16-byte units
                const int np = min(p.panels, kp1 - kp0 - i * p.panels);
                for (int j = 0; j < np; ++j)
#pragma unroll
                    for (int ks = 0; ks < 4; ++ks)
                        umma_f16(tmem, a0 + at + (j * kAPanel >> 4) + ks * 2, b0 + at + (j * b_panel >> 4) + ks * 2, idesc,
                                 (i > 0 || j > 0 || ks > 0) ? 1u : 0u);
                umma_commit_at(empty + s * 8);
                if (i + 1 == kn) umma_commit_at(smem_u32(&sh->acc_full[0]));
                if (++s == S) { s = 0; ph ^= 1u; }
            }
        }
        __syncwarp();
    }
    if (warp > kCopyWarps) {
        if (lane == 0)
            for (int i = warp - kCopyWarps - 1; i < first; i += kSplitThreads / 32 - kCopyWarps - 1) load_x(i, i);
        __syncwarp();
        // the bias, which may be the caller's and the preceding kernel's result (read behind the barrier below)
        for (int i = tid - 32 * (kCopyWarps + 1); i < own_cols; i += kSplitThreads - 32 * (kCopyWarps + 1)) {
            const int n = n0 + rank * own_cols + i;
            sh->bias[0][i] = n < p.N ? p.bias[n] : __float2half(0.f);
        }
    }
    // every copy has landed and every UMMA has read its operands when the accumulator is complete
    const bool fin = mbar_wait(&sh->acc_full[0], 0);
    if ((!ok || !fin) && lane == 0) {
        atomicExch(p.err, 34);
        if (warp < cw)   // copies in flight land before the CTA leaves (bounded)
            for (int i = 0; i < min(S, kn); ++i) mbar_wait(&sh->full[i], 0);
    }
    __syncwarp();
    tc_fence_after();
    const uint32_t tmem = sh->tmem_base;
    pdl_launch_dependents();
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");   // every CTA of the cluster runs
    const int q = warp & 3, h = warp >> 2;   // two warps per 32 rows
    const int row = q * 32 + lane;
    const uint32_t acc = tmem + ((uint32_t)(q * 32) << 16);
    // Every CTA finishes own_cols of the tile's columns and sends the others theirs, straight from tensor memory: stores into the
    // other CTAs' shared memory go on without waiting, loads from it (a round trip each) took 2 us more.
    for (int c = h * 16; c < bn; c += 32) {
        uint32_t r[16];
        tmem_ld16(acc + c, r);
        tmem_ld_wait(r);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int dst = (c + 4 * i) / own_cols, g = (c + 4 * i - dst * own_cols) / 4;
            if (dst == rank) continue;   // the same for the whole CTA
            const int from = rank < dst ? rank : rank - 1;
            st_async_cluster(smem_u32(recv + ((size_t)from * (own_cols / 4) + g) * kBM + row), smem_u32(&sh->received), dst, r + 4 * i);
        }
    }
    __syncthreads();                                                        // the bias lies in shared memory
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");   // this warp has sent everything
    const bool got = mbar_wait_cluster(smem_u32(&sh->received), 0);
    if (!got && lane == 0) atomicExch(p.err, 35);
    __syncwarp();
    auto finish = [&](const uint32_t* own, int c, uint32_t* out) {   // four of the own columns, from c on
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        for (int k = 0; k < split; ++k) {   // in the order of the shares
            float4 x = make_float4(__uint_as_float(own[0]), __uint_as_float(own[1]), __uint_as_float(own[2]), __uint_as_float(own[3]));
            if (k != rank) x = recv[((size_t)(k < rank ? k : k - 1) * (own_cols / 4) + c / 4) * kBM + row];
            v[0] += x.x; v[1] += x.y; v[2] += x.z; v[3] += x.w;
        }
        const half2* bias = reinterpret_cast<const half2*>(sh->bias[0] + c);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const float2 b = __half22float2(bias[j]);
            half2 t = __floats2half2_rn(v[2 * j] + b.x, v[2 * j + 1] + b.y);
            if constexpr (kGelu) t = gelu_tanh_h2(t);
            out[j] = *reinterpret_cast<const uint32_t*>(&t);
        }
    };
    auto not_finite = [&](const uint32_t* out, int n) {   // any of 2 n results
        half2 t = __float2half2_rn(0.f);
        for (int i = 0; i < n; ++i) t = __hfma2(*reinterpret_cast<const half2*>(out + i), __float2half2_rn(0.f), t);
        return !(__low2float(t) + __high2float(t) == 0.f);
    };
    half* const y = p.Y + (size_t)(m0 + row) * p.N + n0 + rank * own_cols;
    const int left = m0 + row < p.T ? p.N - n0 - rank * own_cols : 0;   // columns of this row that exist
    const bool wide = (reinterpret_cast<uintptr_t>(p.Y) & 31) == 0 && ((n0 + rank * own_cols) & 15) == 0;
    for (int c = h * 16; c + 16 <= own_cols; c += 32) {
        uint32_t own[16], out[8];
        tmem_ld16(acc + rank * own_cols + c, own);
        tmem_ld_wait(own);
#pragma unroll
        for (int i = 0; i < 4; ++i) finish(own + 4 * i, c + 4 * i, out + 2 * i);
        if (wide && c + 16 <= left) {   // a whole sector
            asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(y + c), "r"(out[0]), "r"(out[1]), "r"(out[2]), "r"(out[3]), "r"(out[4]),
                         "r"(out[5]), "r"(out[6]), "r"(out[7])
                         : "memory");
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (c + 4 * i < left) *reinterpret_cast<uint2*>(y + c + 4 * i) = make_uint2(out[2 * i], out[2 * i + 1]);
        }
        if constexpr (kPruned) {
            if (not_finite(out, 8))
                for (int i = c; i < min(c + 16, left); i += 4) recompute_segment<kGelu, 4>(p, m0 + row, n0 + rank * own_cols + i);
        }
        __syncwarp();   // the next load from tensor memory needs every lane
    }
    for (int c = own_cols / 16 * 16 + h * 4; c < own_cols; c += 8) {
        uint32_t own[4], out[2];
        tmem_ld4(acc + rank * own_cols + c, own);
        tmem_ld_wait(own);
        finish(own, c, out);
        if (c < left) {
            *reinterpret_cast<uint2*>(y + c) = make_uint2(out[0], out[1]);
            if constexpr (kPruned) {
                if (not_finite(out, 2)) recompute_segment<kGelu, 4>(p, m0 + row, n0 + rank * own_cols + c);
            }
        }
        __syncwarp();
    }
    // Normally all have sent when this CTA has received. One that gave up stays until nothing is on its way to it.
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    if (!got) mbar_wait_cluster(smem_u32(&sh->received), 0);
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == kCopyWarps) tmem_dealloc(tmem, tmem_cols(bn));
}

}  // namespace

// Panels per stage and stages that fit.
static int panels_for(int bn, int split) { return split > 1 || bn <= 128 ? 2 : 1; }

// CTAs of a cluster of `split` that run at once (one CTA per SM; clusters do not straddle the groups of 16-20 SMs, so that of
// the larger ones fewer fit: 74, 33 and 15 of two, four and eight by cudaOccupancyMaxActiveClusters; the model is fitted with 14).
static int split_capacity(int split) { return split == 8 ? 14 * 8 : split == 4 ? 33 * 4 : sm_count() / split * split; }

// Cost in clocks of a launch over `tokens` with tile width bn and the K range split over `split` CTAs: waves of tiles, each
// K panel taking its UMMAs (2 bn clocks) or its copies (an SM gets 55-67 bytes per clock from L2 when all ask), plus what comes
// before the first UMMA and after the last one, and what the columns exchanged within a cluster take. Fitted to launches of 64 to 4096 tokens
// and ten shapes in every width and split: the plan taken is 0.3 % slower than the fastest in the mean, 8 % at most. (64 x 768 -> 2304 5.8 us in 36 tiles split in two, 7.4 in 9
// pairs; 384 x 768 -> 1152 5.6 in 36 pairs' tiles of 64, 6.5 in 72 of 32.)
static double dense_cost(int tokens, int N, int K, int bn, int split) {
    const int tiles_n = (N + bn - 1) / bn;
    const int panels = (K + kBK - 1) / kBK;
    if (split == 1) {
        const int pairs = sm_count() / 2, tiles = (tokens + 2 * kBM - 1) / (2 * kBM) * tiles_n;
        const int waves = (tiles + pairs - 1) / pairs;
        // Where the next launch finds SMs free it starts under this one: 512 x 768 -> 1152 takes 5.6 us on 72 SMs and 6.6 on 144.
        const double full = 2 * tiles > sm_count() - 16 ? 2400.0 : 2 * tiles > sm_count() / 2 ? 1950.0 : 0.0;
        const double panel = std::max({2.0 * bn, (kAPanel + bn * 64.0) / 67.0, 475.0 / panels_for(bn, 1)});
        const double tile = std::max(panels * panel, bn * 9.0);   // the main loop, or the stores of the tile before
        // a long launch of dense UMMAs runs at the power limit: 1.4e15 operations per second on the whole GPU, those for the columns
        // that fill up the last tile included (65536 x 768 -> 384 in tiles of 256 columns 45.4 us, of 192 41.7; 24000 -> 576 25.2 and 23.5)
        const double power = 2.0 * tokens * tiles_n * bn * (double)K / 1.4e15 * 1.9e9;
        return 5800.0 + std::max(full + waves * tile + bn * 15.0, power);
    }
    const int tiles = std::max(1, (tokens + kBM - 1) / kBM) * tiles_n;
    const double panel = std::max({2.0 * bn, (kAPanel + bn * 128.0) / 55.0, 360.0});
    const int waves = (tiles * split + split_capacity(split) - 1) / split_capacity(split);
    // clusters on nearly all SMs: the last ones start late
    const double full = tiles * split > sm_count() - 16 ? 1250.0 : tiles * split > sm_count() - 48 ? 650.0 : 0.0;
    return 6000.0 + full + waves * (((panels + split - 1) / split) * panel + bn * 48.0 * (split - 1) / split);
}

DensePlan dense_plan(int tokens, int N, int K) {
    DensePlan best;
    for (int bn : {256, 192, 128, 96, 64, 32}) {
        if (bn > 32 && bn - 32 >= N) continue;   // no narrower tile would leave columns out
        for (int split : {1, 2, 4, 8}) {
            const int panels = (K + kBK - 1) / kBK;
            if (split > 1 && (split > panels || bn > 128)) continue;
            const double c = dense_cost(tokens, N, K, bn, split);
            if (best.bn == 0 || c < best.cost * 0.98) best = DensePlan{bn, split, c};
        }
    }
    return best;
}

// Weight rows per copy: a tile's width, or half of it for each CTA of a pair.
constexpr int kBoxRows[6] = {16, 32, 48, 64, 96, 128};

int dense_map_weight(DenseWeight* w) {
    for (int i = 0; i < 6; ++i)
        if (!make_tmap_2d_f16(&w->maps[i], w->W, (uint64_t)w->N, (uint64_t)w->K, (uint64_t)w->K, (uint32_t)kBoxRows[i], kBK, 128))
            return fail(ET_ERR_CUDA, "dense linear: cuTensorMapEncodeTiled failed");
    return ET_OK;
}

int dense_run(const DenseWeight& w, const DensePlan& plan, half* Y, const half* X, const half* bias, bool bias_given, int T, int gelu, int* err, cudaStream_t st) {
    const int N = w.N, K = w.K;
    const int box = (int)(std::find(kBoxRows, kBoxRows + 6, plan.split > 1 ? plan.bn : plan.bn / 2) - kBoxRows);
    if (box == 6) return fail(ET_ERR_INVALID, "dense linear: no such tile width");
    const CUtensorMap& tmW = w.maps[box];
    CUtensorMap tmX, tmY;
    if (!make_tmap_2d_f16(&tmX, X, (uint64_t)T, (uint64_t)K, (uint64_t)K, kBM, kBK, 128))
        return fail(ET_ERR_CUDA, "dense linear: cuTensorMapEncodeTiled failed");
    // [gelu][pruned]
    using PairFn = void (*)(CUtensorMap, CUtensorMap, CUtensorMap, DenseParams);
    using SplitFn = void (*)(CUtensorMap, CUtensorMap, DenseParams, int);
    static const PairFn pair[2][2] = {{dense_kernel<false, false>, dense_kernel<false, true>}, {dense_kernel<true, false>, dense_kernel<true, true>}};
    static const SplitFn split[2][2] = {{dense_split_kernel<false, false>, dense_split_kernel<false, true>},
                                        {dense_split_kernel<true, false>, dense_split_kernel<true, true>}};
    const int g = gelu ? 1 : 0, pruned = w.kept ? 1 : 0;
    static PerDeviceOnce once;
    const cudaError_t attr_err = once.run([] {
        cudaError_t e = cudaSuccess;
        for (int i = 0; i < 4 && e == cudaSuccess; ++i) {
            e = cudaFuncSetAttribute(pair[i >> 1][i & 1], cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax);
            if (e == cudaSuccess) e = cudaFuncSetAttribute(split[i >> 1][i & 1], cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax);
        }
        return e;
    });
    if (attr_err != cudaSuccess) return cuda_status(attr_err, "dense linear: shared memory opt-in");
    DenseParams p;
    p.bias = bias; p.bias_given = bias_given; p.Y = Y; p.T = T; p.N = N; p.K = K; p.bn = plan.bn;
    p.X = X; p.W = w.W; p.kept = w.kept;
    p.k_panels = (K + kBK - 1) / kBK;
    p.tiles_n = (N + plan.bn - 1) / plan.bn;
    p.panels = panels_for(plan.bn, plan.split);
    p.err = err;
    cudaLaunchConfig_t cfg = {};
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    if (plan.split > 1) {
        const int stage = p.panels * (kAPanel + plan.bn * kBK * 2);
        p.tiles = ((T + kBM - 1) / kBM) * p.tiles_n;
        const int recv = (plan.split - 1) * (plan.bn / plan.split) * kBM * 4;
        p.stages = ring_stages(std::min({kMaxStages, (kSmemMax - 1024 - (int)sizeof(DenseShared) - recv) / stage,
                                         ((p.k_panels + plan.split - 1) / plan.split + p.panels - 1) / p.panels}));
        cfg.gridDim = dim3((unsigned)(p.tiles * plan.split));
        cfg.blockDim = dim3(kSplitThreads);
        cfg.dynamicSmemBytes = (size_t)p.stages * stage + recv + sizeof(DenseShared) + 1024;
        attr[1].val.clusterDim.x = (unsigned)plan.split;
        return cuda_status(cudaLaunchKernelEx(&cfg, split[g][pruned], tmX, tmW, p, plan.split), "dense linear launch");
    }
    if (!make_tmap_2d_f16(&tmY, Y, (uint64_t)T, (uint64_t)N, (uint64_t)N, 32, kUnitCols, 64))
        return fail(ET_ERR_CUDA, "dense linear: cuTensorMapEncodeTiled failed");
    const int stage = p.panels * (kAPanel + plan.bn * kBK);
    p.tiles = ((T + 2 * kBM - 1) / (2 * kBM)) * p.tiles_n;
    p.stages = ring_stages(std::min(kMaxStages, (kSmemMax - 1024 - (int)sizeof(DenseShared) - kEpiWarps * kUnitBytes) / stage));
    cfg.gridDim = dim3((unsigned)(2 * std::min(p.tiles, sm_count() / 2)));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = (size_t)p.stages * stage + kEpiWarps * kUnitBytes + sizeof(DenseShared) + 1024;
    attr[1].val.clusterDim.x = 2;
    return cuda_status(cudaLaunchKernelEx(&cfg, pair[g][pruned], tmX, tmW, tmY, p), "dense linear launch");
}

}  // namespace et
