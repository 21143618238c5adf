// Host-side layer objects: the row-pruned linear and the three encoder-layer variants, plus their
// C-ABI entry points. Replaces encoder/Linear.cu:60-91 (Linear_row), encoder/encoder.h:7-134 and
// encoder/encoder.cu:4-149 (Encoder_base / Encoder_tile / Encoder_prune / Encoder_length) of the reference.
//
// Differences from the reference by design: one stream, no host synchronisation inside run(), no cuBLAS;
// a batch of packed variable-length sequences is a first-class input (run_batch); every failure is a
// status code instead of exit(1).
#include <algorithm>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <tuple>
#include <vector>
#include "attention.h"
#include "common.h"
#include "formats.h"
#include "handles.h"
#include "tile_gemm.h"


namespace et {

// ------------------------------------------------------------------------------ row-pruned linear
// Only `row_id_size` output features survive (sorted original indices in row_id); the weight is the
// compact [row_id_size x in_feat] matrix. Output is [tokens x nrow] with nrow = row_id_size rounded up
// to 16 (zero columns beyond row_id_size), the pitch every consumer uses. The contraction is a
// tile weight with every tile kept, in whichever form is the shortest launch for it (tile_weight_pack).
struct RowWeight {
    int in_feat = 0, out_feat = 0, nhead = 0, row_id_size = 0, nrow = 0;
    TileWeight* tw = nullptr;
    int* d_row_id = nullptr;
    int* d_head_ptr = nullptr;
    std::vector<int> h_head_ptr, h_row_id;
    std::vector<half> h_weight, h_bias;   // as given, for layers that lay the rows out with padded heads
    ~RowWeight() {
        tile_weight_free(tw);
        cudaFree(d_row_id);
        cudaFree(d_head_ptr);
    }
};

static int dense_to_tiles(const half* weight, int rows, int K, std::vector<half>& data,
                          std::vector<int>& row_ptr, std::vector<int>& row_offset) {
    const int nrow = (rows + 15) / 16 * 16;
    const int brs = nrow / 16, bcs = K / 16;
    data.assign((size_t)brs * bcs * 256, __float2half(0.f));
    row_ptr.resize(brs + 1);
    row_offset.resize((size_t)brs * bcs);
    for (int r = 0; r < brs; ++r) {
        row_ptr[r] = r * bcs;
        for (int c = 0; c < bcs; ++c) {
            const size_t i = (size_t)r * bcs + c;
            row_offset[i] = c * 16;
            for (int n = 0; n < 16 && 16 * r + n < rows; ++n)
                std::memcpy(&data[i * 256 + n * 16], weight + (size_t)(16 * r + n) * K + 16 * c, 32);
        }
    }
    row_ptr[brs] = brs * bcs;
    return nrow;
}

static int row_weight_create(RowWeight** out, int in_feat, int out_feat, int size, const half* weight,
                             const int* row_id, int row_id_size, const half* bias, int nhead) {
    if (!out) return fail(ET_ERR_INVALID, "row weight: null output");
    *out = nullptr;
    if (in_feat <= 0 || in_feat % 16 || out_feat <= 0 || row_id_size <= 0 || row_id_size > out_feat)
        return fail(ET_ERR_INVALID, "row weight: bad dimensions (in_feat must be a multiple of 16)");
    if (!weight || !row_id) return fail(ET_ERR_INVALID, "row weight: null array");
    if (nhead <= 0 || out_feat % nhead) return fail(ET_ERR_INVALID, "row weight: out_feat not divisible by nhead");
    for (int i = 0; i < row_id_size; ++i)
        if (row_id[i] < 0 || row_id[i] >= out_feat || (i && row_id[i] <= row_id[i - 1]))
            return fail(ET_ERR_INVALID, "row weight: row_id must be strictly ascending inside [0, out_feat)");
    auto w = std::make_unique<RowWeight>();
    w->in_feat = in_feat; w->out_feat = out_feat; w->nhead = nhead; w->row_id_size = row_id_size;
    std::vector<half> data;
    std::vector<int> rp, ro;
    w->nrow = dense_to_tiles(weight, row_id_size, in_feat, data, rp, ro);
    std::vector<half> pbias(w->nrow, __float2half(0.f));
    if (bias) std::copy(bias, bias + row_id_size, pbias.begin());
    int rc = tile_weight_pack(&w->tw, in_feat, w->nrow, size, (long)ro.size(), data.data(), rp.data(),
                              ro.data(), pbias.data(), 0);
    if (rc) return rc;
    build_head_ptr(row_id, row_id_size, nhead, out_feat, w->h_head_ptr);
    if (cudaMalloc(&w->d_row_id, sizeof(int) * row_id_size) != cudaSuccess ||
        cudaMalloc(&w->d_head_ptr, sizeof(int) * (nhead + 1)) != cudaSuccess)
        return fail(ET_ERR_CUDA, "row weight: cudaMalloc failed");
    cudaMemcpy(w->d_row_id, row_id, sizeof(int) * row_id_size, cudaMemcpyHostToDevice);
    cudaMemcpy(w->d_head_ptr, w->h_head_ptr.data(), sizeof(int) * (nhead + 1), cudaMemcpyHostToDevice);
    rc = cuda_status(cudaDeviceSynchronize(), "row weight: upload");   // launches on any stream may follow
    if (rc) return rc;
    w->h_row_id.assign(row_id, row_id + row_id_size);
    w->h_weight.assign(weight, weight + (size_t)row_id_size * in_feat);
    w->h_bias.assign(pbias.begin(), pbias.begin() + row_id_size);
    *out = w.release();
    return ET_OK;
}

// The same rows with every head's share padded with zero rows to a multiple of 16 (at least 16): the layout in which the
// attention kernel can address a head's columns. ptr[h]: first row of head h.
static int row_weight_padded(TileWeight** out, const RowWeight* w, int size, std::vector<int>& ptr) {
    ptr.assign(1, 0);
    for (int h = 0; h < w->nhead; ++h) ptr.push_back(ptr.back() + std::max(16, (w->h_head_ptr[h + 1] - w->h_head_ptr[h] + 15) / 16 * 16));
    const int N = ptr.back(), K = w->in_feat;
    std::vector<half> weight((size_t)N * K, __float2half(0.f)), bias((size_t)N, __float2half(0.f)), data;
    for (int h = 0; h < w->nhead; ++h) {
        const int r0 = w->h_head_ptr[h], n = w->h_head_ptr[h + 1] - r0;
        std::copy_n(w->h_weight.begin() + (size_t)r0 * K, (size_t)n * K, weight.begin() + (size_t)ptr[h] * K);
        std::copy_n(w->h_bias.begin() + r0, n, bias.begin() + ptr[h]);
    }
    std::vector<int> rp, ro;
    dense_to_tiles(weight.data(), N, K, data, rp, ro);
    return tile_weight_pack(out, K, N, size, (long)ro.size(), data.data(), rp.data(), ro.data(), bias.data(), 0, true);
}

namespace {
std::mutex g_row_mu;
std::map<std::tuple<const void*, int, int>, TileWeight*> g_row_cache;
}  // namespace

int row_spmm_raw(half* out, const half* in, const half* weight, const half* bias, int M, int N, int K, cudaStream_t st) {
    TileWeight* tw = nullptr;
    {
        std::lock_guard<std::mutex> lk(g_row_mu);
        auto key = std::make_tuple((const void*)weight, N, K);
        auto it = g_row_cache.find(key);
        if (it == g_row_cache.end()) {
            std::vector<half> hw((size_t)N * K);
            if (cudaMemcpy(hw.data(), weight, hw.size() * sizeof(half), cudaMemcpyDeviceToHost) != cudaSuccess)
                return fail(ET_ERR_CUDA, "row spmm: cannot read the weight");
            std::vector<half> data;
            std::vector<int> rp, ro;
            dense_to_tiles(hw.data(), N, K, data, rp, ro);
            int rc = tile_weight_pack(&tw, K, N, M, (long)ro.size(), data.data(), rp.data(), ro.data(), nullptr, 0);
            if (rc) return rc;
            g_row_cache[key] = tw;
        } else {
            tw = it->second;
        }
    }
    return tile_linear_run(tw, out, in, M, 0, st, bias);
}

void row_spmm_cache_clear() {
    std::lock_guard<std::mutex> lk(g_row_mu);
    for (auto& kv : g_row_cache) tile_weight_free(kv.second);
    g_row_cache.clear();
}

// ------------------------------------------------------------------------------ encoder layer
enum EncoderKind { kTile = 0, kPrune = 1, kLength = 2, kPruneQKV = 3 };

// One instantiated CUDA graph per distinct call (buffers, lengths) of a layer or a stack: its launches replayed without the
// host cost of each and without the gaps between them. The first call with a key runs directly, the second is captured, later
// ones replay. Capture takes place on a stream of the cache's own (the legacy default stream cannot be captured); the graph is
// launched into the caller's stream, the legacy one included.
struct ReplayCache {
    struct Entry {
        std::vector<int64_t> key;
        int seen = 0;
        cudaGraphExec_t exec = nullptr;
    };
    static constexpr size_t kEntries = 8;
    std::vector<Entry> entries;
    std::vector<int64_t> key;      // of the call being made
    bool on = true;
    cudaStream_t own = nullptr;
    void drop() {
        for (auto& r : entries)
            if (r.exec) cudaGraphExecDestroy(r.exec);
        entries.clear();
    }
    ~ReplayCache() {
        drop();
        if (own) cudaStreamDestroy(own);
    }
    // Runs `forward(stream)` directly or replays it, for the call that `key` describes.
    template <typename F>
    int run(cudaStream_t st, const char* what, F&& forward) {
        Entry* slot = nullptr;
        for (auto& r : entries)
            if (r.key == key) { slot = &r; break; }
        if (slot && slot->exec) return cuda_status(cudaGraphLaunch(slot->exec, st), what);
        if (!slot) {
            if (entries.size() >= kEntries) {
                if (entries.front().exec) cudaGraphExecDestroy(entries.front().exec);
                entries.erase(entries.begin());
            }
            entries.push_back({key, 0, nullptr});
            slot = &entries.back();
        }
        if (slot->seen++ == 0) return forward(st);
        if ((!own && cudaStreamCreateWithFlags(&own, cudaStreamNonBlocking) != cudaSuccess) ||
            cudaStreamBeginCapture(own, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
            cudaGetLastError();
            return forward(st);
        }
        const int frc = forward(own);
        cudaGraph_t graph = nullptr;
        const cudaError_t ce = cudaStreamEndCapture(own, &graph);
        const bool good = frc == ET_OK && ce == cudaSuccess && graph && cudaGraphInstantiate(&slot->exec, graph, 0) == cudaSuccess;
        if (graph) cudaGraphDestroy(graph);
        if (!good) {
            slot->exec = nullptr;
            cudaGetLastError();
            on = false;   // plain launches from now on
            return forward(st);
        }
        return cuda_status(cudaGraphLaunch(slot->exec, st), what);
    }
};

// Sequence offsets and key counts on the device (offsets of batch + 1, then counts of batch). The array grows geometrically; a
// recorded graph holds its address as a kernel argument, so every graph recorded with the old array is dropped before it is
// freed. A call with the lengths that the array holds already, on the stream that uploaded them, uploads nothing. A call inside
// the caller's own capture gets an array that is filled then and there and never written again: the caller's graph may be
// launched at any time, between direct calls with other lengths and beside them.
struct LengthArray {
    int* d = nullptr;
    int cap = 0;
    std::vector<int> held;
    unsigned long long held_stream = 0;
    std::map<std::vector<int>, int*> captured;   // by content; as long-lived as the object, as the graphs hold them
    ~LengthArray() {
        cudaFree(d);
        for (auto& kv : captured) cudaFree(kv.second);
    }
    int upload(const std::vector<int>& meta, cudaStream_t st, ReplayCache& graphs, const char* what) {
        const int need = (int)meta.size();
        if (cap < need) {
            graphs.drop();
            held.clear();
            const int ncap = std::max(need, std::max(64, 2 * cap));
            int* fresh = nullptr;
            if (cudaMalloc(&fresh, sizeof(int) * (size_t)ncap) != cudaSuccess) return fail(ET_ERR_CUDA, "lengths: cudaMalloc failed");
            cudaFree(d);   // synchronises with work still reading the old array
            d = fresh;
            cap = ncap;
        }
        unsigned long long id = 0;
        const bool known = cudaStreamGetId(st, &id) == cudaSuccess;
        if (known && id == held_stream && held == meta) return ET_OK;
        const int rc = cuda_status(cudaMemcpyAsync(d, meta.data(), sizeof(int) * (size_t)need, cudaMemcpyHostToDevice, st), what);
        held.clear();
        if (rc == ET_OK && known) { held = meta; held_stream = id; }
        return rc;
    }
    // For a call inside the caller's capture: allocates and fills on a stream beside it (the capture mode of this thread is
    // relaxed meanwhile; nothing of this becomes part of the caller's graph).
    int in_capture(const std::vector<int>& meta, const int** out, const char* what) {
        auto it = captured.find(meta);
        if (it != captured.end()) { *out = it->second; return ET_OK; }
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        cudaError_t e = cudaThreadExchangeStreamCaptureMode(&mode);
        if (e != cudaSuccess) return cuda_status(e, what);
        int* fresh = nullptr;
        cudaStream_t side = nullptr;
        e = cudaMalloc(&fresh, sizeof(int) * meta.size());
        if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&side, cudaStreamNonBlocking);
        if (e == cudaSuccess) e = cudaMemcpyAsync(fresh, meta.data(), sizeof(int) * meta.size(), cudaMemcpyHostToDevice, side);
        if (e == cudaSuccess) e = cudaStreamSynchronize(side);
        if (side) cudaStreamDestroy(side);
        if (e != cudaSuccess) cudaFree(fresh);
        cudaThreadExchangeStreamCaptureMode(&mode);
        if (e != cudaSuccess) return cuda_status(e, what);
        captured[meta] = fresh;
        *out = fresh;
        return ET_OK;
    }
};

struct Encoder {
    int kind = kTile, d_model = 0, seq_len = 0, nheads = 0, d_ff = 0;
    half* buffer = nullptr;  // caller-owned scratch for run(): buffer_num * seq_len * d_model halfs (+ scores)
    TileWeight* lin[6] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};  // q k v o mlp1 mlp2
    TileWeight* qkv = nullptr;   // Q|K|V as one weight: one launch, one staging of the activations per CTA
    int qkv_cols[3] = {0, 0, 0}; // output columns of the three parts inside the fused result
    // Row-pruned layers with heads of 64: the row-pruned linears are laid out with padded heads (row_weight_padded), attention
    // works on and produces compact heads, and the output projection has its input features gathered to match. (Expanding the
    // compact operands to 64 per head first, and the projection over all features: 20 us more of 123 at 32 x 256 tokens.)
    TileWeight* o_compact = nullptr;
    int* d_qk_ptr = nullptr; int* d_v_ptr = nullptr;   // first column of each head in Q and K (null: dense) and in V
    RowWeight* rq = nullptr; RowWeight* rk = nullptr; RowWeight* rv = nullptr;
    half* d_ln[4] = {nullptr, nullptr, nullptr, nullptr};  // gamma1 beta1 gamma2 beta2
    std::vector<half> h_ln[4];                             // the same on the host (folded into weights by the layer stack)
    half* d_mask = nullptr;                                // [seq_len x seq_len] additive, may be null
    LengthArray lens;
    bool materialize_scores = false;
    ReplayCache graphs;
    ~Encoder() {
        graphs.drop();
        for (auto* t : lin) tile_weight_free(t);
        tile_weight_free(qkv);
        tile_weight_free(o_compact);
        cudaFree(d_qk_ptr);
        cudaFree(d_v_ptr);
        delete rq; delete rk; delete rv;
        for (auto* p : d_ln) cudaFree(p);
        cudaFree(d_mask);
    }
};

static int upload_half(half** dst, const half* src_host, size_t n) {
    if (cudaMalloc(dst, n * sizeof(half)) != cudaSuccess) return fail(ET_ERR_CUDA, "encoder: cudaMalloc failed");
    return cuda_status(cudaMemcpy(*dst, src_host, n * sizeof(half), cudaMemcpyHostToDevice), "encoder: upload");
}

static int encoder_common(Encoder* e, int d_model, int seq_len, int nheads, half* buffer,
                          const half* g1, const half* b1, const half* g2, const half* b2, const half* mask) {
    if (d_model <= 0 || seq_len <= 0 || nheads <= 0 || d_model % nheads) return fail(ET_ERR_INVALID, "encoder: bad dimensions");
    if (!g1 || !b1 || !g2 || !b2) return fail(ET_ERR_INVALID, "encoder: null LayerNorm parameter");
    {
        // nothing is left to set up when the first attention launch comes (it may sit inside a caller's capture)
        const int rc = attention_prepare_device();
        if (rc) return rc;
    }
    e->d_model = d_model; e->seq_len = seq_len; e->nheads = nheads; e->buffer = buffer;
    const half* src[4] = {g1, b1, g2, b2};
    for (int i = 0; i < 4; ++i) {
        int rc = upload_half(&e->d_ln[i], src[i], d_model);
        if (rc) return rc;
        e->h_ln[i].assign(src[i], src[i] + d_model);
    }
    if (mask) {
        const int rc = upload_half(&e->d_mask, mask, (size_t)seq_len * seq_len);
        if (rc) return rc;
    }
    return cuda_status(cudaDeviceSynchronize(), "encoder: upload");   // launches on any stream may follow
}

// One layer over `T` packed tokens (op order of encoder/encoder.cu:20-45). scratch holds 5*T*d_model halfs:
// [0] Q then the attention-output projection / first LayerNorm result, [1] K, [2] V, [3] attention output,
// [1..4] the T x d_ff hidden activations; scores (materialised variant) follow at 5*T*d_model.
static int encoder_forward(Encoder* e, half* out, const half* in, half* scratch, int T, const int* cu_seqlens,
                           const int* valid_lens, int batch, int uniform_len, cudaStream_t st, int max_len = 0) {
    const size_t td = (size_t)T * e->d_model;
    half* b0 = scratch; half* b1 = scratch + td; half* b2 = scratch + 2 * td; half* b3 = scratch + 3 * td;
    int rc;
    int q_pitch = e->d_model, v_pitch = e->d_model;
    const int *qk_hp = nullptr, *v_hp = nullptr, *v_id = nullptr;
    if (e->o_compact) {
        if ((rc = tile_linear_run(e->qkv, b0, in, T, 0, st))) return rc;
        const int P = e->qkv_cols[0] + e->qkv_cols[1] + e->qkv_cols[2];
        if ((rc = attention_tc_launch(b3, b0, b0 + e->qkv_cols[0], b0 + e->qkv_cols[0] + e->qkv_cols[1], P, P, e->qkv_cols[0],
                                      e->qkv_cols[2], e->d_qk_ptr, e->d_v_ptr, nullptr, e->d_mask, e->seq_len, cu_seqlens, valid_lens,
                                      batch, uniform_len, T, cu_seqlens ? max_len : uniform_len, e->d_model, e->nheads, st)))
            return rc == ET_ERR_UNSUPPORTED ? fail(ET_ERR_INVALID, "encoder: scratch must be 16-byte aligned") : rc;
    } else if (e->qkv) {
        // fused: one launch writes Q | K | V side by side, [T x (q + k + v columns)] over the first three scratch
        // buffers (row-pruned parts are compact, so the three widths may differ)
        if ((rc = tile_linear_run(e->qkv, b0, in, T, 0, st))) return rc;
        q_pitch = v_pitch = e->qkv_cols[0] + e->qkv_cols[1] + e->qkv_cols[2];
        b1 = b0 + e->qkv_cols[0];
        b2 = b1 + e->qkv_cols[1];
        if (e->kind == kPruneQKV) qk_hp = e->rq->d_head_ptr;
        if (e->kind == kPrune || e->kind == kPruneQKV) { v_hp = e->rv->d_head_ptr; v_id = e->rv->d_row_id; }
    } else if (e->kind == kPruneQKV) {
        if ((rc = tile_linear_run(e->rq->tw, b0, in, T, 0, st))) return rc;
        if ((rc = tile_linear_run(e->rk->tw, b1, in, T, 0, st))) return rc;
        q_pitch = e->rq->nrow; qk_hp = e->rq->d_head_ptr;
    } else {
        if ((rc = tile_linear_run(e->lin[0], b0, in, T, 0, st))) return rc;
        if ((rc = tile_linear_run(e->lin[1], b1, in, T, 0, st))) return rc;
    }
    if (e->qkv) {
    } else if (e->kind == kPrune || e->kind == kPruneQKV) {
        if ((rc = tile_linear_run(e->rv->tw, b2, in, T, 0, st))) return rc;
        v_pitch = e->rv->nrow; v_hp = e->rv->d_head_ptr; v_id = e->rv->d_row_id;
    } else {
        if ((rc = tile_linear_run(e->lin[2], b2, in, T, 0, st))) return rc;
    }
    const half* scores = nullptr;
    if (e->kind == kLength && e->materialize_scores && !cu_seqlens) {
        half* sbuf = scratch + 5 * td;
        if ((rc = qk_scores_launch(sbuf, b0, b1, batch, uniform_len, e->d_model, e->nheads, st, q_pitch))) return rc;
        scores = sbuf;
    }
    if (!e->o_compact && (rc = attention_launch(b3, b0, b1, b2, scores, q_pitch, v_pitch, qk_hp, v_id, v_hp, e->d_mask, e->seq_len,
                               cu_seqlens, valid_lens, batch, uniform_len, T, e->d_model, e->nheads, st, max_len)))
        return rc;
    b1 = scratch + td;
    if ((rc = tile_linear_run(e->o_compact ? e->o_compact : e->lin[3], b0, b3, T, 0, st))) return rc;
    if ((rc = et_skip_layernorm(b0, in, e->d_ln[0], e->d_ln[1], T, e->d_model, st))) return rc;
    if ((rc = tile_linear_run(e->lin[4], b1, b0, T, 1, st))) return rc;
    if ((rc = tile_linear_run(e->lin[5], out, b1, T, 0, st))) return rc;
    return et_skip_layernorm(out, b0, e->d_ln[2], e->d_ln[3], T, e->d_model, st);
}


// ------------------------------------------------------------------------------ stack of layers
// N encoder layers run back to back on packed tokens: the caller's side of the reference's one-layer objects
// (test/tile_test.cu:36-41 calls run() once for one layer). The model owns its scratch (grown on demand, kept
// between calls), uploads the lengths once per call, and replays all N x 7 launches as one CUDA graph.
struct Model {
    std::vector<Encoder*> layers;
    half* scratch = nullptr; size_t scratch_halfs = 0;
    LengthArray lens;
    std::vector<int> meta;
    ReplayCache graphs;
    // LayerNorm folded into the linears (tile and length layers): per layer the FFN1 weight folded with the layer's
    // first LayerNorm, the fused Q|K|V weight folded with the PREVIOUS layer's second LayerNorm, fp32 copies of
    // the four LayerNorm vectors; per row the partial sums that the output projection and FFN2 leave behind.
    struct Fused {
        TileWeight* ffn1 = nullptr;
        TileWeight* qkv = nullptr;
        float* lnf[4] = {nullptr, nullptr, nullptr, nullptr};
        int np1 = 0, np2 = 0;   // partial-sum slots per row of the output projection / of FFN2
    };
    std::vector<Fused> fused;
    bool fuse_ln = false;
    float* stats1 = nullptr; float* stats2 = nullptr; size_t stats_floats = 0;
    void drop_fused() {
        for (auto& f : fused) {
            tile_weight_free(f.ffn1);
            tile_weight_free(f.qkv);
            for (float* p : f.lnf) cudaFree(p);
        }
        fused.clear();
        fuse_ln = false;
    }
    ~Model() {
        graphs.drop();
        drop_fused();
        for (auto* e : layers) delete e;
        cudaFree(scratch);
        cudaFree(stats1);
        cudaFree(stats2);
    }
};

int layernorm_launch(half* x, const half* s, const half* g, const half* b, int num, int size, cudaStream_t st);

// Builds the folded weights. Returns ET_OK with fuse_ln left false when the stack is not eligible (a row-pruned
// layer, or a layer without the fused Q|K|V weight): such stacks run layer by layer with separate LayerNorms.
static int model_prepare_fusion(Model* m) {
    m->drop_fused();
    for (const Encoder* e : m->layers)
        if ((e->kind != kTile && e->kind != kLength) || !e->qkv || (e->d_model & 7)) return ET_OK;
    m->fused.resize(m->layers.size());
    for (size_t l = 0; l < m->layers.size(); ++l) {
        Encoder* e = m->layers[l];
        Model::Fused& f = m->fused[l];
        int rc = tile_weight_prepare_fusion(e->lin[3]);
        if (rc == ET_OK) rc = tile_weight_prepare_fusion(e->lin[5]);
        if (rc == ET_OK) rc = tile_weight_fold(&f.ffn1, e->lin[4], e->h_ln[0].data(), e->h_ln[1].data());
        if (rc == ET_OK && l > 0) {
            const Encoder* pe = m->layers[l - 1];
            rc = tile_weight_fold(&f.qkv, e->qkv, pe->h_ln[2].data(), pe->h_ln[3].data());
        }
        if (rc) { m->drop_fused(); return rc; }
        for (int i = 0; i < 4; ++i) {
            std::vector<float> v(e->d_model);
            for (int k = 0; k < e->d_model; ++k) v[k] = __half2float(e->h_ln[i][k]);
            if (cudaMalloc(&f.lnf[i], v.size() * sizeof(float)) != cudaSuccess) { m->drop_fused(); return fail(ET_ERR_CUDA, "model: cudaMalloc failed"); }
            cudaMemcpy(f.lnf[i], v.data(), v.size() * sizeof(float), cudaMemcpyHostToDevice);
        }
        f.np1 = tile_weight_stat_slots(e->lin[3]);
        f.np2 = tile_weight_stat_slots(e->lin[5]);
    }
    const int rc = cuda_status(cudaDeviceSynchronize(), "model: upload");   // launches on any stream may follow
    if (rc) { m->drop_fused(); return rc; }
    m->fuse_ln = true;
    return ET_OK;
}

// The stack with its LayerNorms folded into the linears. Per layer: fused Q|K|V (normalising its input in the
// epilogue from layer 1 on), attention, output projection + residual -> y1 and its row sums, FFN1 (normalises y1 in
// the epilogue, GELU), FFN2 + LayerNorm(y1) as residual -> y2 and its row sums into `out`; the next layer reads
// `out` un-normalised. One plain LayerNorm of `out` ends the stack. 5 launches per layer instead of 7.
static int model_forward_fused(Model* m, half* out, const half* in, int T, const int* cu, const int* vl, int batch,
                               int uniform_len, cudaStream_t st, int max_len) {
    half* scratch = m->scratch;
    const half* yprev = in;
    int rc;
    for (size_t l = 0; l < m->layers.size(); ++l) {
        Encoder* e = m->layers[l];
        const Model::Fused& f = m->fused[l];
        const int d = e->d_model;
        const size_t td = (size_t)T * d;
        half* b0 = scratch; half* b3 = scratch + 3 * td;
        half* b1 = scratch + td;
        if (l == 0) {
            if ((rc = tile_linear_run(e->qkv, b0, in, T, 0, st))) return rc;
        } else {
            GemmFusion fz;
            fz.mode = 1; fz.stats_in = m->stats2; fz.np_in = m->fused[l - 1].np2;
            if ((rc = tile_linear_run(f.qkv, b0, yprev, T, 0, st, nullptr, &fz))) return rc;
        }
        const half* scores = nullptr;
        if (e->kind == kLength && e->materialize_scores && !cu) {
            half* sbuf = scratch + 5 * td;
            if ((rc = qk_scores_launch(sbuf, b0, b0 + d, batch, uniform_len, d, e->nheads, st, 3 * d))) return rc;
            scores = sbuf;
        }
        if ((rc = attention_launch(b3, b0, b0 + d, b0 + 2 * d, scores, 3 * d, 3 * d, nullptr, nullptr, nullptr, e->d_mask,
                                   e->seq_len, cu, vl, batch, uniform_len, T, d, e->nheads, st, max_len)))
            return rc;
        {   // y1 = Z Wo^T + bo + residual
            GemmFusion fz;
            fz.resid = yprev; fz.stats_out = m->stats1; fz.np_out = f.np1;
            if (l == 0) {
                fz.mode = 2;
            } else {
                const Model::Fused& pf = m->fused[l - 1];
                fz.mode = 3; fz.stats_src = m->stats2; fz.np_src = pf.np2; fz.gamma_s = pf.lnf[2]; fz.beta_s = pf.lnf[3];
            }
            if ((rc = tile_linear_run(e->lin[3], b0, b3, T, 0, st, nullptr, &fz))) return rc;
        }
        {   // F = gelu(LN1(y1) W1^T + b1)
            GemmFusion fz;
            fz.mode = 1; fz.stats_in = m->stats1; fz.np_in = f.np1;
            if ((rc = tile_linear_run(f.ffn1, b1, b0, T, 1, st, nullptr, &fz))) return rc;
        }
        {   // y2 = F W2^T + b2 + LN1(y1)
            GemmFusion fz;
            fz.mode = 3; fz.resid = b0; fz.stats_src = m->stats1; fz.np_src = f.np1; fz.gamma_s = f.lnf[0]; fz.beta_s = f.lnf[1];
            fz.stats_out = m->stats2; fz.np_out = f.np2;
            if ((rc = tile_linear_run(e->lin[5], out, b1, T, 0, st, nullptr, &fz))) return rc;
        }
        yprev = out;
    }
    const Encoder* last = m->layers.back();
    return layernorm_launch(out, nullptr, last->d_ln[2], last->d_ln[3], T, last->d_model, st);
}

static size_t model_scratch_halfs(const Model* m, int total_tokens, int batch, int max_len) {
    size_t need = 0;
    for (const Encoder* e : m->layers) {
        size_t n = (size_t)5 * e->d_model * total_tokens;
        if (e->kind == kLength && e->materialize_scores) n += (size_t)batch * e->nheads * max_len * max_len;
        need = std::max(need, n);
    }
    return need;
}

static int model_forward(Model* m, half* out, const half* in, int T, const int* cu, const int* vl, int batch,
                         int uniform_len, cudaStream_t st, int max_len) {
    if (m->fuse_ln) return model_forward_fused(m, out, in, T, cu, vl, batch, uniform_len, st, max_len);
    const half* x = in;
    for (Encoder* e : m->layers) {
        // a layer may write over its own input (the input is consumed before the last two launches write `out`)
        const int rc = encoder_forward(e, out, x, m->scratch, T, cu, vl, batch, uniform_len, st, max_len);
        if (rc) return rc;
        x = out;
    }
    return ET_OK;
}

}  // namespace et

using et::Encoder;
using et::RowWeight;

struct et_row_weight {
    RowWeight* w;
};
struct et_encoder {
    Encoder* e;
};

extern "C" {

int et_row_weight_create(et_row_weight** out, int in_feat, int out_feat, int size, const void* weight_host,
                         const int* row_id_host, int row_id_size, const void* bias_host, int nhead) {
    ET_REQUIRE(out, "et_row_weight_create: null output");
    *out = nullptr;
    RowWeight* w = nullptr;
    int rc = et::row_weight_create(&w, in_feat, out_feat, size, static_cast<const half*>(weight_host), row_id_host,
                                   row_id_size, static_cast<const half*>(bias_host), nhead);
    if (rc) { delete w; return rc; }
    *out = new et_row_weight{w};
    return ET_OK;
}
int et_row_weight_destroy(et_row_weight* w) {
    if (w) { delete w->w; delete w; }
    return ET_OK;
}
int et_row_linear(const et_row_weight* w, void* out, const void* in, int tokens, void* stream) {
    ET_REQUIRE(w, "et_row_linear: null weight");
    return et::tile_linear_run(w->w->tw, static_cast<half*>(out), static_cast<const half*>(in), tokens, 0,
                               static_cast<cudaStream_t>(stream));
}
// Launcher-level form with a DEVICE-resident dense compact weight [N x K] (N a multiple of 16 as the
// reference pads it). The packed form is built on first use (device-to-host copy, synchronous) and cached
// by weight address; et_tile_spmm_cache_clear() drops these entries too.
int et_row_spmm_bias(void* out, const void* in, const void* weight, const void* bias, int M, int N, int K,
                     void* stream) {
    ET_REQUIRE(out && in && weight && bias, "et_row_spmm_bias: null pointer");
    ET_REQUIRE(N > 0 && K > 0 && N % 16 == 0 && K % 16 == 0, "et_row_spmm_bias: N and K must be positive multiples of 16");
    return et::row_spmm_raw(static_cast<half*>(out), static_cast<const half*>(in), static_cast<const half*>(weight),
                            static_cast<const half*>(bias), M, N, K, static_cast<cudaStream_t>(stream));
}
int et_row_weight_meta(const et_row_weight* w, int* nrow, int* row_id_size, const int** row_id_dev,
                       const int** head_ptr_dev, int* head_ptr_host) {
    ET_REQUIRE(w, "et_row_weight_meta: null weight");
    if (nrow) *nrow = w->w->nrow;
    if (row_id_size) *row_id_size = w->w->row_id_size;
    if (row_id_dev) *row_id_dev = w->w->d_row_id;
    if (head_ptr_dev) *head_ptr_dev = w->w->d_head_ptr;
    if (head_ptr_host) std::copy(w->w->h_head_ptr.begin(), w->w->h_head_ptr.end(), head_ptr_host);
    return ET_OK;
}

int et_attention_otf(void* out, const void* Q, const void* K, const void* V, const void* mask, int seq_len,
                     int d_model, int nhead, void* stream) {
    ET_REQUIRE(seq_len >= 0, "et_attention_otf: negative seq_len");
    return et::attention_launch(static_cast<half*>(out), static_cast<const half*>(Q), static_cast<const half*>(K),
                                static_cast<const half*>(V), nullptr, d_model, d_model, nullptr, nullptr, nullptr,
                                static_cast<const half*>(mask), seq_len, nullptr, nullptr, 1, seq_len, seq_len,
                                d_model, nhead, static_cast<cudaStream_t>(stream));
}
int et_attention_prune(void* out, const void* Q, const void* K, const void* V, const int* v_col_id,
                       const int* v_head_ptr, int nnz_col_v, const void* mask, int seq_len, int d_model,
                       int nhead, void* stream) {
    ET_REQUIRE(seq_len >= 0 && nnz_col_v > 0, "et_attention_prune: bad dimensions");
    ET_REQUIRE(v_col_id && v_head_ptr, "et_attention_prune: null index array");
    return et::attention_launch(static_cast<half*>(out), static_cast<const half*>(Q), static_cast<const half*>(K),
                                static_cast<const half*>(V), nullptr, d_model, nnz_col_v, nullptr, v_col_id,
                                v_head_ptr, static_cast<const half*>(mask), seq_len, nullptr, nullptr, 1, seq_len,
                                seq_len, d_model, nhead, static_cast<cudaStream_t>(stream), 0, nnz_col_v);
}
int et_qk_scores(void* QK, const void* Q, const void* K, int seq_len, int d_model, int nhead, void* stream) {
    return et::qk_scores_launch(static_cast<half*>(QK), static_cast<const half*>(Q), static_cast<const half*>(K), 1,
                                seq_len, d_model, nhead, static_cast<cudaStream_t>(stream));
}
int et_attention_sharedqk(void* out, const void* QK, const void* V, const void* mask, int seq_len, int d_model,
                          int nhead, void* stream) {
    ET_REQUIRE(QK, "et_attention_sharedqk: null scores");
    return et::attention_launch(static_cast<half*>(out), nullptr, nullptr, static_cast<const half*>(V),
                                static_cast<const half*>(QK), d_model, d_model, nullptr, nullptr, nullptr,
                                static_cast<const half*>(mask), seq_len, nullptr, nullptr, 1, seq_len, seq_len,
                                d_model, nhead, static_cast<cudaStream_t>(stream));
}
int et_attention_static_scores(void* out, const void* Q, const void* K, const void* V, const void* mask,
                               int seq_len, int d_model, int nhead, void* stream) {
    ET_REQUIRE(out && Q && K && V, "et_attention_static_scores: null pointer");
    return et::attention_static_scores(static_cast<half*>(out), static_cast<const half*>(Q),
                                       static_cast<const half*>(K), static_cast<const half*>(V),
                                       static_cast<const half*>(mask), seq_len, d_model, nhead,
                                       static_cast<cudaStream_t>(stream));
}
int et_attention_batch(void* out, const void* Q, const void* K, const void* V, int qk_pitch, int v_pitch,
                       const int* qk_head_ptr, const int* v_col_id, const int* v_head_ptr, const void* mask,
                       int mask_ld, const int* cu_seqlens, const int* valid_lens, int batch, int uniform_len,
                       int max_seq_len, int total_tokens, int d_model, int nhead, void* stream) {
    return et::attention_launch(static_cast<half*>(out), static_cast<const half*>(Q), static_cast<const half*>(K),
                                static_cast<const half*>(V), nullptr, qk_pitch, v_pitch, qk_head_ptr, v_col_id,
                                v_head_ptr, static_cast<const half*>(mask), mask_ld, cu_seqlens, valid_lens, batch,
                                uniform_len, total_tokens, d_model, nhead, static_cast<cudaStream_t>(stream),
                                max_seq_len);
}

// ------------------------------------------------------------------------------ encoders
static int take_tiles(Encoder* e, et_tile_weight** t, int first, int count, int d_model) {
    for (int i = 0; i < count; ++i)
        if (!t[i] || !t[i]->w) return et::fail(ET_ERR_INVALID, "encoder: null linear");
    for (int i = 0; i < count; ++i) {
        e->lin[first + i] = t[i]->w;   // ownership moves into the encoder, as the reference's rvalue ctor
        t[i]->w = nullptr;
    }
    (void)d_model;
    return ET_OK;
}

// Lays a row-pruned layer out for compact heads (see Encoder::o_compact): q, k, v are the parts of the fused weight, rows[i] the
// row-pruned linear behind part i or null. Leaves the encoder as it was where the output projection cannot be gathered.
static int compact_heads(Encoder* e, const et::TileWeight* const* dense, RowWeight* const* rows) {
    if (et::tile_weight_in_feat(e->lin[3]) != e->d_model) return et::fail(ET_ERR_INVALID, "encoder: the output projection's in_feat must be d_model");
    et::TileWeight* own[3] = {nullptr, nullptr, nullptr};
    const et::TileWeight* parts[3];
    std::vector<int> ptr[3];
    int rc = ET_OK;
    for (int i = 0; i < 3 && rc == ET_OK; ++i) {
        if (rows[i]) rc = et::row_weight_padded(&own[i], rows[i], et::tile_weight_size(rows[i]->tw), ptr[i]);
        parts[i] = rows[i] ? own[i] : dense[i];
    }
    if (rc == ET_OK) {
        std::vector<int> src((size_t)ptr[2].back(), -1);
        for (int h = 0; h < e->nheads; ++h)
            for (int j = rows[2]->h_head_ptr[h]; j < rows[2]->h_head_ptr[h + 1]; ++j)
                src[ptr[2][h] + j - rows[2]->h_head_ptr[h]] = rows[2]->h_row_id[j];
        rc = et::tile_weight_gather_inputs(&e->o_compact, e->lin[3], src.data(), (int)src.size());
        if (rc == ET_ERR_UNSUPPORTED) {
            for (auto* t : own) et::tile_weight_free(t);
            return ET_OK;
        }
    }
    if (rc == ET_OK) rc = et::tile_weight_concat(&e->qkv, parts, 3, 0);
    auto upload = [](int** d, const std::vector<int>& v) {
        if (cudaMalloc(d, v.size() * sizeof(int)) != cudaSuccess) return et::fail(ET_ERR_CUDA, "encoder: cudaMalloc failed");
        return et::cuda_status(cudaMemcpy(*d, v.data(), v.size() * sizeof(int), cudaMemcpyHostToDevice), "encoder: upload");
    };
    if (rc == ET_OK && rows[0]) rc = upload(&e->d_qk_ptr, ptr[0]);
    if (rc == ET_OK) rc = upload(&e->d_v_ptr, ptr[2]);
    if (rc == ET_OK) rc = et::cuda_status(cudaDeviceSynchronize(), "encoder: upload");
    for (int i = 0; i < 3 && rc == ET_OK; ++i) e->qkv_cols[i] = rows[i] ? ptr[i].back() : e->d_model;
    for (auto* t : own) et::tile_weight_free(t);
    return rc;
}

static int finish_create(et_encoder** out, std::unique_ptr<Encoder>& e) {
    *out = new et_encoder{e.release()};
    return ET_OK;
}

int et_encoder_tile_create(et_encoder** out, int kind, int d_model, int seq_len, int nheads, void* buffer,
                           et_tile_weight* q, et_tile_weight* k, et_tile_weight* v, et_tile_weight* o,
                           et_tile_weight* mlp1, et_tile_weight* mlp2, const void* ln_gamma_1,
                           const void* ln_beta_1, const void* ln_gamma_2, const void* ln_beta_2,
                           const void* mask_host) {
    ET_REQUIRE(out, "et_encoder_tile_create: null output");
    *out = nullptr;
    ET_REQUIRE(kind == et::kTile || kind == et::kLength, "et_encoder_tile_create: kind must be 0 (tile) or 2 (length)");
    auto e = std::make_unique<Encoder>();
    e->kind = kind;
    int rc = et::encoder_common(e.get(), d_model, seq_len, nheads, static_cast<half*>(buffer),
                                static_cast<const half*>(ln_gamma_1), static_cast<const half*>(ln_beta_1),
                                static_cast<const half*>(ln_gamma_2), static_cast<const half*>(ln_beta_2),
                                static_cast<const half*>(mask_host));
    if (rc) return rc;
    et_tile_weight* t[6] = {q, k, v, o, mlp1, mlp2};
    if ((rc = take_tiles(e.get(), t, 0, 6, d_model))) return rc;
    if (et::tile_weight_out_feat(e->lin[0]) == d_model && et::tile_weight_out_feat(e->lin[1]) == d_model &&
        et::tile_weight_out_feat(e->lin[2]) == d_model) {
        const et::TileWeight* parts[3] = {e->lin[0], e->lin[1], e->lin[2]};
        if ((rc = et::tile_weight_concat(&e->qkv, parts, 3, 0))) return rc;
        for (int i = 0; i < 3; ++i) e->qkv_cols[i] = d_model;
    }
    return finish_create(out, e);
}

int et_encoder_prune_create(et_encoder** out, int d_model, int seq_len, int nheads, void* buffer,
                            et_tile_weight* q, et_tile_weight* k, et_row_weight* v, et_tile_weight* o,
                            et_tile_weight* mlp1, et_tile_weight* mlp2, const void* ln_gamma_1,
                            const void* ln_beta_1, const void* ln_gamma_2, const void* ln_beta_2,
                            const void* mask_host) {
    ET_REQUIRE(out, "et_encoder_prune_create: null output");
    *out = nullptr;
    ET_REQUIRE(v && v->w, "et_encoder_prune_create: null V linear");
    auto e = std::make_unique<Encoder>();
    e->kind = et::kPrune;
    int rc = et::encoder_common(e.get(), d_model, seq_len, nheads, static_cast<half*>(buffer),
                                static_cast<const half*>(ln_gamma_1), static_cast<const half*>(ln_beta_1),
                                static_cast<const half*>(ln_gamma_2), static_cast<const half*>(ln_beta_2),
                                static_cast<const half*>(mask_host));
    if (rc) return rc;
    et_tile_weight* t01[2] = {q, k};
    et_tile_weight* t35[3] = {o, mlp1, mlp2};
    if ((rc = take_tiles(e.get(), t01, 0, 2, d_model))) return rc;
    if ((rc = take_tiles(e.get(), t35, 3, 3, d_model))) return rc;
    e->rv = v->w; v->w = nullptr;
    if (et::tile_weight_out_feat(e->lin[0]) == d_model && et::tile_weight_out_feat(e->lin[1]) == d_model &&
        e->rv->in_feat == d_model) {
        // Q | K | compact V in one launch
        const et::TileWeight* parts[3] = {e->lin[0], e->lin[1], e->rv->tw};
        if (d_model == 64 * nheads && e->rv->out_feat == d_model && e->rv->nhead == nheads) {
            RowWeight* const rows[3] = {nullptr, nullptr, e->rv};
            if ((rc = compact_heads(e.get(), parts, rows))) return rc;
            if (e->o_compact) return finish_create(out, e);
        }
        if ((rc = et::tile_weight_concat(&e->qkv, parts, 3, 0))) return rc;
        e->qkv_cols[0] = e->qkv_cols[1] = d_model;
        e->qkv_cols[2] = e->rv->nrow;
    }
    return finish_create(out, e);
}

int et_encoder_prune_qkv_create(et_encoder** out, int d_model, int seq_len, int nheads, void* buffer,
                                et_row_weight* q, et_row_weight* k, et_row_weight* v, et_tile_weight* o,
                                et_tile_weight* mlp1, et_tile_weight* mlp2, const void* ln_gamma_1,
                                const void* ln_beta_1, const void* ln_gamma_2, const void* ln_beta_2,
                                const void* mask_host) {
    ET_REQUIRE(out, "et_encoder_prune_qkv_create: null output");
    *out = nullptr;
    ET_REQUIRE(q && q->w && k && k->w && v && v->w, "et_encoder_prune_qkv_create: null linear");
    ET_REQUIRE(q->w->row_id_size == k->w->row_id_size && q->w->h_head_ptr == k->w->h_head_ptr,
               "et_encoder_prune_qkv_create: Q and K must retain the same dimensions per head");
    auto e = std::make_unique<Encoder>();
    e->kind = et::kPruneQKV;
    int rc = et::encoder_common(e.get(), d_model, seq_len, nheads, static_cast<half*>(buffer),
                                static_cast<const half*>(ln_gamma_1), static_cast<const half*>(ln_beta_1),
                                static_cast<const half*>(ln_gamma_2), static_cast<const half*>(ln_beta_2),
                                static_cast<const half*>(mask_host));
    if (rc) return rc;
    et_tile_weight* t35[3] = {o, mlp1, mlp2};
    if ((rc = take_tiles(e.get(), t35, 3, 3, d_model))) return rc;
    e->rq = q->w; q->w = nullptr;
    e->rk = k->w; k->w = nullptr;
    e->rv = v->w; v->w = nullptr;
    if (e->rq->in_feat == d_model && e->rk->in_feat == d_model && e->rv->in_feat == d_model && d_model == 64 * nheads &&
        e->rq->out_feat == d_model && e->rk->out_feat == d_model && e->rv->out_feat == d_model && e->rq->nhead == nheads &&
        e->rk->nhead == nheads && e->rv->nhead == nheads) {
        RowWeight* const rows[3] = {e->rq, e->rk, e->rv};
        if ((rc = compact_heads(e.get(), nullptr, rows))) return rc;
        if (e->o_compact) return finish_create(out, e);
    }
    if (e->rq->in_feat == d_model && e->rk->in_feat == d_model && e->rv->in_feat == d_model &&
        e->rq->nrow + e->rk->nrow + e->rv->nrow <= 3 * d_model) {
        // compact Q | K | V in one launch
        const et::TileWeight* parts[3] = {e->rq->tw, e->rk->tw, e->rv->tw};
        if ((rc = et::tile_weight_concat(&e->qkv, parts, 3, 0))) return rc;
        e->qkv_cols[0] = e->rq->nrow; e->qkv_cols[1] = e->rk->nrow; e->qkv_cols[2] = e->rv->nrow;
    }
    return finish_create(out, e);
}

int et_encoder_destroy(et_encoder* enc) {
    if (enc) { delete enc->e; delete enc; }
    return ET_OK;
}

int et_encoder_set_materialize_scores(et_encoder* enc, int on) {
    ET_REQUIRE(enc && enc->e, "et_encoder_set_materialize_scores: null encoder");
    ET_REQUIRE(enc->e->kind == et::kLength, "et_encoder_set_materialize_scores: only the length encoder has that path");
    enc->e->materialize_scores = on != 0;
    return ET_OK;
}

size_t et_encoder_buffer_size(int kind, int d_model, int seq_len, int nheads) {
    size_t n = (size_t)5 * d_model * seq_len;
    if (kind == et::kLength) n += (size_t)nheads * seq_len * seq_len;
    return n * sizeof(half);
}

size_t et_encoder_batch_buffer_size(int kind, int d_model, int total_tokens, int batch, int max_len, int nheads) {
    size_t n = (size_t)5 * d_model * total_tokens;
    if (kind == et::kLength) n += (size_t)batch * nheads * max_len * max_len;
    return n * sizeof(half);
}

// Whether the stream is inside a capture of the caller's (or its state cannot be told): no graph of our own then.
static bool in_capture(cudaStream_t st) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    return cudaStreamIsCapturing(st, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone;
}

int et_encoder_run(et_encoder* enc, void* out, const void* in, void* stream) {
    ET_REQUIRE(enc && enc->e && out && in, "et_encoder_run: null pointer");
    Encoder* e = enc->e;
    ET_REQUIRE(e->buffer, "et_encoder_run: the encoder was created without a scratch buffer");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    auto forward = [&](cudaStream_t s) {
        return et::encoder_forward(e, static_cast<half*>(out), static_cast<const half*>(in), e->buffer, e->seq_len, nullptr,
                                   nullptr, 1, e->seq_len, s);
    };
    if (!e->graphs.on || in_capture(st)) return forward(st);
    e->graphs.key.assign({(int64_t)(intptr_t)out, (int64_t)(intptr_t)in, -1, (int64_t)e->materialize_scores});
    return e->graphs.run(st, "et_encoder_run: graph launch", forward);
}

int et_encoder_run_batch(et_encoder* enc, void* out, const void* in, const int* seq_lens_host,
                         const int* valid_lens_host, int batch, void* scratch, size_t scratch_bytes, void* stream) {
    ET_REQUIRE(enc && enc->e && out && in && scratch, "et_encoder_run_batch: null pointer");
    ET_REQUIRE(batch >= 0, "et_encoder_run_batch: negative batch");
    Encoder* e = enc->e;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (batch == 0) return ET_OK;
    ET_REQUIRE(seq_lens_host, "et_encoder_run_batch: null seq_lens");
    // The call's own: with equal lengths and without graph replay a layer may be run by several threads at once, each with its
    // own stream and buffers.
    std::vector<int> meta(2 * (size_t)batch + 1);
    meta[0] = 0;
    bool uniform = true;
    int max_len = 0;
    for (int b = 0; b < batch; ++b) {
        ET_REQUIRE(seq_lens_host[b] >= 0, "et_encoder_run_batch: negative sequence length");
        ET_REQUIRE(!e->d_mask || seq_lens_host[b] <= e->seq_len, "et_encoder_run_batch: sequence longer than the mask");
        meta[b + 1] = meta[b] + seq_lens_host[b];
        meta[batch + 1 + b] = valid_lens_host ? valid_lens_host[b] : seq_lens_host[b];
        uniform = uniform && seq_lens_host[b] == seq_lens_host[0];
        max_len = std::max(max_len, seq_lens_host[b]);
    }
    const int T = meta[batch];
    if (T == 0) return ET_OK;
    const bool scores = e->kind == et::kLength && e->materialize_scores && uniform;
    size_t need = (size_t)5 * e->d_model * T;
    if (scores) need += (size_t)batch * e->nheads * max_len * max_len;
    ET_REQUIRE(scratch_bytes >= need * sizeof(half), "et_encoder_run_batch: scratch buffer too small");
    const int* cu = nullptr;
    const int* vl = nullptr;
    const bool capturing = in_capture(st);
    if (!uniform || valid_lens_host) {
        const int* lens = nullptr;
        const int rc = capturing ? e->lens.in_capture(meta, &lens, "et_encoder_run_batch: lengths upload")
                                 : e->lens.upload(meta, st, e->graphs, "et_encoder_run_batch: lengths upload");
        if (rc) return rc;
        if (!capturing) lens = e->lens.d;
        if (!uniform) cu = lens;
        if (valid_lens_host) vl = lens + batch + 1;
    }
    auto forward = [&](cudaStream_t s) {
        return et::encoder_forward(e, static_cast<half*>(out), static_cast<const half*>(in), static_cast<half*>(scratch), T, cu, vl,
                                   batch, uniform ? seq_lens_host[0] : 0, s, max_len);
    };
    if (!e->graphs.on || capturing) return forward(st);
    std::vector<int64_t>& key = e->graphs.key;
    key.assign({(int64_t)(intptr_t)out, (int64_t)(intptr_t)in, (int64_t)(intptr_t)scratch, (int64_t)batch,
                (int64_t)(valid_lens_host != nullptr), (int64_t)e->materialize_scores, (int64_t)(intptr_t)e->lens.d});
    key.insert(key.end(), meta.begin(), meta.end());
    return e->graphs.run(st, "et_encoder_run_batch: graph launch", forward);
}

// Reads and clears the error words of every kernel the layer launches: the tile GEMMs' (one per owned weight) and
// the current device's attention word. Synchronises.
static int encoder_check(Encoder* e, int* code) {
    std::vector<et::TileWeight*> ws(e->lin, e->lin + 6);
    ws.push_back(e->qkv);
    ws.push_back(e->o_compact);
    for (RowWeight* r : {e->rq, e->rk, e->rv})
        if (r) ws.push_back(r->tw);
    for (et::TileWeight* w : ws) {
        if (!w) continue;
        int c = 0;
        const int rc = et::tile_weight_error(w, &c);
        if (rc) return rc;
        if (c && !*code) *code = c;
    }
    int c = 0;
    const int rc = et::attention_tc_error(&c);
    if (rc) return rc;
    if (c && !*code) *code = c;
    return ET_OK;
}

int et_encoder_check(et_encoder* enc, int* code) {
    ET_REQUIRE(enc && enc->e && code, "et_encoder_check: null pointer");
    *code = 0;
    const int rc = encoder_check(enc->e, code);
    if (rc) return rc;
    if (*code) {
        et::set_error("encoder layer: device wait %d gave up", *code);
        return ET_ERR_DEVICE_TIMEOUT;
    }
    return ET_OK;
}

int et_attention_check(int* code) {
    ET_REQUIRE(code, "et_attention_check: null pointer");
    const int rc = et::attention_tc_error(code);
    if (rc) return rc;
    if (*code) {
        et::set_error("attention: device wait %d gave up", *code);
        return ET_ERR_DEVICE_TIMEOUT;
    }
    return ET_OK;
}

int et_encoder_set_graph_replay(et_encoder* enc, int on) {
    ET_REQUIRE(enc && enc->e, "et_encoder_set_graph_replay: null encoder");
    enc->e->graphs.on = on != 0;
    return ET_OK;
}


struct et_model {
    et::Model* m;
};

int et_model_create(et_model** out, et_encoder* const* layers, int n_layers) {
    ET_REQUIRE(out, "et_model_create: null output");
    *out = nullptr;
    ET_REQUIRE(layers && n_layers > 0, "et_model_create: no layers");
    for (int i = 0; i < n_layers; ++i) {
        ET_REQUIRE(layers[i] && layers[i]->e, "et_model_create: null or already consumed layer");
        ET_REQUIRE(layers[i]->e->d_model == layers[0]->e->d_model, "et_model_create: layers differ in d_model");
        for (int j = 0; j < i; ++j) ET_REQUIRE(layers[i] != layers[j], "et_model_create: the same layer twice");
    }
    auto* m = new et::Model();
    for (int i = 0; i < n_layers; ++i) {
        m->layers.push_back(layers[i]->e);
        layers[i]->e = nullptr;   // ownership moves to the model; the caller still destroys the emptied handles
    }
    *out = new et_model{m};
    return ET_OK;
}

int et_model_set_layernorm_fusion(et_model* model, int on) {
    ET_REQUIRE(model && model->m, "et_model_set_layernorm_fusion: null model");
    et::Model* m = model->m;
    m->graphs.drop();
    if (!on) { m->drop_fused(); return ET_OK; }
    return et::model_prepare_fusion(m);
}

int et_model_layernorm_fused(const et_model* model) { return model && model->m && model->m->fuse_ln ? 1 : 0; }

int et_model_destroy(et_model* model) {
    if (model) { delete model->m; delete model; }
    return ET_OK;
}

int et_model_num_layers(const et_model* model) { return model && model->m ? (int)model->m->layers.size() : 0; }

int et_model_check(et_model* model, int* code) {
    ET_REQUIRE(model && model->m && code, "et_model_check: null pointer");
    *code = 0;
    for (Encoder* e : model->m->layers) {
        const int rc = encoder_check(e, code);
        if (rc) return rc;
    }
    for (const auto& f : model->m->fused)
        for (et::TileWeight* w : {f.ffn1, f.qkv}) {
            if (!w) continue;
            int c = 0;
            const int rc = et::tile_weight_error(w, &c);
            if (rc) return rc;
            if (c && !*code) *code = c;
        }
    if (*code) {
        et::set_error("layer stack: device wait %d gave up", *code);
        return ET_ERR_DEVICE_TIMEOUT;
    }
    return ET_OK;
}

int et_model_set_graph_replay(et_model* model, int on) {
    ET_REQUIRE(model && model->m, "et_model_set_graph_replay: null model");
    model->m->graphs.on = on != 0;
    return ET_OK;
}

// Grows the model's scratch to hold a batch of `total_tokens` packed tokens (and, for length layers that
// materialise scores, batch x heads x max_len^2 scores). Graphs recorded with the old scratch are dropped.
int et_model_reserve(et_model* model, int total_tokens, int batch, int max_len) {
    ET_REQUIRE(model && model->m, "et_model_reserve: null model");
    ET_REQUIRE(total_tokens >= 0 && batch >= 0 && max_len >= 0, "et_model_reserve: negative size");
    et::Model* m = model->m;
    const size_t need = et::model_scratch_halfs(m, total_tokens, batch, max_len);
    size_t need_stats = 0;
    for (const auto& f : m->fused) need_stats = std::max(need_stats, (size_t)total_tokens * std::max(f.np1, f.np2) * 2);
    if (need > m->scratch_halfs) {
        m->graphs.drop();
        cudaFree(m->scratch);
        m->scratch = nullptr; m->scratch_halfs = 0;
        if (cudaMalloc(&m->scratch, need * sizeof(half)) != cudaSuccess) return et::fail(ET_ERR_CUDA, "et_model_reserve: cudaMalloc failed");
        m->scratch_halfs = need;
    }
    if (need_stats > m->stats_floats) {
        m->graphs.drop();
        cudaFree(m->stats1); cudaFree(m->stats2);
        m->stats1 = m->stats2 = nullptr; m->stats_floats = 0;
        if (cudaMalloc(&m->stats1, need_stats * sizeof(float)) != cudaSuccess || cudaMalloc(&m->stats2, need_stats * sizeof(float)) != cudaSuccess)
            return et::fail(ET_ERR_CUDA, "et_model_reserve: cudaMalloc failed");
        m->stats_floats = need_stats;
    }
    return ET_OK;
}

int et_model_run_batch(et_model* model, void* out, const void* in, const int* seq_lens_host,
                       const int* valid_lens_host, int batch, void* stream) {
    ET_REQUIRE(model && model->m && out && in, "et_model_run_batch: null pointer");
    ET_REQUIRE(batch >= 0, "et_model_run_batch: negative batch");
    et::Model* m = model->m;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (batch == 0) return ET_OK;
    ET_REQUIRE(seq_lens_host, "et_model_run_batch: null seq_lens");
    std::vector<int>& meta = m->meta;
    meta.resize(2 * (size_t)batch + 1);
    meta[0] = 0;
    bool uniform = true;
    int max_len = 0;
    for (int b = 0; b < batch; ++b) {
        ET_REQUIRE(seq_lens_host[b] >= 0, "et_model_run_batch: negative sequence length");
        for (Encoder* e : m->layers)
            ET_REQUIRE(!e->d_mask || seq_lens_host[b] <= e->seq_len, "et_model_run_batch: sequence longer than a layer's mask");
        meta[b + 1] = meta[b] + seq_lens_host[b];
        meta[batch + 1 + b] = valid_lens_host ? valid_lens_host[b] : seq_lens_host[b];
        uniform = uniform && seq_lens_host[b] == seq_lens_host[0];
        max_len = std::max(max_len, seq_lens_host[b]);
    }
    const int T = meta[batch];
    if (T == 0) return ET_OK;
    const bool capturing = in_capture(st);
    if (capturing) {
        // inside the caller's own capture nothing may be allocated or uploaded from a temporary
        size_t need_stats = 0;
        for (const auto& f : m->fused) need_stats = std::max(need_stats, (size_t)T * std::max(f.np1, f.np2) * 2);
        ET_REQUIRE(et::model_scratch_halfs(m, T, batch, max_len) <= m->scratch_halfs && need_stats <= m->stats_floats,
                   "et_model_run_batch: call et_model_reserve before capturing");
        ET_REQUIRE(uniform && !valid_lens_host, "et_model_run_batch: only equal-length batches can run inside the caller's capture");
    } else {
        int rc = et_model_reserve(model, T, batch, max_len);
        if (rc) return rc;
    }
    const int* cu = nullptr;
    const int* vl = nullptr;
    if (!uniform || valid_lens_host) {
        const int rc = m->lens.upload(meta, st, m->graphs, "et_model_run_batch: lengths upload");
        if (rc) return rc;
        if (!uniform) cu = m->lens.d;
        if (valid_lens_host) vl = m->lens.d + batch + 1;
    }
    auto forward = [&](cudaStream_t s) {
        return et::model_forward(m, static_cast<half*>(out), static_cast<const half*>(in), T, cu, vl, batch,
                                 uniform ? seq_lens_host[0] : 0, s, max_len);
    };
    if (!m->graphs.on || capturing) return forward(st);
    std::vector<int64_t>& key = m->graphs.key;
    key.assign({(int64_t)(intptr_t)out, (int64_t)(intptr_t)in, (int64_t)batch, (int64_t)(valid_lens_host != nullptr),
                (int64_t)(intptr_t)m->lens.d});
    for (Encoder* e : m->layers) key.push_back((int64_t)e->materialize_scores);
    key.insert(key.end(), meta.begin(), meta.end());
    return m->graphs.run(st, "et_model_run_batch: graph launch", forward);
}

}  // extern "C"
