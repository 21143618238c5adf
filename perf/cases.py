"""The work that users of this library have it do, as measurable cases.

A case is a dict of plain values with a "path":
  layer      one encoder layer (tile-pruned, or with row-pruned V / Q, K and V) over a batch of packed sequences
  model      a stack of layers over packed sequences of different lengths
  tile       a tile-pruned linear by itself          row        a row-pruned linear by itself
  attention  the attention operators                 softmax    mask + softmax over score matrices in memory
  layernorm  residual add + LayerNorm in place

Shapes are the BERT-base and BERT-large shapes of the benchmark and the tests (hidden 768 or 1024, heads of 64, FFN four
times the hidden size, 16 x 16 tile sparsity 0 to 0.9, sequences of up to 512 tokens of any length). Activations are
~N(0,1), kept weights ~N(0,0.02), as everywhere in this repository.
"""
import random

import numpy as np
import torch

import et_b200 as et

SHAPES = {768: (12, 3072), 1024: (16, 4096)}   # hidden size: heads, FFN size
KINDS = {"tile": et.KIND_TILE, "length": et.KIND_LENGTH, "prune": et.KIND_PRUNE, "prune_qkv": et.KIND_PRUNE_QKV}


def listed():
    return [
        # the smallest call: one sentence through one unpruned layer, by the one-sequence entry point
        {"name": "layer dense 1x128", "path": "layer", "kind": "tile", "d": 768, "sparsity": 0.0, "batch": 1, "lo": 128, "hi": 128, "call": "run"},
        # a batch of short sentences through a tile-pruned layer
        {"name": "layer tile 16x128", "path": "layer", "kind": "tile", "d": 768, "sparsity": 0.75, "batch": 16, "lo": 128, "hi": 128, "call": "batch"},
        # attention-aware pruning: Q, K and V keep half of every head, the other linears are tile-pruned
        {"name": "layer prune 32x256", "path": "layer", "kind": "prune_qkv", "d": 768, "sparsity": 0.75, "batch": 32, "lo": 256, "hi": 256, "call": "batch"},
        # serving: a stack of layers, sentences of any length packed without padding
        {"name": "model length 12x64", "path": "model", "kind": "length", "d": 768, "layers": 12, "sparsity": 0.75, "batch": 64, "lo": 32, "hi": 512},
        # the largest: offline encoding with the large shapes
        {"name": "model large 24x256x512", "path": "model", "kind": "tile", "d": 1024, "layers": 24, "sparsity": 0.8, "batch": 256, "lo": 512, "hi": 512},
        # the first FFN linear of a half-pruned layer, with GELU, on an odd number of tokens
        {"name": "tile linear gelu 1100", "path": "tile", "tokens": 1100, "k": 768, "n": 3072, "sparsity": 0.5, "gelu": True},
        # the second FFN linear, long reduction, moderate batch
        {"name": "tile linear 8192", "path": "tile", "tokens": 8192, "k": 4096, "n": 1024, "sparsity": 0.8, "gelu": False},
        # a row-pruned projection that keeps half of its outputs
        {"name": "row linear 8192", "path": "row", "tokens": 8192, "k": 768, "n": 768, "keep": 0.5},
        # one document of odd length with an additive mask
        {"name": "attention mask 1x384", "path": "attention", "variant": "otf", "d": 768, "batch": 1, "lo": 384, "hi": 384, "mask": True, "fp32": False},
        # a ragged batch through the batched operator
        {"name": "attention ragged 64", "path": "attention", "variant": "batch", "d": 768, "batch": 64, "lo": 32, "hi": 512, "mask": False, "fp32": False},
        # score matrices of a length that is no multiple of 8, with the mask that they share
        {"name": "softmax 128x500", "path": "softmax", "matrices": 128, "length": 500, "mask": True},
        # the LayerNorm between two linears over the tokens of a ragged batch
        {"name": "layernorm 17771x768", "path": "layernorm", "rows": 17771, "d": 768},
    ]


def _between(rng, lo, hi):
    """Log-uniform whole number in [lo, hi]."""
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def _lengths_range(rng):
    """Equal lengths or a range of lengths, any length up to 512."""
    hi = _between(rng, 32, 512)
    return (hi, hi) if rng.random() < 0.5 else (max(16, hi // _between(rng, 2, 16)), hi)


def draw(rng):
    path = rng.choice(["layer", "layer", "layer", "model", "model", "tile", "tile", "row", "attention", "attention", "softmax", "layernorm"])
    d = rng.choice([768, 768, 1024])
    sparsity = rng.choice([0.0, 0.5, 0.75, 0.75, 0.8, 0.9])
    if path == "layer":
        lo, hi = _lengths_range(rng)
        kind = rng.choice(["tile", "tile", "length", "prune", "prune_qkv"])
        batch = _between(rng, 1, 64)
        call = "batch"
        if batch == 1:
            lo, call = hi, rng.choice(["run", "batch"])
        return {"path": path, "kind": kind, "d": d, "sparsity": sparsity, "batch": batch, "lo": lo, "hi": hi, "call": call}
    if path == "model":
        lo, hi = _lengths_range(rng)
        return {"path": path, "kind": rng.choice(["tile", "length", "prune_qkv"]), "d": d, "layers": _between(rng, 2, 12),
                "sparsity": rng.choice([0.5, 0.75, 0.8, 0.9]), "batch": _between(rng, 2, 128), "lo": lo, "hi": hi}
    if path == "tile":
        k, n = rng.choice([(d, d), (d, 3 * d), (d, 4 * d), (4 * d, d)])
        return {"path": path, "tokens": _between(rng, 64, 65536), "k": k, "n": n, "sparsity": sparsity, "gelu": n == 4 * d}
    if path == "row":
        return {"path": path, "tokens": _between(rng, 64, 65536), "k": d, "n": d, "keep": rng.choice([0.25, 0.5, 0.75])}
    if path == "attention":
        variant = rng.choice(["otf", "batch", "batch", "prune"])
        if variant == "batch":
            lo, hi = _lengths_range(rng)
            return {"path": path, "variant": variant, "d": d, "batch": _between(rng, 2, 128), "lo": lo, "hi": hi,
                    "mask": rng.random() < 0.25, "fp32": rng.random() < 0.25}
        length = _between(rng, 32, 1024)
        return {"path": path, "variant": variant, "d": d, "batch": 1, "lo": length, "hi": length, "mask": rng.random() < 0.5, "fp32": False}
    if path == "softmax":
        return {"path": path, "matrices": _between(rng, 12, 512), "length": _between(rng, 32, 512), "mask": rng.random() < 0.5}
    return {"path": path, "rows": _between(rng, 64, 131072), "d": d}


# ------------------------------------------------------------------------------------------------ inputs
def _lengths(case):
    """The batch's sequence lengths: part of the case, as the work depends on them."""
    rng = random.Random(case["batch"] * 1000003 + case["lo"] * 1009 + case["hi"])
    return [rng.randint(case["lo"], case["hi"]) for _ in range(case["batch"])]


class _Source:
    """Seeded normal values, made on the GPU."""

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda").manual_seed(seed)
        self.count = seed * 1000

    def normal(self, shape, std=1.0, mean=0.0):
        return (torch.randn(shape, generator=self.gen, device="cuda") * std + mean).half()

    def host(self, shape, std=1.0, mean=0.0):
        return self.normal(shape, std, mean).cpu().numpy()

    def next_seed(self):
        self.count += 1
        return self.count


def _tile_weight(src, k, n, sparsity, tokens, gelu=False):
    row_ptr, row_offset = et.gen_sparse_tile_mat(n, k, sparsity, src.next_seed(), bernoulli=True)
    return et.TileWeight(k, n, tokens, src.host((len(row_offset), 256), 0.02), row_ptr, row_offset, src.host((n,), 0.02), is_gelu=gelu)


def _row_ids(src, n, keep, heads):
    return et.gen_sparse_row_mat(n, 1.0 - keep, src.next_seed(), heads)


def _row_weight(src, k, n, ids, heads, tokens):
    return et.RowWeight(k, n, tokens, src.host((len(ids), k), 0.02), ids, src.host((len(ids),), 0.02), heads)


def _layer(src, case, tokens, max_len, buffer):
    d = case["d"]
    heads, ff = SHAPES[d]
    kind = case["kind"]
    ids = _row_ids(src, d, 0.5, heads) if kind.startswith("prune") else None
    q, k, v = (_row_weight(src, d, d, ids, heads, tokens) if kind == "prune_qkv" or (kind == "prune" and name == "v")
               else _tile_weight(src, d, d, case["sparsity"], tokens) for name in "qkv")
    o = _tile_weight(src, d, d, case["sparsity"], tokens)
    mlp1 = _tile_weight(src, d, ff, case["sparsity"], tokens, gelu=True)
    mlp2 = _tile_weight(src, ff, d, case["sparsity"], tokens)
    ln = (src.host((d,), 0.1, 1.0), src.host((d,), 0.1), src.host((d,), 0.1, 1.0), src.host((d,), 0.1))
    return et.Encoder(KINDS[kind], d, max_len, heads, buffer, q, k, v, o, mlp1, mlp2, ln)


def prepare(case, seed):
    src = _Source(seed)
    path = case["path"]
    s = {"case": case}
    if path in ("layer", "model"):
        d = case["d"]
        lens = _lengths(case)
        tokens, longest = sum(lens), max(lens)
        s["lens"] = lens
        s["x"] = src.normal((tokens, d))
        s["out"] = torch.empty_like(s["x"])
        if path == "layer":
            size = et.encoder_batch_buffer_size(KINDS[case["kind"]], d, tokens, len(lens), longest, SHAPES[d][0])
            s["scratch"] = torch.empty(size // 2, dtype=torch.float16, device="cuda")
            s["layer"] = _layer(src, case, tokens, longest, s["scratch"])
        else:
            s["model"] = et.Model([_layer(src, case, tokens, longest, None) for _ in range(case["layers"])])
            s["model"].reserve(tokens, len(lens), longest)
    elif path == "tile":
        s["w"] = _tile_weight(src, case["k"], case["n"], case["sparsity"], case["tokens"], case["gelu"])
        s["x"] = src.normal((case["tokens"], case["k"]))
        s["out"] = torch.empty((case["tokens"], case["n"]), dtype=torch.float16, device="cuda")
    elif path == "row":
        heads = SHAPES[case["n"]][0]
        s["w"] = _row_weight(src, case["k"], case["n"], _row_ids(src, case["n"], case["keep"], heads), heads, case["tokens"])
        s["x"] = src.normal((case["tokens"], case["k"]))
        s["out"] = torch.empty((case["tokens"], s["w"].nrow), dtype=torch.float16, device="cuda")
    elif path == "attention":
        d, heads = case["d"], SHAPES[case["d"]][0]
        lens = _lengths(case)
        tokens, longest = sum(lens), max(lens)
        et.set_attention_scores_fp32(case["fp32"])
        s["q"], s["k"] = src.normal((tokens, d)), src.normal((tokens, d))
        if case["variant"] == "prune":
            ids = _row_ids(src, d, 0.5, heads)
            s["nnz"] = len(ids)
            s["ids"] = torch.from_numpy(ids).cuda()
            s["head_ptr"] = torch.from_numpy(et.build_head_ptr(ids, heads, d)).cuda()
            s["v"] = src.normal((tokens, len(ids)))
        else:
            s["v"] = src.normal((tokens, d))
        s["mask"] = src.normal((longest, longest)) if case["mask"] else None
        s["out"] = torch.empty((tokens, d), dtype=torch.float16, device="cuda")
        s["longest"] = longest
        s["cu"] = torch.tensor(np.concatenate([[0], np.cumsum(lens)]), dtype=torch.int32, device="cuda")
    elif path == "softmax":
        n, length = case["matrices"], case["length"]
        s["scores"] = src.normal((n, length, length))
        s["mask"] = src.normal((length, length)) if case["mask"] else None
    else:
        rows, d = case["rows"], case["d"]
        s["x"], s["skip"] = src.normal((rows, d)), src.normal((rows, d))
        s["gamma"], s["beta"] = src.normal((d,), 0.1, 1.0), src.normal((d,), 0.1)
    return s


def run(s):
    case = s["case"]
    path = case["path"]
    if path == "layer":
        if case["call"] == "run":
            return s["layer"].run(s["out"], s["x"])
        return s["layer"].run_batch(s["out"], s["x"], s["lens"], s["scratch"])
    if path == "model":
        return s["model"].run_batch(s["out"], s["x"], s["lens"])
    if path in ("tile", "row"):
        return s["w"].run(s["out"], s["x"])
    if path == "attention":
        d, heads = case["d"], SHAPES[case["d"]][0]
        if case["variant"] == "batch":
            return et.attention_batch(s["out"], s["q"], s["k"], s["v"], d, heads, cu_seqlens=s["cu"], batch=case["batch"],
                                      max_seq_len=s["longest"], mask=s["mask"], mask_ld=s["longest"] if case["mask"] else 0)
        if case["variant"] == "prune":
            return et.attention_prune(s["out"], s["q"], s["k"], s["v"], s["ids"], s["head_ptr"], s["nnz"], s["mask"], s["longest"], d, heads)
        return et.attention_otf(s["out"], s["q"], s["k"], s["v"], s["mask"], s["longest"], d, heads)
    if path == "softmax":
        return et.softmax_mask(s["scores"], s["mask"])
    return et.skip_layernorm(s["x"], s["skip"], s["gamma"], s["beta"])


# ------------------------------------------------------------------------------------------------ what a pass needs
def _linear(tokens, k, n, density):
    """(weight bytes, operations) of a linear that keeps `density` of its weight."""
    return 2.0 * k * n * density, 2.0 * tokens * k * n * density


def work(case):
    path = case["path"]
    if path in ("layer", "model"):
        d = case["d"]
        ff = SHAPES[d][1]
        lens = _lengths(case)
        tokens = sum(lens)
        keep = 1.0 - case["sparsity"]
        rows = {"prune": ("v",), "prune_qkv": ("q", "k", "v")}.get(case["kind"], ())
        parts = [_linear(tokens, d, d, 0.5 if name in rows else keep) for name in "qkv"]
        parts += [_linear(tokens, d, d, keep), _linear(tokens, d, ff, keep), _linear(tokens, ff, d, keep)]
        pairs = float(sum(n * n for n in lens))
        attention = pairs * d * sum(2.0 * (0.5 if part in rows else 1.0) for part in ("q", "v"))
        layers = case.get("layers", 1)
        return {"bytes": layers * sum(b for b, _ in parts) + 4.0 * tokens * d,
                "flops": layers * (sum(f for _, f in parts) + attention)}
    if path in ("tile", "row"):
        density = 1.0 - case["sparsity"] if path == "tile" else 1.0
        n = case["n"] if path == "tile" else case["n"] * case["keep"]
        weight, flops = _linear(case["tokens"], case["k"], n, density)
        return {"bytes": weight + 2.0 * case["tokens"] * (case["k"] + n), "flops": flops}
    if path == "attention":
        d, lens = case["d"], _lengths(case)
        v = 0.5 if case["variant"] == "prune" else 1.0
        mask = 2.0 * max(lens) ** 2 if case["mask"] else 0.0
        return {"bytes": 2.0 * sum(lens) * d * (3.0 + v) + mask, "flops": 2.0 * sum(n * n for n in lens) * d * (1.0 + v)}
    if path == "softmax":
        n, length = case["matrices"], case["length"]
        return {"bytes": 4.0 * n * length * length + (2.0 * length * length if case["mask"] else 0.0), "flops": 5.0 * n * length * length}
    return {"bytes": 6.0 * case["rows"] * case["d"], "flops": 8.0 * case["rows"] * case["d"]}


def tolerance(case):
    """fp16 in and out (one rounding: 2^-11 at most, 3e-4 in the mean), fp32 sums; attention keeps its probabilities, and by
    default its scores, in fp16; a stack of layers rounds seven times a layer."""
    path = case["path"]
    if path == "model":
        return {"rel": 6e-3}
    if path in ("layer", "attention"):
        return {"rel": 3e-3}
    if path == "tile" and case["gelu"]:
        return {"rel": 2e-3}
    return {"rel": 1e-3}
