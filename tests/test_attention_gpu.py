"""GPU parity tests of the attention family and the row-pruned linear against the CPU oracle."""
import ctypes

import numpy as np
import pytest

from tests import util

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def host(t):
    return t.float().cpu().numpy()


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.fixture(scope="module")
def et():
    import et_b200
    et_b200.lib()
    return et_b200


def _qkv(seed, T, d, std=1.0):
    return [(util.activations(seed + i, (T, d)).astype(np.float32) * std).astype(np.float16) for i in range(3)]


@pytest.mark.parametrize("L,d,H,use_mask", [(128, 768, 12, False), (128, 768, 12, True), (256, 768, 12, True),
                                            (512, 1024, 16, False), (16, 128, 2, True), (77, 768, 12, True),
                                            (1, 64, 1, False), (200, 256, 8, False), (2048, 128, 2, False),
                                            (1100, 128, 2, True)])
def test_attention_otf(et, orc, L, d, H, use_mask):
    Q, K, V = _qkv(1, L, d)
    mask = None
    if use_mask:
        mask = (util.rng(9).standard_normal((L, L)) * 0.5).astype(np.float16)
        mask[:, L // 3] = -10000.0
    want = orc.attention(Q, K, V, [L], d, H, mask=mask)
    out = torch.full((L, d), float("nan"), dtype=torch.float16, device="cuda")
    et.attention_otf(out, dev(Q), dev(K), dev(V), None if mask is None else dev(mask), L, d, H)
    torch.cuda.synchronize()
    util.assert_close(host(out), want, what=f"otf attention L={L}")


@pytest.mark.parametrize("scale,fp32_scores,max_abs,mean_abs", [(1.0, False, 4e-3, 2e-4), (1.0, True, 4e-3, 2e-4),
                                                                  (3.0, True, 6e-3, 4e-4), (3.0, False, 6e-3, 4e-4)])
def test_attention_score_precision(et, orc, scale, fp32_scores, max_abs, mean_abs):
    """Q K^T accumulates in fp32 under both settings of the score precision: with unit-variance operands (|q.k| up to ~45) and
    with operands three times larger (|q.k| up to ~390, softmax close to one-hot; scores rounded to fp16 would be off by 3e-2)
    the result stays within a third of the parity tolerance."""
    L, d, H = 512, 768, 12
    Q, K, V = _qkv(1, L, d)
    Q = (Q.astype(np.float32) * scale).astype(np.float16)
    K = (K.astype(np.float32) * scale).astype(np.float16)
    want = orc.attention(Q, K, V, [L], d, H)
    assert not et.attention_scores_fp32()
    et.set_attention_scores_fp32(fp32_scores)
    try:
        assert et.attention_scores_fp32() == fp32_scores
        out = torch.full((L, d), float("nan"), dtype=torch.float16, device="cuda")
        et.attention_otf(out, dev(Q), dev(K), dev(V), None, L, d, H)
        torch.cuda.synchronize()
    finally:
        et.set_attention_scores_fp32(False)
    util.assert_close(host(out), want, max_abs=max_abs, mean_abs=mean_abs, what=f"scores fp32={fp32_scores}, scale {scale}")


def test_attention_otf_matches_reference_kernel_in_base2_mode(et, orc, ref):
    """The shipped kernel exponentiates in base 2 and floors the row max at 0; with its scale multiplied by
    log2(e) and scores that stay positive-max it computes a true softmax, comparable with ours."""
    L, d, H = 128, 768, 12
    Q, K, V = _qkv(3, L, d, std=0.5)
    mask = np.zeros((L, L), dtype=np.float16)
    Qd, Kd, Vd, Md = dev(Q), dev(K), dev(V), dev(mask)
    outr = torch.zeros((L, d), dtype=torch.float16, device="cuda")
    scale = float(1.4426950408889634 / np.sqrt(d // H))
    rc = ref.ref_otf_attention(_p(outr), _p(Qd), _p(Kd), _p(Vd), _p(Md), L, d, H, ctypes.c_float(scale), None)
    torch.cuda.synchronize()
    assert rc == 0
    want = orc.attention(Q, K, V, [L], d, H)
    util.assert_close(host(outr), want, max_abs=6e-2, mean_abs=6e-3, what="reference OTF vs oracle")
    out = torch.zeros((L, d), dtype=torch.float16, device="cuda")
    et.attention_otf(out, Qd, Kd, Vd, Md, L, d, H)
    torch.cuda.synchronize()
    util.assert_close(host(out), host(outr), max_abs=6e-2, mean_abs=6e-3, what="new vs reference OTF")
    # as shipped (scale without log2 e): the oracle's compatibility mode reproduces it
    rc = ref.ref_otf_attention(_p(outr), _p(Qd), _p(Kd), _p(Vd), _p(Md), L, d, H, ctypes.c_float(-1.0), None)
    torch.cuda.synchronize()
    assert rc == 0
    from tests.oracle_lib import REF_COMPAT
    want2 = orc.attention(Q, K, V, [L], d, H, flags=REF_COMPAT)
    util.assert_close(host(outr), want2, max_abs=6e-2, mean_abs=6e-3, what="reference OTF as shipped vs compat oracle")


def test_attention_fully_masked_row_and_zero_valid(et, orc):
    L, d, H = 64, 128, 2
    Q, K, V = _qkv(5, L, d)
    mask = np.zeros((L, L), dtype=np.float16)
    mask[7, :] = -np.inf
    out = torch.full((L, d), float("nan"), dtype=torch.float16, device="cuda")
    et.attention_otf(out, dev(Q), dev(K), dev(V), dev(mask), L, d, H)
    torch.cuda.synchronize()
    got = host(out)
    assert np.isfinite(got).all() and (got[7] == 0).all()
    util.assert_close(got, orc.attention(Q, K, V, [L], d, H, mask=mask.astype(np.float32)), what="masked row")


@pytest.mark.parametrize("lens", [[5, 16, 23, 64, 65, 130], [512, 32, 33, 100], [1], [0, 7, 0, 128]])
def test_attention_batch_varlen(et, orc, lens):
    d, H = 768, 12
    T = sum(lens)
    Q, K, V = _qkv(11, max(T, 1), d)
    Q, K, V = Q[:T], K[:T], V[:T]
    want = orc.attention(Q, K, V, lens, d, H)
    cu = dev(np.concatenate([[0], np.cumsum(lens)]).astype(np.int32))
    out = torch.full((T, d), float("nan"), dtype=torch.float16, device="cuda")
    et.attention_batch(out, dev(Q), dev(K), dev(V), d, H, cu_seqlens=cu, batch=len(lens), total_tokens=T,
                       max_seq_len=max(lens))          # tensor-core kernel (all lengths <= 512)
    torch.cuda.synchronize()
    util.assert_close(host(out), want, what=f"varlen attention {lens}")
    out2 = torch.full((T, d), float("nan"), dtype=torch.float16, device="cuda")
    et.attention_batch(out2, dev(Q), dev(K), dev(V), d, H, cu_seqlens=cu, batch=len(lens), total_tokens=T)
    torch.cuda.synchronize()                           # longest length not given: general kernel
    util.assert_close(host(out2), want, what=f"varlen attention, general kernel {lens}")


def test_attention_batch_key_padding_equals_unpadded(et, orc):
    """Padded layout with valid_lens gives, on the valid rows, exactly the unpadded result."""
    d, H, S = 256, 4, 96
    lens = [40, 96, 17, 64]
    B = len(lens)
    Q, K, V = _qkv(21, B * S, d)
    valid = dev(np.array(lens, dtype=np.int32))
    out_pad = torch.zeros((B * S, d), dtype=torch.float16, device="cuda")
    et.attention_batch(out_pad, dev(Q), dev(K), dev(V), d, H, valid_lens=valid, batch=B, uniform_len=S)
    rows = np.concatenate([np.arange(b * S, b * S + lens[b]) for b in range(B)])
    cu = dev(np.concatenate([[0], np.cumsum(lens)]).astype(np.int32))
    out_var = torch.zeros((len(rows), d), dtype=torch.float16, device="cuda")
    et.attention_batch(out_var, dev(Q[rows]), dev(K[rows]), dev(V[rows]), d, H, cu_seqlens=cu, batch=B,
                       max_seq_len=max(lens))
    torch.cuda.synchronize()
    assert torch.equal(out_pad[torch.from_numpy(rows).cuda()], out_var)
    want = orc.attention(Q, K, V, [S] * B, d, H, valid_lens=lens)
    util.assert_close(host(out_pad), want, what="key-padded attention")


def test_attention_prune_scatter(et, orc):
    L, d, H = 256, 768, 12
    row_id = orc.gen_sparse_row_mat(d, 0.5, seed=5, nhead=H)
    hp = orc.head_ptr(row_id, H, d)
    nnz = len(row_id)
    Q, K = util.activations(1, (L, d)), util.activations(2, (L, d))
    Vc = util.activations(3, (L, nnz))
    want = orc.attention(Q, K, Vc, [L], d, H, v_col_id=row_id, v_head_ptr=hp)
    out = torch.full((L, d), float("nan"), dtype=torch.float16, device="cuda")
    et.attention_prune(out, dev(Q), dev(K), dev(Vc), dev(row_id), dev(hp), nnz, None, L, d, H)
    torch.cuda.synchronize()
    got = host(out)
    util.assert_close(got, want, what="pruned-V attention")
    dropped = np.setdiff1d(np.arange(d), row_id)
    assert (got[:, dropped] == 0).all()          # pruned columns are exactly zero


@pytest.mark.parametrize("L,mask", [(63, True), (64, False), (65, True), (127, False), (129, True), (192, True), (193, True), (383, True)])
def test_attention_block_edges(et, orc, L, mask):
    """Both sides of a half and of a whole block of 128 keys and queries, with mask rows at every alignment."""
    d, H = 192, 3
    Q, K, V = _qkv(51, L, d)
    M = (util.rng(L).standard_normal((L, L))).astype(np.float16) if mask else None
    out = torch.full((L, d), float("nan"), dtype=torch.float16, device="cuda")
    et.attention_otf(out, dev(Q), dev(K), dev(V), None if M is None else dev(M), L, d, H)
    torch.cuda.synchronize()
    et.attention_check()
    util.assert_close(host(out), orc.attention(Q, K, V, [L], d, H, mask=M), what=f"attention L={L}")


@pytest.mark.parametrize("sparsity,L,mask", [(0.03, 129, False), (0.1, 77, True), (0.5, 65, True), (0.75, 200, False)])
def test_attention_prune_window_widths(et, orc, sparsity, L, mask):
    """Compact windows from a few columns to nearly the whole head: the wide ones do not fit one copied box of 64 columns at
    their alignment and are done in two passes."""
    d, H = 512, 8
    row_id = orc.gen_sparse_row_mat(d, sparsity, seed=15, nhead=H)
    row_id = row_id[:len(row_id) // 8 * 8]           # a row pitch in whole 16-byte units
    hp = orc.head_ptr(row_id, H, d)
    nnz = len(row_id)
    Q, K, Vc = util.activations(1, (L, d)), util.activations(2, (L, d)), util.activations(3, (L, nnz))
    M = util.rng(L).standard_normal((L, L)).astype(np.float16) if mask else None
    out = torch.full((L, d), float("nan"), dtype=torch.float16, device="cuda")
    et.attention_prune(out, dev(Q), dev(K), dev(Vc), dev(row_id), dev(hp), nnz, None if M is None else dev(M), L, d, H)
    torch.cuda.synchronize()
    et.attention_check()
    got = host(out)
    util.assert_close(got, orc.attention(Q, K, Vc, [L], d, H, mask=M, v_col_id=row_id, v_head_ptr=hp), what=f"pruned V, sparsity {sparsity}")
    assert (got[:, np.setdiff1d(np.arange(d), row_id)] == 0).all()


@pytest.mark.parametrize("mask", [False, True])
def test_attention_ragged_batch_with_empty_and_padded_sequences(et, orc, mask):
    """More items than CTAs that fit at once, sequences without tokens or without valid keys among them."""
    d, H = 256, 4
    rng = util.rng(99)
    lens = [int(n) for n in rng.integers(1, 300, size=150)] + [0, 128, 0, 1]
    valid = [int(rng.integers(0, n + 1)) if i % 3 == 0 else n for i, n in enumerate(lens)]
    T, L = sum(lens), max(lens)
    Q, K, V = _qkv(61, T, d)
    M = util.rng(5).standard_normal((L, L)).astype(np.float16) if mask else None
    cu = dev(np.concatenate([[0], np.cumsum(lens)]).astype(np.int32))
    out = torch.full((T, d), float("nan"), dtype=torch.float16, device="cuda")
    et.attention_batch(out, dev(Q), dev(K), dev(V), d, H, cu_seqlens=cu, valid_lens=dev(np.array(valid, dtype=np.int32)),
                       batch=len(lens), max_seq_len=L, mask=None if M is None else dev(M), mask_ld=L if mask else 0)
    torch.cuda.synchronize()
    et.attention_check()
    want = np.zeros((T, d), dtype=np.float32)
    o = 0
    for n, v in zip(lens, valid):
        if n:
            want[o:o + n] = orc.attention(Q[o:o + n], K[o:o + n], V[o:o + n], [n], d, H, mask=None if M is None else M[:n, :n].copy(), valid_lens=[v])
        o += n
    util.assert_close(host(out), want, what="ragged batch")


@pytest.mark.parametrize("batch,mask,pruned_keys", [(150, False, False), (160, True, True), (256, False, True), (257, False, False)])
def test_attention_ragged_batch_longer_than_a_wave(et, orc, batch, mask, pruned_keys):
    """More items than places: sequences are taken longest first (up to 256 of them; 257 are searched in order), every class of
    lengths among them. The caller's bound on the length may exceed the longest sequence, and the mask ends with that sequence's
    last key."""
    lens = [int(n) for n in util.rng(batch).integers(0, 140, size=batch)]
    lens[3], lens[batch - 2], lens[7] = 261, 129, 0
    lens[20:27] = [1100, 128, 900, 500, 700, 385, 1024]
    T, L = sum(lens), max(lens)
    places = 2 * torch.cuda.get_device_properties(0).multi_processor_count
    H = places // -(-T // 128) + 1   # heads enough that the blocks of 128 tokens known to exist outnumber the places
    d = 64 * H
    valid = [int(n) for n in util.rng(batch + 1).integers(0, 270, size=batch)] if pruned_keys else None
    if pruned_keys:
        valid[20], valid[22], valid[26] = 1100, 890, 2000
    Q, K, V = _qkv(batch, T, d)
    m = (util.rng(5).standard_normal((L, L)) * 0.5).astype(np.float16) if mask else None
    want = orc.attention(Q, K, V, lens, d, H, mask=m, valid_lens=None if valid is None else [min(v, n) for v, n in zip(valid, lens)])
    out = torch.full((T, d), float("nan"), dtype=torch.float16, device="cuda")
    et.attention_batch(out, dev(Q), dev(K), dev(V), d, H, cu_seqlens=dev(np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)), batch=batch,
                       max_seq_len=L + 100, mask=None if m is None else dev(m), mask_ld=L if mask else 0,
                       valid_lens=None if valid is None else dev(np.array(valid, dtype=np.int32)))
    torch.cuda.synchronize()
    et.attention_check()
    util.assert_close(host(out), want, what=f"{batch} ragged sequences")


@pytest.mark.parametrize("batch,L,ld", [(1, 136, 136), (1, 200, 208), (40, 136, 136), (40, 130, 130), (3, 300, 301)])
def test_attention_masks_of_every_row_alignment(et, orc, batch, L, ld):
    """Rows on 16-byte boundaries come by TMA, others in granules; with an SM per item two blocks' masks are held."""
    d, H = 256, 4
    Q, K, V = _qkv(L + batch, batch * L, d)
    m = (util.rng(L).standard_normal((L, ld)) * 0.5).astype(np.float16)
    m[:, L // 3] = -np.inf
    want = orc.attention(Q, K, V, [L] * batch, d, H, mask=m[:, :L])
    out = torch.full((batch * L, d), float("nan"), dtype=torch.float16, device="cuda")
    et.attention_batch(out, dev(Q), dev(K), dev(V), d, H, batch=batch, uniform_len=L, mask=dev(m), mask_ld=ld)
    torch.cuda.synchronize()
    util.assert_close(host(out), want, what=f"mask of pitch {ld}")


@pytest.mark.parametrize("batch,L,ld", [(2, 200, 8), (1, 136, 64), (3, 72, 16)])
def test_attention_masks_whose_rows_overlap(et, orc, batch, L, ld):
    """A pitch below the length: each row begins inside the one before."""
    d, H = 128, 2
    Q, K, V = _qkv(L + ld, batch * L, d)
    flat = (util.rng(ld).standard_normal((L - 1) * ld + L) * 0.5).astype(np.float16)
    m = np.lib.stride_tricks.as_strided(flat, (L, L), (2 * ld, 2))
    want = orc.attention(Q, K, V, [L] * batch, d, H, mask=np.ascontiguousarray(m))
    out = torch.full((batch * L, d), float("nan"), dtype=torch.float16, device="cuda")
    et.attention_batch(out, dev(Q), dev(K), dev(V), d, H, batch=batch, uniform_len=L, mask=dev(flat), mask_ld=ld)
    torch.cuda.synchronize()
    util.assert_close(host(out), want, what=f"mask of pitch {ld} below {L}")


@pytest.mark.parametrize("mask,prune", [(False, False), (True, False), (False, True)])
def test_attention_keys_that_are_not_numbers_reach_every_query(et, orc, mask, prune):
    """A key that is not a number makes every score with it, and so every row of the result, not a number, wherever in a block
    the key lies (exponentials are taken in different ways by position); other heads stay clean."""
    L, d, H = 136, 128, 2
    Q, K, V = (dev(x) for x in _qkv(91, L, d))
    M = dev(util.rng(92).standard_normal((L, L)).astype(np.float16)) if mask else None
    ids = np.arange(0, d, 2, dtype=np.int32)
    lost = []
    for key in range(L):
        Kn = K.clone()
        Kn[key, 5] = float("nan")
        out = torch.zeros((L, d), dtype=torch.float16, device="cuda")
        if prune:
            et.attention_prune(out, Q, Kn, V[:, :len(ids)].contiguous(), dev(ids), dev(orc.head_ptr(ids, H, d)), len(ids), M, L, d, H)
        else:
            et.attention_otf(out, Q, Kn, V, M, L, d, H)
        cols = ids[ids < 64] if prune else np.arange(64)
        if not torch.isnan(out[:, cols.tolist()]).all() or not torch.isfinite(out[:, 64:]).all():
            lost.append(key)
    et.attention_check()
    assert not lost, lost


@pytest.mark.parametrize("layout,H", [("padded", 2), ("packed", 1), ("packed", 5)])
def test_attention_keys_beyond_the_end_of_every_remainder(et, orc, layout, H):
    """Valid keys up to every place of a block, and keys that are large or not finite right behind them in memory: the padding's,
    or the next sequence's (with five heads in more items than places, longest first). They count for nothing."""
    d = 64 * H
    poison = np.array([np.nan, np.inf, -np.inf, 60000.0, -60000.0], dtype=np.float16)
    if layout == "padded":
        S, valid = 256, list(range(1, 257))
        T = S * len(valid)
        behind = np.concatenate([np.arange(b * S + v, (b + 1) * S) for b, v in enumerate(valid)])
        lens, kw = [S] * len(valid), dict(uniform_len=S, valid_lens=dev(np.array(valid, dtype=np.int32)))
    else:
        valid = lens = [n for i in range(1, 129) for n in (i, 1)]   # every other sequence is a token whose key is not finite
        T = sum(lens)
        starts = np.concatenate([[0], np.cumsum(lens)])
        behind = starts[1:-1:2]
        kw = dict(cu_seqlens=dev(starts.astype(np.int32)), max_seq_len=128)
    Q, K, V = _qkv(T, T, d)
    want = orc.attention(Q, K, V, lens, d, H, valid_lens=valid)
    K[behind] = poison[(np.arange(len(behind))[:, None] + np.arange(d)[None, :]) % len(poison)]
    out = torch.full((T, d), float("nan"), dtype=torch.float16, device="cuda")
    et.attention_batch(out, dev(Q), dev(K), dev(V), d, H, batch=len(lens), **kw)
    torch.cuda.synchronize()
    et.attention_check()
    rows = np.arange(T) if layout == "padded" else np.setdiff1d(np.arange(T), np.concatenate([behind, starts[-2:-1]]))
    util.assert_close(host(out)[rows], want[rows], what=f"{layout}, every remainder")


@pytest.mark.parametrize("L", [40, 128, 200])
def test_attention_many_items_per_cta_repeat_exactly(et, orc, L):
    """Items of one or two key blocks taken over one after the other, so that the next item's first block is often, but not
    always, there when the current one's last is multiplied: the same bits on every launch."""
    d, H, B = 256, 4, 400
    Q, K, V = _qkv(71, B * L, d)
    dq, dk, dv = dev(Q), dev(K), dev(V)
    outs = [torch.full((B * L, d), float("nan"), dtype=torch.float16, device="cuda") for _ in range(8)]
    for out in outs:
        et.attention_batch(out, dq, dk, dv, d, H, batch=B, uniform_len=L)
    torch.cuda.synchronize()
    et.attention_check()
    assert all(torch.equal(outs[0], out) for out in outs[1:])
    n = 3 * L
    util.assert_close(host(outs[0])[-n:], orc.attention(Q[-n:], K[-n:], V[-n:], [L] * 3, d, H), what=f"last sequences of {B} x {L}")


@pytest.mark.parametrize("mask,bound", [(False, 2.84e-4), (True, 2.7e-4)])
def test_attention_prune_precision(et, orc, mask, bound):
    """Against 64 bits over many key blocks. What the data types give is the rounding of the probabilities, of which the largest
    is exactly 1, and of the result, ~2e-4 each: 2.78e-4 and 2.60e-4 (with the mask the largest probabilities weigh more).
    Probabilities taken relative to an earlier block's maximum gave 2.90e-4 and 2.89e-4."""
    L, d, H = 1000, 768, 12
    ids = orc.gen_sparse_row_mat(d, 0.5, seed=6, nhead=H)
    hp = orc.head_ptr(ids, H, d)
    ids, hp = ids[:len(ids) // 8 * 8], np.minimum(hp, len(ids) // 8 * 8)
    Q, K, V = (util.activations(s, (L, n)) for s, n in ((1, d), (2, d), (3, len(ids))))
    M = util.activations(4, (L, L)) if mask else None
    out = torch.zeros((L, d), dtype=torch.float16, device="cuda")
    et.attention_prune(out, dev(Q), dev(K), dev(V), dev(ids), dev(hp.astype(np.int32)), len(ids), None if M is None else dev(M), L, d, H)
    et.attention_check()
    q, k, v = (torch.from_numpy(x).double().cuda() for x in (Q, K, V))
    want = torch.zeros((L, d), dtype=torch.float64, device="cuda")
    for h in range(H):
        s = q[:, 64 * h:64 * h + 64] @ k[:, 64 * h:64 * h + 64].T / 8
        if mask:
            s = s + torch.from_numpy(M).double().cuda()
        want[:, ids[hp[h]:hp[h + 1]].tolist()] = torch.softmax(s, -1) @ v[:, hp[h]:hp[h + 1]]
    rel = float((out.double() - want).norm() / want.norm())
    assert rel <= bound, rel


def test_attention_qk_and_v_pruned(et, orc):
    L, d, H = 100, 768, 12
    row_id = orc.gen_sparse_row_mat(d, 0.5, seed=6, nhead=H)
    hp = orc.head_ptr(row_id, H, d)
    nnz = len(row_id)
    Qc, Kc, Vc = (util.activations(s, (L, nnz)) for s in (1, 2, 3))
    want = orc.attention(Qc, Kc, Vc, [L], d, H, qk_head_ptr=hp, v_col_id=row_id, v_head_ptr=hp)
    out = torch.full((L, d), float("nan"), dtype=torch.float16, device="cuda")
    hpd, rid = dev(hp), dev(row_id)
    et.attention_batch(out, dev(Qc), dev(Kc), dev(Vc), d, H, batch=1, uniform_len=L, qk_head_ptr=hpd,
                       v_col_id=rid, v_head_ptr=hpd)
    torch.cuda.synchronize()
    util.assert_close(host(out), want, what="Q/K/V-pruned attention")


@pytest.mark.parametrize("L", [128, 72])
def test_scores_then_sharedqk(et, orc, L):
    d, H = 768, 12
    Q, K, V = _qkv(31, L, d)
    mask = (util.rng(9).standard_normal((L, L)) * 0.5).astype(np.float16)
    S = torch.zeros((H, L, L), dtype=torch.float16, device="cuda")
    et.qk_scores(S, dev(Q), dev(K), L, d, H)
    torch.cuda.synchronize()
    util.assert_close(host(S), orc.scores(Q, K, d, H), what="qk scores")
    out = torch.zeros((L, d), dtype=torch.float16, device="cuda")
    et.attention_sharedqk(out, S, dev(V), dev(mask), L, d, H)
    torch.cuda.synchronize()
    want = orc.sharedqk_attention(host(S), V, d, H, mask=mask)
    util.assert_close(host(out), want, what="sharedQK attention")
    util.assert_close(host(out), orc.attention(Q, K, V, [L], d, H, mask=mask), what="sharedQK vs on-the-fly")


def test_sharedqk_matches_reference_kernel_with_zero_mask(et, orc, ref):
    L, d, H = 128, 768, 12
    Q, K, V = _qkv(41, L, d, std=0.5)
    S = (orc.scores(Q, K, d, H) * 1.4426950408889634).astype(np.float16)   # base-2 kernel: pre-scale by log2 e
    Sd, Vd, Md = dev(S), dev(V), torch.zeros((L, L), dtype=torch.float16, device="cuda")
    outr = torch.zeros((L, d), dtype=torch.float16, device="cuda")
    rc = ref.ref_sharedqk_attention(_p(outr), _p(Sd), _p(Vd), _p(Md), L, d, H)
    torch.cuda.synchronize()
    assert rc == 0
    want = orc.attention(Q, K, V, [L], d, H)
    util.assert_close(host(outr), want, max_abs=6e-2, mean_abs=6e-3, what="reference sharedQK vs oracle")


def test_row_linear_and_meta(et, orc):
    T, K, N, H = 300, 768, 768, 12
    row_id = orc.gen_sparse_row_mat(N, 0.5, seed=8, nhead=H)
    W = util.weights(1, (len(row_id), K))
    b = util.weights(2, (len(row_id),), 0.1)
    X = util.activations(3, (T, K))
    w = et.RowWeight(K, N, T, W, row_id, b, H)
    assert w.row_id_size == len(row_id) and w.nrow == (len(row_id) + 15) // 16 * 16
    assert (w.head_ptr == orc.head_ptr(row_id, H, N)).all()                 # bit-exact index structure
    out = torch.full((T, w.nrow), float("nan"), dtype=torch.float16, device="cuda")
    w.run(out, dev(X))
    torch.cuda.synchronize()
    want = orc.row_linear(X, W, b, out_pitch=w.nrow)
    util.assert_close(host(out), want, what="row-pruned linear")
    # ragged keep count (not a multiple of 16): padding columns are exactly zero
    row_id2 = row_id[:-5]
    w2 = et.RowWeight(K, N, T, W[:-5], row_id2, b[:-5], H)
    out2 = torch.full((T, w2.nrow), float("nan"), dtype=torch.float16, device="cuda")
    w2.run(out2, dev(X))
    torch.cuda.synchronize()
    got2 = host(out2)
    util.assert_close(got2, orc.row_linear(X, W[:-5], b[:-5], out_pitch=w2.nrow), what="row-pruned ragged")
    assert (got2[:, len(row_id2):] == 0).all()


def test_row_linear_matches_reference_cublas_path(et, orc, ref):
    T, K, N, H = 256, 768, 768, 12
    row_id = orc.gen_sparse_row_mat(N, 0.5, seed=8, nhead=H)     # 384 rows: a multiple of 16
    W = util.weights(1, (len(row_id), K))
    b = util.weights(2, (len(row_id),), 0.1)
    X = util.activations(3, (T, K))
    Xd, Wd, bd = dev(X), dev(W), dev(b)
    outr = torch.zeros((T, len(row_id)), dtype=torch.float16, device="cuda")
    rc = ref.ref_row_spmm(_p(outr), _p(Xd), _p(Wd), _p(bd), T, len(row_id), K, None)
    torch.cuda.synchronize()
    assert rc == 0
    w = et.RowWeight(K, N, T, W, row_id, b, H)
    out = torch.zeros((T, w.nrow), dtype=torch.float16, device="cuda")
    w.run(out, Xd)
    torch.cuda.synchronize()
    util.assert_close(host(out), host(outr), what="row-pruned linear vs reference cuBLAS path")


def test_generators_bit_exact_with_oracle(et, orc):
    for (nrow, ncol, s, seed, bern) in [(768, 768, 0.5, 1, False), (3072, 768, 0.9, 2, False),
                                        (768, 3072, 0.75, 3, True), (1024, 4096, 0.8, 4, True),
                                        (64, 64, 0.0, 5, False), (64, 64, 1.0, 6, True)]:
        rp, ro = et.gen_sparse_tile_mat(nrow, ncol, s, seed, bern)
        rp2, ro2 = orc.gen_sparse_tile_mat(nrow, ncol, s, seed, bern)
        assert (rp == rp2).all() and (ro == ro2).all()
    for (nrow, s, seed, H) in [(768, 0.5, 1, 12), (1024, 0.75, 2, 16), (768, 0.9, 3, 12)]:
        a, b = et.gen_sparse_row_mat(nrow, s, seed, H), orc.gen_sparse_row_mat(nrow, s, seed, H)
        assert (a == b).all()
        assert (et.build_head_ptr(a, H, nrow) == orc.head_ptr(b, H, nrow)).all()
