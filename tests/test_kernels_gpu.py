"""GPU parity tests: every CUDA entry point of the C-ABI library against the CPU oracle on the same
seeded inputs (fp16 result vs fp32 oracle: max-abs <= 2e-2, mean-abs <= 2e-3), plus the reference
project's own CUDA kernels where they are usable as shipped."""
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


# ------------------------------------------------------------------ skip LayerNorm
@pytest.mark.parametrize("num,size", [(1, 768), (7, 768), (2048, 768), (515, 1024), (33, 256),
                                      (5, 2048), (9, 200), (3, 1538)])
def test_skip_layernorm(et, orc, num, size):
    x, s = util.activations(1, (num, size)), util.activations(2, (num, size))
    g = (1.0 + util.weights(3, (size,), 0.2).astype(np.float32)).astype(np.float16)
    b = util.weights(4, (size,), 0.2)
    want = orc.skip_layernorm(x, s, g, b)
    xd = dev(x)
    et.skip_layernorm(xd, dev(s), dev(g), dev(b))
    torch.cuda.synchronize()
    util.assert_close(host(xd), want, what=f"skip_layernorm {num}x{size}")


@pytest.mark.parametrize("num,size", [(1, 1024), (9, 768), (148 * 24, 768), (148 * 24 + 1, 768), (148 * 48 + 5, 768), (148 * 16 + 1, 1024), (5003, 1024)])
def test_skip_layernorm_rows_beyond_a_wave(et, num, size):
    """Warps that take one row, two, and one fewer than their neighbours, each requested while the one before is reduced."""
    gen = torch.Generator(device="cuda").manual_seed(num)
    x, s = (torch.randn((num, size), generator=gen, device="cuda").half() for _ in range(2))
    g, b = (torch.randn((size,), generator=gen, device="cuda").half() for _ in range(2))
    want = torch.nn.functional.layer_norm(x.double() + s.double(), (size,), g.double(), b.double(), 1e-6)
    et.skip_layernorm(x, s, g, b)
    torch.cuda.synchronize()
    # one fp16 rounding of values up to ~20 (half a unit: 8e-3)
    util.assert_close(host(x), want.float().cpu().numpy(), max_abs=1e-2, mean_abs=4e-4, what=f"skip_layernorm {num}x{size}")


def _fma(a, b, c):
    """One rounding (the product of two fp32 numbers is exact in 64 bits)."""
    return (a.double() * b.double() + c.double()).float()


def _layernorm_in_fp32(x, s, g, b):
    """skip LayerNorm operation by operation: 32 lanes with chunks of 8 elements, sums over the lanes in pairs."""
    rows, size = x.shape
    chunks = -(-size // 256)
    lay = lambda t: torch.nn.functional.pad(t, (0, chunks * 256 - size)).view(-1, chunks, 32, 8).float()
    there = lay(torch.ones_like(g[None])) != 0
    lanes = torch.arange(32, device="cuda")

    def over_lanes(t):
        for m in (16, 8, 4, 2, 1):
            t = t + t[:, lanes ^ m]
        return t[:, :1, None, None].view(rows, 1, 1, 1)
    v = lay(x) + lay(s)
    inv = torch.ones((), device="cuda") / torch.full((), float(size), device="cuda")
    total, sq = (torch.zeros((rows, 32), device="cuda") for _ in range(2))
    for i in range(chunks):
        for j in range(0, 8, 2):
            total = total + (v[:, i, :, j] + v[:, i, :, j + 1])
    d = _fma(-over_lanes(total), inv, v)
    for i in range(chunks):
        for j in range(8):
            more = _fma(d[:, i, :, j], d[:, i, :, j], sq) if i == 0 else sq + d[:, i, :, j] * d[:, i, :, j]
            sq = torch.where(there[:, i, :, j], more, sq)
    rstd = torch.rsqrt(_fma(over_lanes(sq), inv, torch.full((), 1e-6, device="cuda")))
    return _fma(d * rstd, lay(g[None]), lay(b[None])).half().view(rows, -1)[:, :size]


@pytest.mark.parametrize("num,size", [(8000, 256), (5003, 512), (3000, 768), (3000, 1024), (3000, 1280), (2999, 1536), (1200, 1792), (1201, 2048), (1000, 200),
                                      (1000, 1000), (1000, 2000)])
def test_skip_layernorm_rounds_alike_in_every_kernel(et, num, size):
    """The bits of a row do not depend on which kernel reduces it: stacks of layers amplify a different rounding."""
    gen = torch.Generator(device="cuda").manual_seed(size)
    x, s = (torch.randn((num, size), generator=gen, device="cuda").half() for _ in range(2))
    g, b = (torch.randn((size,), generator=gen, device="cuda").half() for _ in range(2))
    want = _layernorm_in_fp32(x, s, g, b)
    et.skip_layernorm(x, s, g, b)
    torch.cuda.synchronize()
    assert torch.equal(x, want), f"{int((x != want).sum())} results differ"


@pytest.mark.parametrize("num,size", [(1, 256), (3121, 256), (3122, 256), (3, 512), (2072, 512), (2073, 512), (1040, 768), (1041, 768), (2072, 768), (2073, 768), (780, 1024),
                                      (781, 1024), (5, 1280), (520, 1536), (445, 1792), (390, 2048), (391, 2048)])
def test_skip_layernorm_of_few_rows_rounds_alike(et, num, size):
    """One row to a warp, in blocks of one and two warps, and the first sizes that are not: the bits of the other kernels."""
    gen = torch.Generator("cuda").manual_seed(num + size)
    x, s = (torch.randn((num, size), generator=gen, device="cuda").half() for _ in range(2))
    g, b = (torch.randn((size,), generator=gen, device="cuda").half() for _ in range(2))
    want = _layernorm_in_fp32(x, s, g, b)
    et.skip_layernorm(x, s, g, b)
    torch.cuda.synchronize()
    assert torch.equal(x, want), f"{int((x != want).sum())} results differ"


@pytest.mark.parametrize("num,size,offset", [(3, 1, 0), (5, 33, 0), (4, 769, 0), (2, 2049, 0), (5, 200, 1), (3, 768, 3), (2, 1538, 1), (7, 2, 0), (9, 770, 2)])
def test_skip_layernorm_rows_anywhere(et, orc, num, size, offset):
    """Odd widths, and bases on 2-byte and 4-byte boundaries: single elements and pairs."""
    x, s = util.activations(1, (num, size)), util.activations(2, (num, size))
    g = (1.0 + util.weights(3, (size,), 0.2).astype(np.float32)).astype(np.float16)
    b = util.weights(4, (size,), 0.2)
    buf = torch.full((num * size + 16,), 7.0, dtype=torch.float16, device="cuda")
    view = buf[offset:offset + num * size].view(num, size)
    view.copy_(dev(x))
    et.skip_layernorm(view, dev(s), dev(g), dev(b))
    torch.cuda.synchronize()
    util.assert_close(host(view), orc.skip_layernorm(x, s, g, b), what=f"skip_layernorm {num}x{size} at {offset}")
    assert (buf[:offset] == 7).all() and (buf[offset + num * size:] == 7).all()


def test_skip_layernorm_matches_reference_kernels(et, orc, ref):
    for num, size in [(128, 768), (2048, 768), (1024, 1024)]:   # v1 and v2 kernels of the reference
        x, s = util.activations(1, (num, size)), util.activations(2, (num, size))
        g = (1.0 + util.weights(3, (size,), 0.2).astype(np.float32)).astype(np.float16)
        b = util.weights(4, (size,), 0.2)
        want = orc.skip_layernorm(x, s, g, b)
        xr, sd, gd, bd = dev(x), dev(s), dev(g), dev(b)   # keep the tensors alive across the launch
        rc = ref.ref_skip_layernorm(_p(xr), _p(sd), _p(gd), _p(bd), num, size, None)
        torch.cuda.synchronize()
        assert rc == 0
        # the reference adds, centres and scales in fp16 in its second kernel: looser bound
        util.assert_close(host(xr), want, max_abs=6e-2, mean_abs=6e-3, what="reference LN vs oracle")
        xd = dev(x)
        et.skip_layernorm(xd, sd, gd, bd)
        torch.cuda.synchronize()
        util.assert_close(host(xd), host(xr), max_abs=6e-2, mean_abs=6e-3, what="new vs reference LN")


def test_skip_layernorm_bad_args(et):
    x = torch.zeros(4, 768, dtype=torch.float16, device="cuda")
    with pytest.raises(et.EtError):
        et.check(et.lib().et_skip_layernorm(None, _p(x), _p(x), _p(x), 4, 768, None))
    with pytest.raises(et.EtError):
        et.check(et.lib().et_skip_layernorm(_p(x), _p(x), _p(x), _p(x), 4, 0, None))
    et.check(et.lib().et_skip_layernorm(_p(x), _p(x), _p(x), _p(x), 0, 768, None))  # empty is fine


def test_skip_layernorm_of_any_width_fills_the_gpu(et):
    """Widths that are no multiple of 8 make three passes over a row, by pairs of elements (770: 2.0 times the time of 768 at 17771
    rows, 18 against 9 us) or one by one (769: 3.7 times; 5.0 with a grid of six blocks per SM instead of the eight that fit)."""
    rows, times = 17771, {}
    for size in (768, 769, 770):
        x, s = (torch.randn((rows, size), device="cuda").half() for _ in range(2))
        g, b = torch.ones(size, device="cuda").half(), torch.zeros(size, device="cuda").half()
        best = float("inf")
        for _ in range(8):
            start, stop = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            start.record()
            for _ in range(20):
                et.skip_layernorm(x, s, g, b)
            stop.record()
            torch.cuda.synchronize()
            best = min(best, start.elapsed_time(stop))
        times[size] = best
    assert times[770] < 2.8 * times[768] and times[769] < 4.4 * times[768], times


# ------------------------------------------------------------------ mask + softmax
@pytest.mark.parametrize("nmat,L,valid,use_mask", [(12, 128, None, True), (3, 256, 200, True),
                                                   (2, 512, None, False), (5, 40, 33, True),
                                                   (2, 77, None, True), (1, 1024, 1000, False)])
def test_softmax_mask(et, orc, nmat, L, valid, use_mask):
    S = (util.rng(5).standard_normal((nmat, L, L)) * 3).astype(np.float16)
    mask = (util.rng(6).standard_normal((L, L))).astype(np.float16) if use_mask else None
    if use_mask:
        mask[:, L // 2] = -10000.0          # a padded key column
    want = orc.softmax_mask(S, mask, valid)
    Sd = dev(S)
    et.softmax_mask(Sd, None if mask is None else dev(mask), valid)
    torch.cuda.synchronize()
    got = host(Sd)
    util.assert_close(got, want, what=f"softmax {nmat}x{L}")
    if valid is not None:
        assert (got[:, :, valid:] == 0).all()


def test_softmax_fully_masked_row_is_zero(et):
    L = 64
    S = dev(util.activations(1, (2, L, L)))
    et.softmax_mask(S, None, 0)
    torch.cuda.synchronize()
    assert (host(S) == 0).all()


@pytest.mark.parametrize("nmat,L,offset,use_mask,cut", [(1131, 63, 1, True, 0), (5000, 15, 0, False, 2), (283, 127, 3, True, 30), (280, 127, 0, False, 0),
                                                         (71, 255, 5, True, 0), (51, 509, 0, True, 9), (49, 365, 7, True, 0), (36, 500, 0, False, 1)])
def test_softmax_many_rows_of_any_alignment(et, orc, nmat, L, offset, use_mask, cut):
    """Enough rows that a group of lanes takes several, and with a mask several matrices for each of its rows."""
    S = (util.rng(L).standard_normal((nmat, L, L)) * 3).astype(np.float16)
    mask = util.rng(L + 1).standard_normal((L, L)).astype(np.float16) if use_mask else None
    buf = torch.full((nmat * L * L + 16,), 7.0, dtype=torch.float16, device="cuda")
    buf[offset:offset + nmat * L * L] = dev(S).reshape(-1)
    view = buf[offset:offset + nmat * L * L].view(nmat, L, L)
    mbuf = torch.zeros(L * L + 8, dtype=torch.float16, device="cuda")
    if use_mask:
        mbuf[offset:offset + L * L] = dev(mask).reshape(-1)
    et.softmax_mask(view, mbuf[offset:offset + L * L].view(L, L) if use_mask else None, L - cut)
    torch.cuda.synchronize()
    util.assert_close(host(view), orc.softmax_mask(S, mask, L - cut), what=f"softmax {nmat}x{L}")
    assert (host(view)[:, :, L - cut:] == 0).all()
    assert (buf[:offset] == 7).all() and (buf[offset + nmat * L * L:] == 7).all()


@pytest.mark.parametrize("nmat,L,use_mask", [(90, 231, True), (85, 233, True), (85, 233, False), (80, 255, True), (75, 255, False), (70, 257, False), (50, 463, True),
                                             (50, 465, True), (50, 465, False), (49, 511, True), (190, 233, False), (330, 255, True)])
def test_softmax_rows_in_flight_by_length(et, orc, nmat, L, use_mask):
    """Lengths around which another number of rows is in flight, with enough matrices for it, three tokens masked at the end."""
    S, mask = util.activations(L, (nmat, L, L)), util.activations(L + 1, (L, L))
    Sd = dev(S)
    et.softmax_mask(Sd, dev(mask) if use_mask else None, L - 3)
    torch.cuda.synchronize()
    some = [0, 1, 7, nmat // 2, nmat - 1]
    util.assert_close(host(Sd)[some], orc.softmax_mask(S[some], mask if use_mask else None, L - 3), what=f"softmax {nmat}x{L}")


@pytest.mark.parametrize("nmat,L", [(109, 429), (109, 431), (110, 431), (93, 510)])
def test_softmax_rows_in_flight_of_long_rows_without_a_mask(et, orc, nmat, L):
    """Both sides of 430 elements, from where one row in flight wants ten to a group, and both sides of ten."""
    test_softmax_rows_in_flight_by_length(et, orc, nmat, L, False)


@pytest.mark.parametrize("L", [1, 7, 241, 242, 243, 499, 1017, 1019, 2034, 2035])
@pytest.mark.parametrize("offset", [0, 3])
def test_softmax_mask_rows_of_any_alignment(et, orc, L, offset):
    """Lengths that are no multiple of 8 (both sides of each granule count per lane, and of the three-pass kernel), in a
    buffer that starts anywhere: rows share 16-byte granules with their neighbours, which must stay untouched."""
    nmat = 3
    S = (util.rng(L).standard_normal((nmat, L, L)) * 3).astype(np.float16)
    mask = util.rng(L + 1).standard_normal((L, L)).astype(np.float16)
    valid = max(1, L - L // 5)
    buf = torch.full((nmat * L * L + 16,), 7.0, dtype=torch.float16, device="cuda")
    buf[offset:offset + nmat * L * L] = dev(S).reshape(-1)
    mbuf = torch.zeros(L * L + 8, dtype=torch.float16, device="cuda")
    mbuf[offset:offset + L * L] = dev(mask).reshape(-1)
    view = buf[offset:offset + nmat * L * L].view(nmat, L, L)
    et.softmax_mask(view, mbuf[offset:offset + L * L].view(L, L), valid)
    torch.cuda.synchronize()
    util.assert_close(host(view), orc.softmax_mask(S, mask, valid), what=f"softmax L={L} offset={offset}")
    assert (host(view)[:, :, valid:] == 0).all()
    assert (buf[:offset] == 7).all() and (buf[offset + nmat * L * L:] == 7).all()


def test_softmax_mask_more_rows_than_31_bits_count(et):
    """2^30 + 3 matrices of 2 x 2 (8.6 GB): of two scores the softmax is known."""
    nmat, L = (1 << 30) + 3, 2
    if torch.cuda.mem_get_info()[0] < 30 << 30:
        pytest.skip("needs 30 GB of device memory")
    S = torch.zeros((nmat, L, L), dtype=torch.float16, device="cuda")
    S[:, :, 1] = 1.0
    S[-1, 1, 0] = 2.0
    et.softmax_mask(S)
    torch.cuda.synchronize()
    p = 1.0 / (1.0 + np.exp(1.0))
    half_unit = 2.0 ** -12                     # of fp16 between 0.25 and 1
    for at in range(0, nmat - 1, 1 << 28):
        assert float((S[at:min(at + (1 << 28), nmat - 1), :, 0].float() - p).abs().max()) <= half_unit, at
    assert abs(float(S[-1, 0, 0]) - p) <= half_unit and abs(float(S[-1, 1, 0]) - (1 - p)) <= half_unit
    del S
    torch.cuda.empty_cache()


# ------------------------------------------------------------------ tile-pruned linear
def _run_tile(et, orc, T, K, N, sparsity, seed, gelu=False, bernoulli=True, bias_std=0.05, size=None):
    rp, ro, data, bias = util.make_tile_linear(orc, K, N, sparsity, seed, bernoulli, bias_std)
    X = util.activations(seed + 10, (T, K))
    want = orc.tile_linear(X, rp, ro, data, bias, N, gelu=gelu)
    w = et.TileWeight(K, N, T if size is None else size, data, rp, ro, bias, is_gelu=gelu)
    Y = torch.full((T, N), float("nan"), dtype=torch.float16, device="cuda")
    w.run(Y, dev(X))
    torch.cuda.synchronize()
    w.check()
    return host(Y), want, w


@pytest.mark.parametrize("T,K,N,sparsity,gelu", [
    (128, 64, 16, 0.0, False),        # one tile column, one block-row
    (128, 768, 768, 0.5, False),
    (2048, 768, 768, 0.75, False),
    (2048, 768, 3072, 0.5, True),
    (2048, 3072, 768, 0.9, False),
    (300, 768, 768, 0.0, False),      # dense, ragged token count
    (1, 256, 48, 0.5, True),
    (4096, 1024, 1024, 0.8, False),
    (200, 80, 112, 0.3, False),       # K not a multiple of 64, N not a multiple of the chunk
])
def test_tile_linear(et, orc, T, K, N, sparsity, gelu):
    got, want, _ = _run_tile(et, orc, T, K, N, sparsity, seed=T + K + N, gelu=gelu)
    util.assert_close(got, want, what=f"tile linear T={T} K={K} N={N} s={sparsity}")


@pytest.mark.parametrize("T,K,N,sparsity,gelu,size,form", [
    (1, 3072, 768, 0.75, False, 128, "dense"),       # K split over a cluster, one row of a tile
    (129, 3072, 784, 0.0, True, 512, "dense"),       # ragged tokens and features
    (300, 1040, 1168, 0.0, False, 2048, "dense"),    # a K range of an odd number of panels, the last one partial
    (511, 768, 2304, 0.0, True, 32768, "dense"),     # pairs of CTAs, second CTA's tokens partly outside
    (1, 768, 2304, 0.75, False, 32768, "resident"),
    (700, 768, 3088, 0.75, True, 32768, "resident"),     # last group of one block-row
    (257, 752, 2320, 0.5, False, 32768, "resident"),     # a partial chunk of K
    (20000, 768, 768, 0.9, False, 32768, "resident"),    # several items per CTA
    (260, 1024, 1024, 0.9, False, 32768, "resident"),    # K beyond the tensor-memory part
    (5000, 1024, 4096, 0.9, True, 32768, "resident"),
    (300, 768, 2304, 0.995, False, 32768, "resident"),   # block-rows without tiles
    (700, 3072, 768, 0.75, False, 17792, "tile"),        # weight blocks back to back in their ring, many times round
    (701, 3072, 768, 0.6, False, 17792, "tile"),         # weight blocks in slots
])
def test_tile_linear_forms(et, orc, T, K, N, sparsity, gelu, size, form):
    """The forms a weight is packed in for an expected token count (`size`), run with other token counts too: edges of the
    slabs and tiles, partial chunks, and repeated calls give the same bits."""
    got, want, w = _run_tile(et, orc, T, K, N, sparsity, seed=T + K + N, gelu=gelu, size=size)
    info = w.info()
    assert form == ("tile" if info["stage_bytes"] else "dense" if info["stages"] else "resident"), info
    util.assert_close(got, want, what=f"{form} linear T={T} K={K} N={N} s={sparsity}")
    X = dev(util.activations(7, (T, K)))
    ys = [torch.full((T, N), float("nan"), dtype=torch.float16, device="cuda") for _ in range(3)]
    for y in ys:
        w.run(y, X)
    torch.cuda.synchronize()
    w.check()
    assert torch.equal(ys[0], ys[1]) and torch.equal(ys[0], ys[2])


@pytest.mark.parametrize("T,K,N,sparsity,gelu", [
    (1, 768, 768, 0.0, False),        # K in four shares of three panels, the last stage of one panel
    (128, 768, 2304, 0.0, False),     # two shares
    (130, 4096, 1024, 0.0, True),     # a second tile of two tokens
    (128, 4096, 1040, 0.5, False),    # columns beyond N, zeros among the tiles
    (256, 8192, 768, 0.0, False),     # more stages than the ring holds: stages filled again by the copying warps
    (96, 1040, 400, 0.0, True),       # a partial last panel, shares of unequal length
    (200, 528, 336, 0.25, False),
])
def test_dense_linear_split_over_a_cluster(et, orc, T, K, N, sparsity, gelu):
    """The K range split over a cluster: first stages and later ones, sums from all shares, repeated calls with other activations in
    between give the same bits."""
    got, want, w = _run_tile(et, orc, T, K, N, sparsity, seed=T + K + N, gelu=gelu, size=T)
    util.assert_close(got, want, what=f"split dense linear T={T} K={K} N={N}")
    xs = [dev(util.activations(7 + i, (T, K))) for i in range(2)]
    ys = [torch.full((T, N), float("nan"), dtype=torch.float16, device="cuda") for _ in range(6)]
    for i, y in enumerate(ys):
        w.run(y, xs[i % 2])
    torch.cuda.synchronize()
    w.check()
    assert all(torch.equal(ys[i % 2], y) for i, y in enumerate(ys))


@pytest.mark.parametrize("T,K,N,sparsity,gelu,shares,columns", [
    (1, 768, 768, 0.0, False, 4, 8),
    (128, 768, 1152, 0.0, False, 2, 16),
    (130, 4096, 1024, 0.0, True, 4, 16),
    (128, 4096, 1040, 0.5, False, 4, 8),
    (256, 8192, 768, 0.0, False, 8, 16),
    (96, 1040, 400, 0.0, True, 4, 8),
    (64, 1552, 2304, 0.25, False, 4, 24),    # pruned, a partial last panel, 24 columns to a CTA
    (700, 2064, 784, 0.25, True, 2, 48),
])
def test_dense_linear_in_shares(et, orc, T, K, N, sparsity, gelu, shares, columns):
    """Linears that are split over a cluster, with the shares and the columns of a CTA that they are to be split into."""
    rp, ro, data, bias = util.make_tile_linear(orc, K, N, sparsity, T + K + N, False, 0.05)
    info = et.TileWeight(K, N, T, data, rp, ro, bias, is_gelu=gelu).info()
    assert info["stage_bytes"] == 0 and info["stages"] == shares and 16 * info["nb"] == shares * columns, info
    test_dense_linear_split_over_a_cluster(et, orc, T, K, N, sparsity, gelu)


@pytest.mark.parametrize("T,K,N,sparsity,form", [(300, 1024, 1024, 0.24, "tile"), (400, 1024, 1024, 0.24, "tile"),
                                                 (32768, 768, 2304, 0.75, "resident"), (131072, 1024, 4096, 0.9, "resident"),
                                                 (17771, 3072, 768, 0.75, "tile"), (32768, 4096, 1024, 0.75, "tile"), (128, 3072, 768, 0.75, "dense")])
def test_the_form_that_was_measured_as_the_fastest_is_taken(et, orc, T, K, N, sparsity, form):
    """Where another form takes at least 5 % longer."""
    rp, ro, data, bias = util.make_tile_linear(orc, K, N, sparsity, K + N, False, 0.05)
    info = et.TileWeight(K, N, T, data, rp, ro, bias).info()
    assert form == ("tile" if info["stage_bytes"] else "dense" if info["stages"] else "resident"), info


@pytest.mark.parametrize("T,K,N,sparsity,form", [
    (8192, 768, 3072, 0.4, "resident"), (8192, 768, 1152, 0.5, "resident"), (17771, 768, 1152, 0.4, "resident"), (4096, 768, 2304, 0.25, "dense"),
    (32768, 768, 3072, 0.25, "dense"), (65536, 768, 2304, 0.25, "dense"), (65536, 768, 3072, 0.25, "dense"), (32768, 768, 3072, 0.4, "resident"),
    (32768, 1024, 4096, 0.4, "dense"), (65536, 4096, 1024, 0.4, "dense"), (65536, 1536, 1536, 0.4, "dense"), (6502, 4096, 1024, 0.75, "tile"),
    (65536, 1024, 512, 0.9, "tile"), (65536, 1024, 1024, 0.9, "resident"), (32768, 1024, 3072, 0.75, "resident"), (2299, 768, 768, 0.0, "tile"),
    (9195, 768, 192, 0.0, "tile"), (12000, 1024, 1536, 0.95, "resident"), (12000, 768, 1536, 0.9, "resident"),
])
def test_the_form_is_the_fastest_where_the_models_had_gone_wrong(et, orc, T, K, N, sparsity, form):
    """Where another form takes at least 5 % longer: long dense launches, which come to the power limit in the tile form, slabs that come from memory, many
    slabs that lie in L2."""
    test_the_form_that_was_measured_as_the_fastest_is_taken(et, orc, T, K, N, sparsity, form)


@pytest.mark.parametrize("K,N,sparsity,size,form,rows", [(768, 2304, 0.75, 32768, "resident", 2), (768, 3088, 0.75, 32768, "resident", 2), (1024, 1024, 0.9, 32768, "resident", 2),
                                                         (3072, 768, 0.75, 17792, "tile", None), (3072, 784, 0.0, 512, "dense", None)])
def test_weight_info_tells_how_the_features_are_cut(et, orc, K, N, sparsity, size, form, rows):
    """Block-rows per chunk times chunks cover the features, without a chunk too many, in every form; a group of the resident form is two block-rows
    (an odd number of block-rows leaves the last group with one)."""
    rp, ro, data, bias = util.make_tile_linear(orc, K, N, sparsity, K + N, True, 0.05)
    info = et.TileWeight(K, N, size, data, rp, ro, bias).info()
    assert form == ("tile" if info["stage_bytes"] else "dense" if info["stages"] else "resident"), info
    assert rows in (None, info["nb"])
    assert info["n_chunks"] == -(-N // (16 * info["nb"])) and info["k_chunks"] == -(-K // 128), info


@pytest.mark.parametrize("N,tokens", [(384, 65536), (576, 24000), (576, 65536)])
def test_long_dense_launches_have_no_columns_to_fill_up(et, orc, N, tokens):
    """A launch at the power limit takes the tile width that divides its columns."""
    rp, ro, data, bias = util.make_tile_linear(orc, 768, N, 0.0, N, True, 0.05)
    info = et.TileWeight(768, N, tokens, data, rp, ro, bias).info()
    assert info["nb"] * 16 * info["n_chunks"] == N


@pytest.mark.parametrize("T,N", [(24000, 576), (23933, 592)])
def test_long_dense_launches_against_the_oracle(et, orc, T, N):
    """Three tiles of 192 columns, and four of which the last is nearly empty: first and last tokens, those on both sides of a
    CTA's and of a pair's last one, and bits that do not depend on the launch."""
    rp, ro, data, bias = util.make_tile_linear(orc, 768, N, 0.0, N, True, 0.05)
    w = et.TileWeight(768, N, T, data, rp, ro, bias)
    X = util.activations(T, (T, 768))
    ys = [w.run(torch.full((T, N), float("nan"), dtype=torch.float16, device="cuda"), dev(X)) for _ in range(2)]
    torch.cuda.synchronize()
    w.check()
    assert torch.equal(ys[0], ys[1]) and torch.isfinite(ys[0]).all()
    for first in (0, 120, 12150, T - 140):
        rows = slice(first, first + 140)
        util.assert_close(host(ys[0][rows]), orc.tile_linear(X[rows], rp, ro, data, bias, N), what=f"tokens from {first}")


@pytest.mark.parametrize("K,N", [(3072, 768), (4096, 1040)])
def test_dense_weights_run_alike_whatever_count_they_were_made_for(et, orc, K, N):
    """How a dense weight is cut into tiles and shares of the K range is chosen for the tokens of the call: the same bits from
    weights made for few and for many, at both sides of where the choice changes."""
    rp, ro, data, bias = util.make_tile_linear(orc, K, N, 0.0, K, True, 0.05)
    made = [et.TileWeight(K, N, size, data, rp, ro, bias) for size in (1, 64, 512, 2048, 32768)]
    assert all(w.info()["stage_bytes"] == 0 and w.info()["stages"] for w in made)
    for T in (1, 64, 300, 1025, 5000):
        X = util.activations(T, (T, K))
        ys = [w.run(torch.full((T, N), float("nan"), dtype=torch.float16, device="cuda"), dev(X)) for w in made]
        torch.cuda.synchronize()
        assert all(torch.equal(ys[0], y) for y in ys[1:]), T
        rows = slice(max(0, T - 130), T)
        util.assert_close(host(ys[0])[rows], orc.tile_linear(X[rows], rp, ro, data, bias, N), what=f"dense linear T={T}")
    for w in made:
        w.check()


@pytest.mark.parametrize("T,K,N,gelu,columns", [(1, 3072, 16, False, 4), (64, 4096, 48, True, 4), (130, 1024, 784, False, 16), (257, 3072, 1040, True, 24),
                                                (400, 2048, 272, False, 12), (128, 768, 768, True, 8), (700, 3072, 768, False, 32),
                                                (855, 3072, 784, True, 48), (916, 4096, 1024, False, 64)])
def test_dense_shares_meet_at_every_width(et, orc, T, K, N, gelu, columns):
    """The K range in shares over a cluster: widths of 4 to 64 columns per CTA, outputs that begin between two sectors, and results
    that are not finite (found per column group and computed again)."""
    rp, ro, data, bias = util.make_tile_linear(orc, K, N, 0.5 if columns < 48 else 0.1, T + N, bernoulli=True, bias_std=0.1)
    X = util.activations(T, (T, K))
    w = et.TileWeight(K, N, T, data, rp, ro, bias, is_gelu=gelu)
    info = w.info()
    assert info["stage_bytes"] == 0 and info["stages"] > 1 and 16 * info["nb"] // info["stages"] == columns, info
    x = dev(X)
    buf = torch.full((T * N + 24,), 7.0, dtype=torch.float16, device="cuda")
    y = buf[8:8 + T * N].view(T, N)
    w.run(y, x)
    torch.cuda.synchronize()
    util.assert_close(host(y), orc.tile_linear(X, rp, ro, data, bias, N, gelu), what=f"dense linear {T} x {K} -> {N}")
    assert (buf[:8] == 7).all() and (buf[8 + T * N:] == 7).all()
    k0 = 16 * (K // 32)
    x[T // 2, k0:k0 + 16] = float("inf")   # one tile's inputs of one token
    z = torch.empty_like(y)
    w.run(z, x)
    torch.cuda.synchronize()
    dropped = torch.tensor([k0 not in ro[rp[r]:rp[r + 1]].tolist() for r in range(N // 16)]).repeat_interleave(16).cuda()
    assert torch.isfinite(z[T // 2][dropped]).all()
    keep = torch.arange(T, device="cuda") != T // 2
    assert torch.equal(z[keep], y[keep])


@pytest.mark.parametrize("T,K,N,sparsity,gelu,size,form", [
    (200, 3072, 768, 0.75, False, 128, "dense"),         # K split over a cluster
    (200, 3072, 784, 0.75, True, 128, "dense"),
    (700, 768, 2304, 0.5, False, 4096, "dense"),         # pairs of CTAs
    (700, 768, 2320, 0.5, True, 4096, "dense"),
    (300, 768, 2304, 0.98, False, 32768, "resident"),    # block-rows without tiles among them
    (300, 1024, 1040, 0.9, True, 32768, "resident"),
    (300, 3072, 768, 0.9, False, 17792, "tile"),
])
def test_tile_linear_activations_that_are_not_finite_pass_pruned_tiles_by(et, orc, T, K, N, sparsity, gelu, size, form):
    """An activation that is infinite or not a number reaches the outputs whose block-row keeps a tile at its input feature, and
    those of its token alone; every other output is what it is without that activation, in whichever form the weight is packed."""
    rp, ro, data, bias = util.make_tile_linear(orc, K, N, sparsity, T + K, True, 0.05)
    w = et.TileWeight(K, N, size, data, rp, ro, bias, is_gelu=gelu)
    info = w.info()
    assert form == ("tile" if info["stage_bytes"] else "dense" if info["stages"] else "resident"), info
    X = util.activations(5, (T, K))
    clean, reached = X.copy(), np.zeros((T, N), dtype=bool)
    for t, k, v in ((0, 3, np.inf), (1, K - 1, np.nan), (T // 2, 100, -np.inf), (T - 1, 7, np.nan), (T - 1, 500, np.inf)):
        X[t, k], clean[t, k] = v, 0
        for r in range(N // 16):
            reached[t, 16 * r:16 * r + 16] |= (ro[rp[r]:rp[r + 1]] == k // 16 * 16).any()
    assert reached.any() and not reached.all(axis=1).any()
    Y = torch.zeros((T, N), dtype=torch.float16, device="cuda")
    w.run(Y, dev(X))
    torch.cuda.synchronize()
    w.check()
    got, want = host(Y), orc.tile_linear(clean, rp, ro, data, bias, N, gelu=gelu)
    finite = np.isfinite(got)
    if not gelu:   # (GELU turns minus infinity into not a number, and an infinite sum of either sign may come)
        assert (finite == ~reached).all()
    assert finite[~reached].all()
    got[reached] = want[reached]
    util.assert_close(got, want, what=f"{form} linear, activations that are not finite")


def test_tile_linear_exact_count_shuffled_order_and_empty_rows(et, orc):
    # exact-count generator lists a block-row's tiles in shuffle order; at 95 % many block-rows are empty
    got, want, _ = _run_tile(et, orc, 256, 768, 768, 0.95, seed=77, bernoulli=False)
    util.assert_close(got, want, what="tile linear exact-count")
    got, want, _ = _run_tile(et, orc, 256, 768, 768, 1.0, seed=78, bernoulli=False, bias_std=0.3)
    util.assert_close(got, want, what="tile linear all tiles pruned (bias only)")


@pytest.mark.parametrize("size_hint", [128, 2048, 131072])
def test_tile_linear_all_chunkings(et, orc, size_hint):
    got, want, w = _run_tile(et, orc, 384, 768, 3072, 0.75, seed=3, gelu=True, size=size_hint)
    util.assert_close(got, want, what=f"tile linear hint {size_hint} {w.info()}")


@pytest.mark.parametrize("T,K,N,sparsity,gelu", [
    (2048, 768, 2304, 0.75, False),   # the fused Q|K|V shape of the 16 x 128 tile layer
    (2048, 768, 768, 0.75, False),
    (2048, 768, 3072, 0.75, True),
    (2048, 3072, 768, 0.75, False),
    (2048, 768, 768, 0.5, False),
    (4096, 1024, 4096, 0.8, True),    # BERT-large FFN1 slab count above one wave of two-tile CTAs
    (300, 768, 3072, 0.9, True),      # ragged token count, under-filled grid, odd tile count per CTA
])
def test_tile_linear_packed_for_throughput(et, orc, T, K, N, sparsity, gelu):
    """Weights packed under the throughput goal (larger chunks, two tiles per CTA): the configuration a caller
    with several batches in flight uses. Same oracle, same tolerance."""
    et.set_tuning_goal("throughput")
    try:
        got, want, w = _run_tile(et, orc, T, K, N, sparsity, seed=T + K + N + 1, gelu=gelu)
    finally:
        et.set_tuning_goal("latency")
    util.assert_close(got, want, what=f"tile linear (throughput packing) T={T} K={K} N={N} s={sparsity} {w.info()}")


@pytest.mark.parametrize("T,gelu", [(128, False), (129, True)])
def test_tile_linear_lists_of_every_length(et, orc, T, gelu):
    """An issuing warp has every eighth block-row and a list for each 128 inputs: of every length from none to 24 tiles, the last
    ones of a block included."""
    K, N = 25 * 128, 384
    have = {}                                   # (block-row, chunk of 128 inputs) -> number of tiles
    for chunk in range(25):
        for w in range(8):
            n = (chunk + 3 * w) % 25
            for i, row in enumerate((w, w + 8, w + 16)):
                have[row, chunk] = n // 3 + (i < n % 3)
    rp, ro = [0], []
    for row in range(24):
        for chunk in range(25):
            ro += [chunk * 128 + 16 * int(c) for c in sorted(util.rng(row * 31 + chunk).permutation(8)[:have[row, chunk]])]
        rp.append(len(ro))
    rp, ro = np.array(rp, np.int32), np.array(ro, np.int32)
    data, bias, X = util.weights(5, (len(ro), 256)), util.weights(6, (N,), 0.05), util.activations(7, (T, K))
    et.set_tuning_goal("throughput")            # always the tile form, 24 block-rows to a CTA
    try:
        w = et.TileWeight(K, N, T, data, rp, ro, bias, is_gelu=gelu)
    finally:
        et.set_tuning_goal("latency")
    assert w.info()["nb"] == 24
    Y = torch.full((T, N), float("nan"), dtype=torch.float16, device="cuda")
    w.run(Y, dev(X))
    torch.cuda.synchronize()
    w.check()
    util.assert_close(host(Y), orc.tile_linear(X, rp, ro, data, bias, N, gelu=gelu), what="lists of every length")


@pytest.mark.parametrize("goal", ["latency", "throughput"])
@pytest.mark.parametrize("T,K,sparse,full,sparsity", [(1665, 1024, 2048, 544, 0.75), (300, 1024, 2048, 544, 0.9), (1665, 4096, 512, 384, 0.8), (200, 2048, 16, 368, 0.5)])
def test_tile_linear_of_sparse_and_full_block_rows(et, orc, T, K, sparse, full, sparsity, goal):
    """Block-rows of every tile behind sparse ones, as where a compact V follows Q and K: the fullest block decides how many
    block-rows a CTA takes, not the mean."""
    rp, ro = orc.gen_sparse_tile_mat(sparse, K, sparsity, 3, True)
    rp = np.concatenate([rp, rp[-1] + np.arange(1, full // 16 + 1) * (K // 16)]).astype(np.int32)
    ro = np.concatenate([ro, np.tile(np.arange(0, K, 16), full // 16)]).astype(np.int32)
    N = sparse + full
    data, bias, X = util.weights(5, (len(ro), 256)), util.weights(6, (N,), 0.05), util.activations(7, (T, K))
    et.set_tuning_goal(goal)
    try:
        w = et.TileWeight(K, N, T, data, rp, ro, bias)
    finally:
        et.set_tuning_goal("latency")
    Y = w.run(torch.full((T, N), float("nan"), dtype=torch.float16, device="cuda"), dev(X))
    torch.cuda.synchronize()
    w.check()
    rows = slice(max(0, T - 140), T)
    util.assert_close(host(Y)[rows], orc.tile_linear(X[rows], rp, ro, data, bias, N), what=f"{sparse} sparse and {full} full outputs {w.info()}")


@pytest.mark.parametrize("T,K,full,gelu", [(129, 1024, (0, 1, 2, 3), False), (129, 1024, (5, 190), True), (20000, 768, (0, 1, 2, 3, 143), False), (257, 1008, (7, 64, 65), True),
                                           (300, 832, (3, 100), False), (130, 848, (0, 191), True), (1, 784, (17,), False)])
def test_resident_linear_with_groups_in_several_blocks(et, orc, T, K, full, gelu):
    """Groups of block-rows whose tiles exceed a slot of the weight ring are cut into blocks, first and last groups among them, beside groups in one block
    and block-rows without tiles; a block may hold none of a block-row, and its first tile may come in any of them. Inputs that tensor memory just holds, and one
    slice more."""
    rows = 192 if K > 768 else 144
    rng = np.random.default_rng(K + T)
    kept = [np.arange(K // 16) if r in full else np.sort(rng.choice(K // 16, rng.integers(0, K // 96), replace=False)) for r in range(rows)]
    kept[9] = np.array([K // 16 - 1])
    kept[10] = np.array([], np.int64)
    rp, ro = np.concatenate([[0], np.cumsum([len(k) for k in kept])]).astype(np.int32), (np.concatenate(kept) * 16).astype(np.int32)
    N = 16 * rows
    data, bias, X = util.weights(5, (len(ro), 256)), util.weights(6, (N,), 0.05), util.activations(7, (T, K))
    w = et.TileWeight(K, N, 32768, data, rp, ro, bias, is_gelu=gelu)
    info = w.info()
    assert info["stage_bytes"] == info["stages"] == 0, info   # the resident form
    Y = w.run(torch.full((T, N), float("nan"), dtype=torch.float16, device="cuda"), dev(X))
    torch.cuda.synchronize()
    w.check()
    part = slice(max(0, T - 140), T)
    util.assert_close(host(Y)[part], orc.tile_linear(X[part], rp, ro, data, bias, N, gelu=gelu), what=f"{full} full block-rows")


@pytest.mark.parametrize("K,rows,full,gelu", [(768, 144, (0, 1, 2, 3, 143), False), (1024, 192, (0, 5, 100, 190, 191), True)])
def test_resident_linear_of_several_items_to_a_cta(et, orc, K, rows, full, gelu):
    """20000 tokens are three or four items to a CTA: rings, parities and the turn of the sets go on from one to the next, with groups cut into blocks and
    block-rows without tiles among them. Every element is written, and repeated calls give the same bits."""
    T, N = 20000, 16 * rows
    rng = np.random.default_rng(K + T)
    kept = [np.arange(K // 16) if r in full else np.sort(rng.choice(K // 16, rng.integers(0, K // 96), replace=False)) for r in range(rows)]
    rp = np.concatenate([[0], np.cumsum([len(k) for k in kept])]).astype(np.int32)
    ro = (np.concatenate(kept) * 16).astype(np.int32)
    data, bias, X = util.weights(3, (len(ro), 256)), util.weights(4, (N,), 0.05), util.activations(5, (T, K))
    w = et.TileWeight(K, N, 32768, data, rp, ro, bias, is_gelu=gelu)
    info = w.info()
    assert info["stage_bytes"] == info["stages"] == 0, info   # the resident form
    Y, again = (w.run(torch.full((T, N), float("nan"), dtype=torch.float16, device="cuda"), dev(X)) for _ in range(2))
    torch.cuda.synchronize()
    w.check()
    assert torch.isfinite(Y).all() and torch.equal(Y, again)
    for first in (0, 128 * 49 - 70, 128 * 99 - 70, T - 140):   # two of them where CTAs pass on to their next item
        part = slice(first, first + 140)
        util.assert_close(host(Y[part]), orc.tile_linear(X[part], rp, ro, data, bias, N, gelu=gelu), what=f"{full} full block-rows, tokens from {first}")


def test_tile_linear_pruned_tiles_do_not_contribute(et, orc):
    """Mask exactness: output equals the dense product with the pruned tiles zeroed, and does not
    change when garbage is placed where the pruned tiles would be."""
    T, K, N = 128, 256, 64
    rp, ro, data, bias = util.make_tile_linear(orc, K, N, 0.5, seed=4)
    W = orc.bsr_to_dense(rp, ro, data, N, K)
    X = util.activations(5, (T, K))
    w = et.TileWeight(K, N, T, data, rp, ro, bias)
    Y = torch.zeros((T, N), dtype=torch.float16, device="cuda")
    w.run(Y, dev(X))
    torch.cuda.synchronize()
    w.check()
    want = X.astype(np.float32) @ W.T
    util.assert_close(host(Y), want, what="tile linear vs masked dense")


def test_tile_linear_matches_reference_kernel(et, orc, ref):
    T, K, N = 768, 768, 768
    for gelu in (0, 1):
        rp, ro, data, bias = util.make_tile_linear(orc, K, N, 0.5, seed=31, bias_std=0.05)
        X = util.activations(32, (T, K))
        want = orc.tile_linear(X, rp, ro, data, bias, N, gelu=bool(gelu))
        Yr = torch.zeros((T, N), dtype=torch.float16, device="cuda")
        Xd, rpd, rod, dd, bd = dev(X), dev(rp), dev(ro), dev(data), dev(bias)
        rc = ref.ref_tile_spmm(_p(Yr), _p(Xd), _p(rpd), _p(rod), _p(dd), T, N, K, _p(bd), gelu, None)
        torch.cuda.synchronize()
        assert rc == 0
        util.assert_close(host(Yr), want, max_abs=4e-2, mean_abs=4e-3, what="reference tile GEMM vs oracle")
        w = et.TileWeight(K, N, T, data, rp, ro, bias)
        Y = torch.zeros((T, N), dtype=torch.float16, device="cuda")
        w.run(Y, Xd, gelu=bool(gelu))
        torch.cuda.synchronize()
        util.assert_close(host(Y), host(Yr), max_abs=4e-2, mean_abs=4e-3, what="new vs reference tile GEMM")


def test_tile_spmm_raw_launcher(et, orc):
    T, K, N = 256, 768, 768
    rp, ro, data, bias = util.make_tile_linear(orc, K, N, 0.75, seed=41, bias_std=0.05)
    X = util.activations(42, (T, K))
    want = orc.tile_linear(X, rp, ro, data, bias, N)
    Y = torch.zeros((T, N), dtype=torch.float16, device="cuda")
    drp, dro, dd, db = dev(rp), dev(ro), dev(data), dev(bias)
    for _ in range(2):   # second call hits the packed-weight cache
        et.tile_spmm_bias(Y, dev(X), drp, dro, dd, db, K=K)
        torch.cuda.synchronize()
        util.assert_close(host(Y), want, what="raw tile launcher")
    et.tile_spmm_cache_clear()


@pytest.mark.parametrize("T,K,N,sparsity,form", [(128, 3072, 768, 0.0, "shares"), (4096, 768, 768, 0.0, "pairs"), (32768, 768, 2304, 0.75, "resident"),
                                                 (17792, 3072, 768, 0.75, "tile")])
def test_tile_spmm_bias_may_be_the_preceding_kernels_result(et, orc, T, K, N, sparsity, form):
    """The caller's bias is read in the order of the stream: a LayerNorm of one long row, which lets the next kernel start at once
    and ends long after, writes it right before the call."""
    rp, ro, data, bias = util.make_tile_linear(orc, K, N, sparsity, T + K, bernoulli=True)
    info = et.TileWeight(K, N, T, data, rp, ro, bias).info()
    assert form == ("tile" if info["stage_bytes"] else "resident" if not info["stages"] else "shares" if info["stages"] > 1 else "pairs"), info
    drp, dro, dd, X = dev(rp), dev(ro), dev(data), dev(util.activations(7, (T, K)))
    size = 60001
    before, s = (torch.randn((1, size), device="cuda").half() for _ in range(2))
    g, b = torch.full((size,), 3.0, device="cuda").half(), torch.ones(size, device="cuda").half()
    row = before.clone()
    at = (size - N) // 8 * 8
    Y, want = (torch.full((T, N), float("nan"), dtype=torch.float16, device="cuda") for _ in range(2))
    et.tile_spmm_bias(Y, X, drp, dro, dd, row[0, at:at + N], K=K)   # (the weight is packed here)
    torch.cuda.synchronize()
    try:
        for _ in range(3):
            row.copy_(before)
            torch.cuda.synchronize()
            et.skip_layernorm(row, s, g, b)
            et.tile_spmm_bias(Y, X, drp, dro, dd, row[0, at:at + N], K=K)
            torch.cuda.synchronize()
            assert not torch.equal(row, before)
            et.tile_spmm_bias(want, X, drp, dro, dd, row[0, at:at + N], K=K)
            torch.cuda.synchronize()
            assert torch.equal(Y, want)
    finally:
        et.tile_spmm_cache_clear()


def test_tile_weight_rejects_malformed_format(et):
    data = np.zeros((2, 256), dtype=np.float16)
    ok_rp = np.array([0, 1, 2], dtype=np.int32)
    with pytest.raises(et.EtError):   # offset not a multiple of 16
        et.TileWeight(64, 32, 128, data, ok_rp, np.array([8, 16], dtype=np.int32))
    with pytest.raises(et.EtError):   # offset beyond in_feat
        et.TileWeight(64, 32, 128, data, ok_rp, np.array([0, 64], dtype=np.int32))
    with pytest.raises(et.EtError):   # row_ptr does not end at ntile
        et.TileWeight(64, 32, 128, data, np.array([0, 1, 1], dtype=np.int32), np.array([0, 16], dtype=np.int32))
    with pytest.raises(et.EtError):   # not monotone
        et.TileWeight(64, 48, 128, data, np.array([0, 2, 1, 2], dtype=np.int32), np.array([0, 16], dtype=np.int32))
    with pytest.raises(et.EtError):   # features not multiples of 16
        et.TileWeight(60, 32, 128, data, ok_rp, np.array([0, 16], dtype=np.int32))
