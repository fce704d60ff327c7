"""The persistent decode kernel (launches of many pages that leave the split to the library) against the chunked one, which
takes any call with an explicit chunk_pages and is held to the oracle in test_gpu_decode.py, and against the oracle.

Both kernels round the softmax weights times the value norm to fp16 once (relative 2^-11 each, independent) and the
output to the io type: two outputs differ by at most 2 * 2^-11 of the weighted sum of |v| and one rounding of the output."""
import math

import pytest
import torch

from tests.test_gpu_decode import DEV, assert_attn_close, oracle_decode, random_fields
from turboquant.core.codebook import make_codebook
from turboquant.kernels import _native, paged_layout
from turboquant.kernels.paged import CacheFormat, Codebooks, paged_decode_attention

pytestmark = pytest.mark.gpu

RAGGED = [8192 + 5, 0, 1, 16, 17, 700, 15, 4000]              # 513 pages wide: sizes the launch, few pages in fact
SHORT_TOTAL = [8200, 3, 3, 3, 3, 3, 3, 3]                     # fewer pages than warps: empty shares
MANY_ITEMS = [64 + i % 40 for i in range(600)] + [2100]       # several whole items inside one warp's share


def _random_cache(fmt, blocks, hkv, bs, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    L = fmt.layout
    pages = torch.randint(0, 256, (blocks, hkv, bs // 16, L.page_bytes), dtype=torch.uint8, device=DEV, generator=g)
    norms = lambda lo, hi: (torch.rand(blocks, hkv, bs // 16, 16, device=DEV, generator=g) * (hi - lo) + lo).half().view(torch.uint8)
    pages[..., L.k_norm_offset:L.k_norm_offset + 32] = norms(8, 12)
    if fmt.use_qjl:
        pages[..., L.k_rnorm_offset:L.k_rnorm_offset + 32] = norms(0, 3)
    pages[..., L.v_norm_offset:L.v_norm_offset + 32] = norms(8, 12)
    return pages.reshape(blocks, hkv, -1)


def _tables(lens, bs, seed):
    blocks = [-(-n // bs) for n in lens]
    perm = torch.randperm(sum(blocks), generator=torch.Generator().manual_seed(seed)).int()
    bt = torch.zeros(len(lens), max(blocks), dtype=torch.int32)
    o = 0
    for i, n in enumerate(blocks):
        bt[i, :n] = perm[o:o + n]
        o += n
    return bt, sum(blocks)


@pytest.mark.parametrize("kb,vb,qjl", [(2, 2, True), (3, 3, True), (4, 4, False), (4, 3, False), (3, 2, True), (2, 4, True), (4, 4, True)])
@pytest.mark.parametrize("lens,hq,hkv,bs,dtype", [(RAGGED, 32, 4, 16, torch.float16), (SHORT_TOTAL, 24, 2, 32, torch.bfloat16),
                                                  (MANY_ITEMS, 4, 1, 16, torch.float16)])
def test_persistent_matches_chunked(kb, vb, qjl, lens, hq, hkv, bs, dtype):
    fmt = CacheFormat(kb, vb, qjl)
    books = Codebooks(fmt, DEV)
    bt, blocks = _tables(lens, bs, kb + vb)
    cache = _random_cache(fmt, blocks, hkv, bs, kb * 7 + vb)
    g = torch.Generator(device=DEV).manual_seed(1)
    q = torch.randn(len(lens), hq, 128, generator=g, device=DEV, dtype=dtype)
    args = (q, cache, bt.to(DEV), torch.tensor(lens, dtype=torch.int32, device=DEV), books, bs)
    eps = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8
    for kw in (dict(), dict(rotate_q=True, derotate_out=True), dict(q_proj=q.flip(0).contiguous())):
        want = paged_decode_attention(*args, chunk_pages=64, **kw).float()
        got = paged_decode_attention(*args, **kw).float()
        assert _native.read_status(DEV) == 0
        assert (got[want == 0] == 0).all()                    # empty sequences
        # |v| <= 12 * max |centroid|, which the de-rotation spreads over dims without growing it by more than sqrt(128)
        bound = 2 * 2.0 ** -11 * 12 * books.vc.abs().max().item() * (math.sqrt(128) if kw.get("derotate_out") else 1)
        assert ((got - want).abs() <= bound + 2 * eps * want.abs()).all(), (got - want).abs().max()
        assert (got - want).norm() <= 4 * eps * want.norm()


def test_persistent_matches_oracle_and_flags_bad_tables():
    fmt = CacheFormat.named("turbo3")
    books = Codebooks(fmt, DEV)
    lens = [16384 + 5, 0, 40, 16, 17, 700, 15, 1]
    bt, blocks = _tables(lens, 16, 3)
    f = random_fields(fmt, blocks, 16, 2, 5)
    cache = paged_layout.pack_cache(f, 16, 3, 3, True).to(DEV)
    q = torch.randn(8, 16, 128, generator=torch.Generator().manual_seed(2)).half()
    sm, cs = 1 / math.sqrt(128), math.sqrt(math.pi / 2) / 128
    lens_t = torch.tensor(lens, dtype=torch.int32)
    ref = oracle_decode(q, None, f, fmt, books, bt, lens_t, sm, cs, 16)
    stats = torch.zeros(2, dtype=torch.int32, device=DEV)
    for kw in (dict(), dict(sparse_thresh=1e-6, skip_stats=stats)):
        out = paged_decode_attention(q.to(DEV), cache, bt.to(DEV), lens_t.to(DEV), books, 16, sm, cs, **kw)
        assert _native.read_status(DEV) == 0
        assert_attn_close(out.float().cpu().numpy(), ref)
    assert stats[0].item() == 2 * sum(-(-n // 16) for n in lens)
    bad = bt.clone()
    bad[5, 3] = blocks + 7
    paged_decode_attention(q.to(DEV), cache, bad.to(DEV), lens_t.to(DEV), books, 16, sm, cs)
    assert _native.read_status(DEV) == _native.STATUS_BAD_BLOCK
    cut = lens_t.clone()
    cut[0] = 17000                                            # beyond the table: cut to its width and flagged
    out = paged_decode_attention(q.to(DEV), cache, bt.to(DEV), cut.to(DEV), books, 16, sm, cs)
    assert _native.read_status(DEV) == _native.STATUS_BAD_BLOCK
    assert_attn_close(out[1:].float().cpu().numpy(), ref[1:])


@pytest.mark.parametrize("ns,live", [(701, 40), (2500, 33), (150, 0)])
def test_padded_batches(ns, live):
    """Batches of mostly empty sequences: zeros wherever nothing is attended to, more sequences than warps among them."""
    fmt = CacheFormat.named("turbo4")
    books = Codebooks(fmt, DEV)
    lens = [1700] * live + [0] * (ns - live)
    lens = [lens[(7 * i) % ns] for i in range(ns)]                # 7 divides no ns: a permutation
    bt, blocks = _tables(lens + [2000], 16, 4)                    # the table is wide though every sequence may be empty
    cache = _random_cache(fmt, blocks, 4, 16, 8)
    q = torch.randn(ns, 20, 128, generator=torch.Generator(device=DEV).manual_seed(1), device=DEV).half()
    lens_t = torch.tensor(lens, dtype=torch.int32, device=DEV)
    args = (q, cache, bt[:ns].contiguous().to(DEV), lens_t, books, 16)
    got = paged_decode_attention(*args, out=torch.full_like(q, float("nan")))
    assert _native.read_status(DEV) == 0
    assert (got[lens_t == 0] == 0).all()
    if live:
        some = (lens_t > 0).nonzero()[:, 0]
        want = paged_decode_attention(q[some], cache, args[2][some].contiguous(), lens_t[some].contiguous(), books, 16, chunk_pages=64)
        bound = 2 * 2.0 ** -11 * 12 * books.vc.abs().max().item()
        assert ((got[some].float() - want.float()).abs() <= bound + 2.0 ** -10 * want.float().abs()).all()


@pytest.mark.parametrize("G", [1, 4, 6, 8, 12])
@pytest.mark.parametrize("chunk", [0, 256])
def test_sparse_v_skips_for_every_group_size(G, chunk):
    """Groups of fewer than eight heads, and the last four of twelve: the zero queries that fill up the tile must not keep
    pages.  chunk 0 runs the persistent kernel, 256 pages the chunked one."""
    fmt = CacheFormat.named("turbo3")
    books = Codebooks(fmt, DEV)
    lens = [32768, 16384 + 5] * 8
    bt, blocks = _tables(lens, 16, 9)
    cache = _random_cache(fmt, blocks, 2, 16, 11)
    q = torch.randn(16, 2 * G, 128, generator=torch.Generator(device=DEV).manual_seed(3), device=DEV).half() * 12
    args = (q, cache, bt.to(DEV), torch.tensor(lens, dtype=torch.int32, device=DEV), books, 16)
    stats = torch.zeros(2, dtype=torch.int32, device=DEV)
    got = paged_decode_attention(*args, sparse_thresh=1e-6, skip_stats=stats, chunk_pages=chunk).float()
    want = paged_decode_attention(*args, chunk_pages=chunk).float()
    assert _native.read_status(DEV) == 0
    seen, skipped = stats.tolist()
    assert seen == 2 * -(-G // 8) * 8 * (2048 + 1025) and 0 < skipped < seen
    # as above: the skipped weights add up to at most 1e-6 of the maximum for each of 32768 tokens, times |v|
    bound = (2 * 2.0 ** -11 + 32768e-6) * 12 * books.vc.abs().max().item()
    assert ((got - want).abs() <= bound + 2.0 ** -10 * want.abs()).all()


@pytest.mark.parametrize("kw", [dict(), dict(chunk_pages=64), dict(chunk_pages=2048), dict(tcgen05=True)])
@pytest.mark.parametrize("length", [2 ** 31 - 1, 2 ** 31 - 16, 2 ** 31 - 17])
def test_lengths_near_2_31_are_cut_and_flagged(kw, length):
    """Such an entry is cut to the table's width like any other that is too long, and its neighbours are untouched."""
    fmt = CacheFormat.named("turbo3")
    books = Codebooks(fmt, DEV)
    lens = [40, 16384, 0, 700, 1, 33]
    bt, blocks = _tables(lens, 16, 3)                         # 1024 pages wide
    f = random_fields(fmt, blocks, 16, 4, 6)
    cache = paged_layout.pack_cache(f, 16, 3, 3, True).to(DEV)
    q = torch.randn(6, 32, 128, generator=torch.Generator().manual_seed(2)).half().to(DEV)
    bt, good = bt.to(DEV), torch.tensor(lens, dtype=torch.int32, device=DEV)
    want = paged_decode_attention(q, cache, bt, good, books, 16, **kw)
    assert _native.read_status(DEV) == 0
    bad = good.clone()
    bad[1] = length
    got = paged_decode_attention(q, cache, bt, bad, books, 16, **kw)
    assert _native.read_status(DEV) == _native.STATUS_BAD_BLOCK
    assert torch.equal(got, want)


def test_persistent_sparse_v_skips_and_stays_close():
    """A peaked softmax over long sequences: V parts are left in memory, the result is the dense one within the threshold."""
    fmt = CacheFormat.named("turbo3")
    books = Codebooks(fmt, DEV)
    lens = [32768, 16384 + 5] * 8                             # about 40 pages a warp: the first four always come whole
    bt, blocks = _tables(lens, 16, 9)
    cache = _random_cache(fmt, blocks, 4, 16, 11)
    q = torch.randn(16, 32, 128, generator=torch.Generator(device=DEV).manual_seed(3), device=DEV).half() * 12
    args = (q, cache, bt.to(DEV), torch.tensor(lens, dtype=torch.int32, device=DEV), books, 16)
    stats = torch.zeros(2, dtype=torch.int32, device=DEV)
    got = paged_decode_attention(*args, sparse_thresh=1e-6, skip_stats=stats).float()
    want = paged_decode_attention(*args, chunk_pages=256).float()
    assert _native.read_status(DEV) == 0
    seen, skipped = stats.tolist()
    assert seen == 8 * 4 * (2048 + 1025) and 0 < skipped < seen
    # the skipped weights add up to at most 1e-6 of the maximum for each of 32768 tokens, times |v|
    bound = (2 * 2.0 ** -11 + 32768e-6) * 12 * books.vc.abs().max().item()
    assert ((got - want).abs() <= bound + 2.0 ** -10 * want.abs()).all()


def _attend64(q, qp, cache, blocks, books, bs, n, hkv):
    """Attention of one sequence in 64 bits: q, qp [hkv, G, 128] of the rotated domain, its first n tokens in `blocks` of the cache."""
    fmt = books.fmt
    f = paged_layout.unpack_cache(cache[blocks.long().to(DEV)], bs, fmt.k_bits, fmt.v_bits, fmt.use_qjl)
    rows = lambda name, h: f[name].flatten(0, 1)[:n, h].double()
    out = []
    for h in range(hkv):
        s = q[h].double() @ (books.kc.double()[rows("k_idx", h).long()] * rows("k_norm", h)[:, None]).T
        if fmt.use_qjl:
            s += qp[h].double() @ ((2 * rows("k_signs", h) - 1) * rows("k_rnorm", h)[:, None]).T * (math.sqrt(math.pi / 2) / 128)
        out.append(torch.softmax(s / math.sqrt(128), -1) @ (books.vc.double()[rows("v_idx", h).long()] * rows("v_norm", h)[:, None]))
    return torch.stack(out)


def _uneven_rows(*shape, g):
    """Query rows of eight kinds: one coordinate up to 100 times as large as the others, subnormal ones (fp16), constant, zero, one-hot."""
    q = torch.randn(*shape, 8, 128, generator=g, device=DEV)
    for head, factor in ((1, 10), (2, 30), (3, 100)):
        q[..., head, 17] *= factor
    q[..., 4, :] *= 1e-6
    q[..., 5, :] = 0.7
    q[..., 6:, :] = 0
    q[..., 7, 90] = -3
    return q


def _offset_rows(*shape, g):
    """Rows with an offset: after the rotation one coordinate is up to 110 times as large as the others."""
    return torch.randn(*shape, 8, 128, generator=g, device=DEV) + torch.tensor([0, 0.3, 1, 3, 10, -1, -3, -10], device=DEV)[:, None]


UNEVEN_BOOK = (torch.tensor([-0.5, -0.02, -0.009, -0.002, 0.003, 0.011, 0.025, 0.4]), torch.linspace(-0.1, 0.1, 7))
LONG = [24576 + 5, 4000, 700, 3000, 5001, 2000, 333, 8000]   # with four KV heads three times the pages the persistent kernel asks for


@pytest.mark.parametrize("kb,vb,qjl,form,dtype", [
    (3, 3, True, "", torch.float16), (3, 3, True, "rotate", torch.float16), (3, 3, True, "rotate", torch.bfloat16),
    (3, 3, True, "q_proj", torch.float16), (3, 2, True, "q_proj", torch.bfloat16), (3, 3, True, "uneven book", torch.float16),
    (3, 4, False, "", torch.float16), (3, 4, False, "uneven book", torch.bfloat16), (2, 2, True, "rotate", torch.float16),
    (4, 4, False, "", torch.float16)])
def test_scores_of_uneven_queries(kb, vb, qjl, form, dtype):
    """No kind of query row or codebook may cost the persistent kernel precision: against 64 bits it is as close as the chunked one.
    Both round the operands and the output alike; what differs is the fp16 rounding of the weights, about 1e-4 (2-norm), which the
    chunked kernel may be spared (a weight of exactly 1), next to 2.4e-4 or more of the shared ones: a factor of 1.09 at most.
    A row with NaN or infinity gives NaN and leaves the others as they are, in either query."""
    fmt = CacheFormat(kb, vb, qjl)
    books = Codebooks(fmt, DEV, k_codebook=UNEVEN_BOOK if form == "uneven book" else None)
    ns, hkv = len(LONG), 4
    bt, blocks = _tables(LONG, 16, 6)
    cache = _random_cache(fmt, blocks, hkv, 16, 5)
    g = torch.Generator(device=DEV).manual_seed(2)
    make = lambda: (_offset_rows if form == "rotate" else _uneven_rows)(ns, hkv, g=g).reshape(ns, hkv * 8, 128).to(dtype)
    kw = dict(q=make(), q_proj=make() if form == "q_proj" else None, rotate_q=form == "rotate")
    common = dict(cache=cache, block_tables=bt.to(DEV), seq_lens=torch.tensor(LONG, dtype=torch.int32, device=DEV), books=books, block_size=16)
    call = lambda **more: paged_decode_attention(**{**common, **kw, **more})
    got, chunked = call(), call(chunk_pages=64)
    assert _native.read_status(DEV) == 0
    assert not torch.equal(got, chunked)                      # two kernels, then
    q = (_native.wht_rows(kw["q"]) if kw["rotate_q"] else kw["q"]).view(ns, hkv, 8, 128)
    qp = q if kw["q_proj"] is None else kw["q_proj"].view(ns, hkv, 8, 128)
    ref = torch.stack([_attend64(q[i], qp[i], cache, bt[i, :-(-n // 16)], books, 16, n, hkv) for i, n in enumerate(LONG)])
    error = lambda x: (x.double().view(ref.shape) - ref).pow(2).sum(dim=(0, 1, 3)).sqrt()
    assert (error(got) <= 1.1 * error(chunked)).all(), (error(got) / error(chunked))
    # What Sparse-V leaves out below 1e-9 rounds to zero in fp16 (value norms are at most 12): the same arithmetic, the same output.
    assert torch.equal(call(sparse_thresh=1e-9), got)
    for name in ("q", "q_proj"):
        for bad in (float("nan"), float("inf")):
            if kw[name] is None:
                continue
            dirty = kw[name].clone()
            dirty[0, 9, 5] = bad
            out = call(**{name: dirty})
            assert out[0, 9].isnan().all()
            out[0, 9] = got[0, 9]
            assert torch.equal(out, got)


@pytest.mark.parametrize("kb,vb", [(2, 2), (3, 3), (4, 4)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("kw", [dict(), dict(chunk_pages=64), dict(chunk_pages=64, sparse_thresh=1e-6), dict(sparse_thresh=1e-9)])
@pytest.mark.parametrize("separate", [False, True])
def test_sign_term_of_large_queries(kb, vb, dtype, kw, separate):
    """Coordinates on both sides of 511, where rows begin to be divided, at each of the four dims of a quarter that the sign term scales by
    2^7; far larger ones at others; a row of many: no overflow to NaN, no place treated wrongly.
    The scores reach thousands, so one rounding in 32 bits moves a weight by up to 5e-4; next to that weights and output are rounded
    to 11 bits (bf16: the output to 8).  Without a split Sparse-V runs the persistent kernel on sequences four times as long, 20 pages a warp,
    of which all but the first four can come without their V part (4000 of 47624 pages and more do); what is left out adds up to 1e-9 for each
    of 98324 tokens at most."""
    fmt = CacheFormat(kb, vb, True)
    c, b = make_codebook(128, kb)
    books = Codebooks(fmt, DEV, k_codebook=(c.half().float(), b))   # fp16 operands: rounding a centroid moves a score of thousands by more
    skips = "sparse_thresh" in kw and "chunk_pages" not in kw
    lens = [4 * n for n in LONG] if skips else LONG
    ns, hkv = len(lens), 4
    bt, blocks = _tables(lens, 16, 6)
    cache = _random_cache(fmt, blocks, hkv, 16, 5)
    g = torch.Generator(device=DEV).manual_seed(2)

    def make():
        q = torch.randn(ns, hkv, 8, 128, generator=g, device=DEV)
        if skips:
            q *= 100                                          # a softmax so peaked that many pages weigh nothing in any row
        for head, dim, value in ((1, 4, 508), (2, 32 + 12, 511.5), (3, 64 + 20, -512), (4, 96 + 28, 1000), (5, 18, 30000), (6, 16, -40000)):
            q[:, :, head, dim] = value
        q[:, :, 7] *= 4 if skips else 400
        return q.to(dtype)

    q = make()
    qp = make() if separate else q
    stats = torch.zeros(2, dtype=torch.int32, device=DEV)
    out = paged_decode_attention(q.view(ns, -1, 128), cache, bt.to(DEV), torch.tensor(lens, dtype=torch.int32, device=DEV), books, 16,
                                 q_proj=qp.view(ns, -1, 128) if separate else None, skip_stats=stats, **kw)
    assert _native.read_status(DEV) == 0
    if skips:
        seen, skipped = stats.tolist()
        assert seen == hkv * sum(-(-n // 16) for n in lens) and skipped > seen // 25, (seen, skipped)
    ref = torch.stack([_attend64(q[i], qp[i], cache, bt[i, :-(-n // 16)], books, 16, n, hkv) for i, n in enumerate(lens)])
    error = (out.double().view(ref.shape) - ref).pow(2).sum(dim=(0, 1, 3)).sqrt() / ref.pow(2).sum(dim=(0, 1, 3)).sqrt()
    assert (error <= (2e-3 if dtype == torch.float16 else 4e-3)).all(), error


@pytest.mark.parametrize("fmt,hq", [((2, 2, True), 16), ((3, 3, True), 64), ((4, 4, False), 32), ((4, 4, True), 8)])
@pytest.mark.parametrize("kw", [dict(), dict(rotate_q=True, derotate_out=True), dict(sparse_thresh=1e-9)])
def test_more_partials_than_shared_memory_keeps(fmt, hq, kw):
    """Sequences of one and a half shares: in every CTA about ten items end inside a share they did not start, more than shared memory has
    room for in the wider formats.  Both kernels round the weights (2-norm 1e-4) and the output (2.8e-4) to fp16 on their own."""
    fmt = CacheFormat(*fmt)
    books = Codebooks(fmt, DEV)
    lens = [370 + 7 * (i % 5) for i in range(197)]
    bt, blocks = _tables(lens, 16, 9)
    cache = _random_cache(fmt, blocks, 8, 16, 10)
    q = torch.randn(len(lens), hq, 128, generator=torch.Generator(device=DEV).manual_seed(11), device=DEV).half()
    call = lambda **more: paged_decode_attention(q, cache, bt.to(DEV), torch.tensor(lens, dtype=torch.int32, device=DEV), books, 16, **kw, **more)
    got, chunked = call().float(), call(chunk_pages=64).float()
    assert _native.read_status(DEV) == 0
    assert not torch.equal(got, chunked)
    rows = (got - chunked).pow(2).sum(-1).sqrt() / chunked.pow(2).sum(-1).sqrt()
    assert rows.max() < 2e-3 and rows.pow(2).mean().sqrt() < 8e-4, (rows.max(), rows.pow(2).mean().sqrt())


@pytest.mark.parametrize("value", [500.0, 511.0, 512.0, 65000.0])
@pytest.mark.parametrize("kw", [dict(), dict(chunk_pages=64)])
def test_sign_operands_at_the_edge_of_fp16(value, kw):
    """The sign term scales the query by 2^7 at dims 4, 12, 20 and 28 of a quarter and by less up to 1 at the next seven: rows are divided from
    511 on, and no place overflows.  Weights and output are rounded to 11 bits, scores of thousands to 2^-12 in 32 bits."""
    fmt, hkv, n = CacheFormat(3, 3, True), 4, 24576 + 5
    books = Codebooks(fmt, DEV)
    lens = [n, 3000, 8000, 5000]
    bt, blocks = _tables(lens, 16, 6)
    cache = _random_cache(fmt, blocks, hkv, 16, 5)
    q = torch.randn(len(lens), hkv, 8, 128, generator=torch.Generator(device=DEV).manual_seed(3), device=DEV)
    for head, dim in enumerate((4, 12, 20, 28, 11, 32 + 19, 64 + 27, 96 + 3)):
        q[:, :, head, dim] = value if head & 1 else -value
    q = q.half()
    out = paged_decode_attention(q.view(len(lens), -1, 128), cache, bt.to(DEV), torch.tensor(lens, dtype=torch.int32, device=DEV), books, 16, **kw)
    assert _native.read_status(DEV) == 0
    ref = torch.stack([_attend64(q[i], q[i], cache, bt[i, :-(-m // 16)], books, 16, m, hkv) for i, m in enumerate(lens)])
    error = (out.double().view(ref.shape) - ref).pow(2).sum(dim=(0, 1, 3)).sqrt() / ref.pow(2).sum(dim=(0, 1, 3)).sqrt()
    assert (error <= 2e-3).all(), error


@pytest.mark.parametrize("fmt", [(4, 4, False), (3, 3, True), (2, 2, True), (4, 3, False)])
@pytest.mark.parametrize("ns,persistent", [(31, False), (32, True)])
def test_which_kernel_takes_a_batch(fmt, ns, persistent):
    """1024 tokens and 8 KV heads: below 16384 pages the chunked kernel runs as if its split had been asked for, from there the persistent
    one, with the workspace that the host path names.  Both round the weights (2-norm 1e-4) and the output (2.8e-4) to fp16 on their own."""
    fmt = CacheFormat(*fmt)
    books = Codebooks(fmt, DEV)
    lens = [1024 - 37 * (i % 4) for i in range(ns)]
    bt, blocks = _tables(lens, 16, 9)
    cache = _random_cache(fmt, blocks, 8, 16, 10)
    q = torch.randn(ns, 32, 128, generator=torch.Generator(device=DEV).manual_seed(11), device=DEV).half()
    call = lambda **kw: paged_decode_attention(q, cache, bt.to(DEV), torch.tensor(lens, dtype=torch.int32, device=DEV), books, 16, **kw)
    got, chunked = call(), call(chunk_pages=_native.lib().tq_decode_auto_chunk_pages(ns, 8, 32, 64))
    assert _native.read_status(DEV) == 0
    assert torch.equal(got, chunked) != persistent
    rows = (got.float() - chunked.float()).pow(2).sum(-1).sqrt() / chunked.float().pow(2).sum(-1).sqrt()
    assert rows.max() < 2e-3 and rows.pow(2).mean().sqrt() < 8e-4, (rows.max(), rows.pow(2).mean().sqrt())
