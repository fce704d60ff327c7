"""The persistent decode kernel (launches of many pages that leave the split to the library) against the chunked one, which
takes any call with an explicit chunk_pages and is held to the oracle in test_gpu_decode.py, and against the oracle.

Both kernels round the softmax weights times the value norm to fp16 once (relative 2^-11 each, independent) and the
output to the io type: two outputs differ by at most 2 * 2^-11 of the weighted sum of |v| and one rounding of the output."""
import math

import pytest
import torch

from tests.test_gpu_decode import DEV, assert_attn_close, oracle_decode, random_fields
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


@pytest.mark.parametrize("kb,vb,qjl", [(3, 3, True), (3, 4, False), (3, 2, True)])
@pytest.mark.parametrize("separate", [False, True])
def test_integer_scores_of_uneven_queries(kb, vb, qjl, separate):
    """3-bit keys are scored in 16-bit integers scaled by the row's largest value: rows with outliers, tiny, constant and zero rows
    are no further from 64 bits than the chunked kernel's half-precision products of the same call, up to the roundings that both
    share (weights and output, 2^-11 each, which differ from one another), and a row with NaN or infinity gives NaN alone."""
    if separate and not qjl:
        pytest.skip("a query of the sign term's own")
    fmt = CacheFormat(kb, vb, qjl)
    books = Codebooks(fmt, DEV)
    lens, hkv, G = [8192 + 5, 513, 16, 1, 700, 40, 333, 1025], 4, 8
    bt, blocks = _tables(lens, 16, 6)
    cache = _random_cache(fmt, blocks, hkv, 16, 5)
    g = torch.Generator(device=DEV).manual_seed(2)
    q = torch.randn(len(lens), hkv, G, 128, generator=g, device=DEV)
    q[:, :, 1, 17] *= 30
    q[:, :, 2] *= 1e-6                                        # subnormal in fp16
    q[:, :, 3] = 0
    q[:, :, 4] = 0.7
    q[:, :, 5] = 0
    q[:, :, 5, 90] = -3
    q[:, :, 6, ::2] *= 8
    q = q.half().reshape(len(lens), hkv * G, 128)
    qp = torch.randn(q.shape, generator=g, device=DEV).half() * 2 if separate else None
    args = (q, cache, bt.to(DEV), torch.tensor(lens, dtype=torch.int32, device=DEV), books, 16)
    ref = torch.empty(q.shape, dtype=torch.float64, device=DEV)
    for i, n in enumerate(lens):
        f = paged_layout.unpack_cache(cache[bt[i, :-(-n // 16)].long().to(DEV)], 16, kb, vb, qjl)
        rows = lambda name: f[name].flatten(0, 1)[:n]
        for h in range(hkv):
            heads = slice(h * G, (h + 1) * G)
            s = q[i, heads].double() @ (books.kc.double()[rows("k_idx")[:, h].long()] * rows("k_norm")[:, h, None].double()).T
            if qjl:
                signs = (2 * rows("k_signs")[:, h].double() - 1) * rows("k_rnorm")[:, h, None].double() * math.sqrt(math.pi / 2) / 128
                s += (q if qp is None else qp)[i, heads].double() @ signs.T
            ref[i, heads] = torch.softmax(s / math.sqrt(128), -1) @ (books.vc.double()[rows("v_idx")[:, h].long()] * rows("v_norm")[:, h, None].double())
    kw = {} if qp is None else dict(q_proj=qp)
    by_head = lambda x: (x.double() - ref).reshape(len(lens), hkv, G, 128).pow(2).sum(dim=(0, 1, 3)).sqrt()
    got, half = paged_decode_attention(*args, **kw), paged_decode_attention(*args, chunk_pages=64, **kw)
    assert _native.read_status(DEV) == 0
    size = ref.reshape(len(lens), hkv, G, 128).pow(2).sum(dim=(0, 1, 3)).sqrt()
    assert (by_head(got) <= by_head(half) + 2.0 ** -11 * size).all(), (by_head(got) / size, by_head(half) / size)
    for bad in (float("nan"), float("inf")):
        q2 = q.clone()
        q2[0, 9, 5] = bad
        out = paged_decode_attention(q2, *args[1:], **kw)
        assert out[0, 9].isnan().all()
        out[0, 9] = got[0, 9]
        assert torch.equal(out, got)
