"""The native host path of eager calls against the general path (torch custom ops / checked ctypes calls): same results,
and what it does not handle is declined and behaves as before."""
import math

import pytest
import torch

from turboquant.core import PolarQuantConfig, make_codebook, make_wht_matrix, polarquant_compress
from turboquant.kernels import _native
from turboquant.kernels.packed_attention import packed_attention
from turboquant.kernels.packed_compress import compress_k, compress_k_permuted, compress_v
from turboquant.kernels.paged import CacheFormat, Codebooks, allocate_cache, compress_and_scatter, paged_decode_attention

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


class _Declines:
    """Stands in for the native module: every call takes the general path."""

    def __getattr__(self, name):
        return lambda *a: None


@pytest.fixture
def general(monkeypatch):
    def call(f, *a, **k):
        with monkeypatch.context() as m:
            m.setattr(_native, "_host", _Declines())
            return f(*a, **k)
    return call


def _filled(fmt, lens, hkv, bs, dtype, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    nb = [-(-n // bs) for n in lens]
    tables = torch.zeros(len(lens), max(nb), dtype=torch.int32, device=DEV)
    perm = torch.randperm(sum(nb), generator=g, device=DEV).int()
    slots, o = [], 0
    for i, n in enumerate(lens):
        tables[i, :nb[i]] = perm[o:o + nb[i]]
        pos = torch.arange(n, device=DEV)
        slots.append(tables[i, pos // bs].long() * bs + pos % bs)
        o += nb[i]
    K = torch.randn(sum(lens), hkv, 128, generator=g, device=DEV, dtype=dtype)
    V = torch.randn(sum(lens), hkv, 128, generator=g, device=DEV, dtype=dtype)
    return allocate_cache(sum(nb), bs, hkv, fmt, DEV), tables, torch.tensor(lens, dtype=torch.int32, device=DEV), K, V, torch.cat(slots)


@pytest.mark.parametrize("fmt,dtype,bs", [(CacheFormat(2, 2, True), torch.float16, 16), (CacheFormat(3, 3, True), torch.bfloat16, 32),
                                          (CacheFormat(4, 3, False), torch.float16, 16)])
def test_paged_calls_match_the_general_path(general, fmt, dtype, bs):
    cache, tables, lens, K, V, slots = _filled(fmt, [1, 17, 900, 33], 2, bs, dtype)
    books = Codebooks(fmt, DEV)
    other = cache.clone()
    version = cache._version
    compress_and_scatter(K, V, cache, slots, books, bs)
    assert cache._version > version
    general(compress_and_scatter, K, V, other, slots, books, bs)
    assert torch.equal(cache, other)
    qkv = torch.randn(4, 8 * 128 + 64, device=DEV, dtype=dtype)
    q = qkv[:, :8 * 128].view(4, 8, 128)                         # rows of a wider projection: not contiguous
    for kw in (dict(), dict(rotate_q=True, derotate_out=True, max_seq_len=900), dict(sparse_thresh=1e-6, chunk_pages=16),
               dict(q_proj=q.contiguous().flip(0), rotate_q=True)):
        a = paged_decode_attention(q, cache, tables, lens, books, bs, **kw)
        b = general(paged_decode_attention, q, cache, tables, lens, books, bs, **kw)
        assert a.dtype == dtype and torch.equal(a, b), kw
    out = torch.empty(4, 8, 128, dtype=dtype, device=DEV)
    stats = torch.zeros(2, dtype=torch.int32, device=DEV)
    res = paged_decode_attention(q, cache, tables, lens, books, bs, sparse_thresh=1e-6, out=out, skip_stats=stats)
    assert res is out and torch.equal(out, paged_decode_attention(q, cache, tables, lens, books, bs, sparse_thresh=1e-6))
    assert stats[0].item() == 2 * (1 + 2 + 57 + 3)                # pages of both KV heads
    assert torch.equal(paged_decode_attention(q, cache, tables.long(), lens.long(), books, bs),
                       paged_decode_attention(q, cache, tables, lens, books, bs))       # converted on the general path
    assert _native.read_status(DEV) == 0


@pytest.mark.parametrize("bits", [2, 3, 4])
@pytest.mark.parametrize("n", [1, 130])
def test_contiguous_calls_match_the_general_path(general, bits, n):
    c, b = make_codebook(128, bits, device=DEV)
    h = make_wht_matrix(128, device=DEV)
    g = torch.Generator(device=DEV).manual_seed(n)
    X = torch.randn(2 * n, 128, generator=g, device=DEV)
    for x in (X, X.half(), X.half()[::2], X.double()):
        for f, a in ((compress_k, (h, None, c, b)), (compress_k_permuted, (None, None, c, b)), (compress_v, (h, c, b))):
            got, want = f(x, *a), general(f, x, *a)
            assert all(torch.equal(p, q) and p.dtype == q.dtype for p, q in zip(got, want))
    for qjl in (True, False):
        got = polarquant_compress(X.view(n, 2, 128), c, b, PolarQuantConfig(bits=bits, use_qjl=qjl), h)
        want = general(polarquant_compress, X.view(n, 2, 128), c, b, PolarQuantConfig(bits=bits, use_qjl=qjl), h)
        assert got.keys() == want.keys() and all(torch.equal(got[k], want[k]) for k in want)
    k, v = compress_k_permuted(X, h, None, c, b), compress_v(X, h, c, b)
    packed = [t.view(2, n, *t.shape[1:]) for t in (*k, *v)]
    q = torch.randn(2, 128, generator=g, device=DEV).half()
    for splits in (None, 3):
        assert torch.equal(packed_attention(q, q, *packed, c, 0.01, num_splits=splits),
                           general(packed_attention, q, q, *packed, c, 0.01, num_splits=splits))
    assert torch.equal(_native.wht_rows(X, 0.5), general(_native.wht_rows, X, 0.5))


def test_declined_inputs_behave_as_before():
    fmt = CacheFormat.named("turbo3")
    cache, tables, lens, K, V, slots = _filled(fmt, [40], 2, 16, torch.float16)
    books = Codebooks(fmt, DEV)
    with pytest.raises(RuntimeError, match="no CPU path"):
        compress_and_scatter(K.cpu(), V, cache, slots, books, 16)
    with pytest.raises(ValueError, match="share a dtype"):
        compress_and_scatter(K, V.float(), cache, slots, books, 16)
    with pytest.raises(ValueError, match="cache shape"):
        compress_and_scatter(K, V, cache, slots, books, 32)
    compress_and_scatter(K, V, cache, slots, books, 16)
    q = torch.randn(1, 8, 128, device=DEV, dtype=torch.float16)
    want = paged_decode_attention(q, cache, tables, lens, books, 16)
    with pytest.raises(ValueError, match="fp16 or bf16"):
        paged_decode_attention(q.float(), cache, tables, lens, books, 16)
    with pytest.raises(ValueError, match="multiple of kv heads"):
        paged_decode_attention(q[:, :7], cache, tables, lens, books, 16)
    with torch._subclasses.FakeTensorMode(allow_non_fake_inputs=True) as mode:
        fake = mode.from_tensor(q)
        assert type(paged_decode_attention(fake, cache, tables, lens, books, 16)).__name__ == "FakeTensor"
    traced = q.clone().requires_grad_(True)                      # autograd sees the operator
    assert torch.equal(paged_decode_attention(traced, cache, tables, lens, books, 16), want)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):                                # launches follow the current stream
        again = paged_decode_attention(q, cache, tables, lens, books, 16, chunk_pages=1, sm_scale=1 / math.sqrt(128))
    side.synchronize()
    assert (again.float() - want.float()).abs().max() <= 2e-3


@pytest.mark.parametrize("bits", [2, 3, 4])
@pytest.mark.parametrize("BH,Sk", [(1, 1), (3, 15), (2, 257), (5, 8192), (37, 1100), (150, 300), (301, 40), (149, 513)])
def test_packed_attention_work_sharing(bits, BH, Sk):
    """Rows cut by the even sharing of steps over CTAs, whole rows, several rows per CTA, tails of a step: the result of
    explicit splits, which is held to the oracle elsewhere.  Weights, values and sums are fp32 on both sides, in another
    order (2^-24 times the number of tokens, at worst); the output is rounded to fp16."""
    c, b = make_codebook(128, bits, device=DEV)
    g = torch.Generator(device=DEV).manual_seed(BH + Sk)
    r = lambda w: torch.randint(0, 256, (BH, Sk, w), generator=g, dtype=torch.uint8, device=DEV)
    norm = lambda lo, hi: (torch.rand(BH, Sk, generator=g, device=DEV) * (hi - lo) + lo).half()
    q = torch.randn(BH, 128, generator=g, device=DEV).half()
    args = (q, q, r(16 * bits), r(16), norm(0, 3), norm(8, 12), r(16 * bits), norm(8, 12), c, 0.0098)
    got = packed_attention(*args).float()
    for splits in (1, 3):
        want = packed_attention(*args, num_splits=splits).float()
        # logits reach |q| |k| ~ 11 * 12: their own rounding, 2^-24 * 132 * log2(e), moves a weight by 2^-16 of itself
        assert ((got - want).abs() <= 2.0 ** -10 * want.abs() + (2.0 ** -15 + Sk * 2.0 ** -24) * 12 * c.abs().max()).all()


@pytest.mark.parametrize("bits", [2, 3])
@pytest.mark.parametrize("BH,Sk", [(1, 129), (1, 1000), (2, 257), (16, 500), (30, 255), (74, 250), (148, 130), (148, 700), (50, 9000)])
def test_packed_attention_few_steps(bits, BH, Sk):
    """Calls of few steps: CTAs of 8 warps, one to an SM or two, whole rows or steps shared evenly."""
    test_packed_attention_work_sharing(bits, BH, Sk)


@pytest.mark.parametrize("bits", [2, 3])
@pytest.mark.parametrize("BH,Sk", [(150, 700), (180, 700), (290, 1500), (600, 200)])
def test_packed_attention_deals_whole_rows_where_they_cost_least(bits, BH, Sk):
    """Rows of some steps, about as many as CTAs run at a time: dealt out whole to CTAs of 8 warps, the arrangement of num_splits = 1."""
    c, b = make_codebook(128, bits, device=DEV)
    g = torch.Generator(device=DEV).manual_seed(BH + Sk)
    r = lambda w: torch.randint(0, 256, (BH, Sk, w), generator=g, dtype=torch.uint8, device=DEV)
    norm = lambda: torch.rand(BH, Sk, generator=g, device=DEV).half()
    q = torch.randn(BH, 128, generator=g, device=DEV).half()
    args = (q, q, r(16 * bits), r(16), norm(), norm(), r(16 * bits), norm(), c, 0.0098)
    # another arrangement adds the same fp32 weights in another order: some fp16 output of thousands differs
    assert torch.equal(packed_attention(*args), packed_attention(*args, num_splits=1))


@pytest.mark.parametrize("bits", [2, 3])
@pytest.mark.parametrize("BH,Sk", [(149, 128), (150, 600), (296, 129), (297, 128), (593, 17), (700, 500)])
def test_packed_attention_two_ctas_per_sm(bits, BH, Sk):
    """More rows than SMs: CTAs of 8 warps, two per SM, around one and two waves of them and the ends of a 128-token step."""
    test_packed_attention_work_sharing(bits, BH, Sk)


@pytest.mark.parametrize("bits", [2, 3, 4])
def test_codebook_written_on_the_stream_just_before_the_call(bits):
    """The kernel before may be the one that makes the codebook: a cast (general path) or a copy into the caller's tensors
    (native path).  Every entry point gives what it gives for a codebook that was there all along."""
    good = tuple(t.clone() for t in make_codebook(128, bits, device=DEV))
    h = make_wht_matrix(128, device=DEV)
    fmt = CacheFormat(bits, bits, bits < 4)
    cache, tables, lens, K, V, slots = _filled(fmt, [4000, 17, 900, 33], 2, 16, torch.float16)
    short, tall = tables[:2, :4].contiguous(), tables.repeat(64, 1)
    lens_short, lens_tall = torch.tensor([60, 17], dtype=torch.int32, device=DEV), lens.repeat(64)
    q = torch.randn(256, 16, 128, device=DEV, dtype=torch.float16)
    X = torch.randn(40000, 128, device=DEV, dtype=torch.float16)
    k, v = compress_k_permuted(X[:1000], h, None, *good), compress_v(X[:1000], h, *good)
    packed = [t.view(2, 500, *t.shape[1:]) for t in (*k, *v)]

    def all_calls(fresh, books, c):
        def call(f):
            fresh()
            r = f()
            return list(r.values()) if isinstance(r, dict) else list(r) if isinstance(r, tuple) else [r]
        def append(n):
            out = torch.zeros_like(cache)
            fresh()
            compress_and_scatter(K[:n], V[:n], out, slots[:n], books, 16)
            return out
        filled = append(K.shape[0])
        res = [append(64), filled]                                                    # small and persistent kernel
        res += call(lambda: paged_decode_attention(q[:2], filled, short, lens_short, books, 16))          # chunked
        res += call(lambda: paged_decode_attention(q, filled, tall, lens_tall, books, 16))                # persistent
        res += call(lambda: packed_attention(q[0, :2], q[0, :2], *packed, c[0], 0.01))
        for x in (X[:100], X):
            res += call(lambda: compress_k(x, h, None, *c)) + call(lambda: compress_v(x, h, *c))
        return res + call(lambda: polarquant_compress(X[:100], *c, PolarQuantConfig(bits=bits, use_qjl=True), h))

    want = all_calls(lambda: None, Codebooks(fmt, DEV, good, None), good)
    own = [t.clone() for t in good]
    books = Codebooks(fmt, DEV, own, None)

    def copied():
        for t in own:
            t.zero_()
        torch.empty(1 << 24, device=DEV).normal_()
        for t, g in zip(own, good):
            t.copy_(g)

    for got in (all_calls(copied, books, own), all_calls(lambda: None, books, [t.double() for t in good])):
        assert len(got) == len(want) and all(torch.equal(a, b) for a, b in zip(got, want))


def test_general_path_on_two_streams_at_once(general):
    """Partials and the records of what is split live in the workspace: calls that overlap must not share one."""
    fmt = CacheFormat.named("turbo3")
    books = Codebooks(fmt, DEV)
    lens = [700, 4000, 33, 2100] * 16
    cache, tables, lens_t, K, V, slots = _filled(fmt, lens, 2, 16, torch.float16)
    compress_and_scatter(K, V, cache, slots, books, 16)
    g = torch.Generator(device=DEV).manual_seed(3)
    q = torch.randn(64, 16, 128, generator=g, device=DEV).half()
    h, (c, b) = make_wht_matrix(128, device=DEV), make_codebook(128, 3, device=DEV)
    X = torch.randn(40 * 3000, 128, generator=g, device=DEV).half()
    packed = [t.view(40, 3000, *t.shape[1:]) for t in (*compress_k_permuted(X, h, None, c, b), *compress_v(X, h, c, b))]
    few = [t[:3].contiguous() for t in packed]
    jobs = [(lambda: paged_decode_attention(q, cache, tables, lens_t, books, 16),
             lambda: paged_decode_attention(q[:6], cache, tables[:6], lens_t[:6], books, 16)),
            (lambda: packed_attention(q[0, :1].repeat(40, 1), q[0, :1].repeat(40, 1), *packed, c, 0.01),
             lambda: packed_attention(q[0, :3], q[0, :3], *few, c, 0.01))]
    for pair in jobs:
        want = [general(f) for f in pair]
        streams = [torch.cuda.Stream(), torch.cuda.Stream()]
        torch.cuda.synchronize()
        got = [[], []]
        for _ in range(20):
            for i in (0, 1):
                with torch.cuda.stream(streams[i]):
                    got[i].append(general(pair[i]))
        torch.cuda.synchronize()
        for i in (0, 1):
            assert all(torch.equal(r, want[i]) for r in got[i])
    assert _native.read_status(DEV) == 0


def test_packed_attention_takes_a_query_and_an_output_that_start_anywhere():
    """A query at an odd offset is copied, packed K/V at one are refused; the C call accepts any output address and any
    workspace that tq_packed_attention_workspace_bytes names for the split count of tq_packed_attention_auto_splits."""
    h, (c, b) = make_wht_matrix(128, device=DEV), make_codebook(128, 3, device=DEV)
    g = torch.Generator(device=DEV).manual_seed(8)
    BH, Sk = 3, 1500
    X = torch.randn(BH * Sk, 128, generator=g, device=DEV).half()
    packed = [t.view(BH, Sk, *t.shape[1:]) for t in (*compress_k_permuted(X, h, None, c, b), *compress_v(X, h, c, b))]
    q = torch.randn(BH, 128, generator=g, device=DEV).half()

    def moved(t):
        buf = torch.empty(t.numel() + 1, dtype=t.dtype, device=DEV)
        buf[1:] = t.reshape(-1)
        return buf[1:].view(t.shape)

    want = packed_attention(q, q, *packed, c, 0.01)
    k_idx, k_signs, k_rnorm, k_norm, v_idx, v_norm = packed
    assert torch.equal(packed_attention(moved(q), moved(q), k_idx, k_signs, moved(k_rnorm), moved(k_norm), v_idx, moved(v_norm), c, 0.01), want)
    for i in (0, 1, 4):
        with pytest.raises(RuntimeError, match="bad argument"):
            packed_attention(q, q, *(moved(t) if i == j else t for j, t in enumerate(packed)), c, 0.01)
    L = _native.lib()
    splits = L.tq_packed_attention_auto_splits(BH, Sk)
    ws = torch.empty(L.tq_packed_attention_workspace_bytes(BH, splits), dtype=torch.uint8, device=DEV)
    assert ws.numel() < L.tq_packed_attention_workspace_bytes(BH, 0)
    out = torch.zeros(BH * 128 + 1, dtype=torch.float16, device=DEV)
    p = _native._ptr
    rc = L.tq_packed_attention(p(q), p(q), *(p(t) for t in packed), p(c), 0.01, BH, Sk, 3, 0, p(ws), ws.numel(), p(out[1:]),
                               _native._stream(torch.device(DEV)))
    assert rc == 0
    assert torch.equal(out[1:].view(BH, 128), packed_attention(q, q, *packed, c, 0.01, num_splits=splits))


def test_tracing_modes_and_autograd_see_the_operators():
    fmt = CacheFormat.named("turbo3")
    books = Codebooks(fmt, DEV)
    cache, tables, lens, K, V, slots = _filled(fmt, [40, 7], 2, 16, torch.float16)
    compress_and_scatter(K, V, cache, slots, books, 16)
    q, other = (torch.randn(2, 8, 128, device=DEV, dtype=torch.float16) for _ in range(2))
    attend = lambda q: paged_decode_attention(q, cache, tables, lens, books, 16)

    traced = torch.jit.trace(attend, (q,), check_trace=False)
    assert "tq_b200::decode_paged" in str(traced.graph)
    assert torch.equal(traced(other), attend(other))                       # not the result of the traced query

    class Names(torch.overrides.TorchFunctionMode):
        def __init__(self):
            super().__init__()
            self.names = []

        def __torch_function__(self, func, types, args=(), kwargs=None):
            self.names.append(str(func))
            return func(*args, **(kwargs or {}))

    with Names() as mode:
        attend(q)
        compress_and_scatter(K, V, cache, slots, books, 16)
    assert any("decode_paged" in n for n in mode.names) and any("compress_paged" in n for n in mode.names)

    proj = other.clone().requires_grad_(True)                              # no formula for its gradient: not dropped silently
    out = paged_decode_attention(q, cache, tables, lens, books, 16, q_proj=proj)
    assert out.requires_grad
    with torch.no_grad():
        assert torch.equal(out, paged_decode_attention(q, cache, tables, lens, books, 16, q_proj=proj))
    with pytest.raises(RuntimeError):
        out.float().sum().backward()
