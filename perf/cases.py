"""Workloads of the TurboQuant kernels, each one pass through a public entry point.

  listed()      the workloads that are tracked
  draw(rng)     one more workload of the same ranges
  prepare()     what a user's program holds before the call (inputs, paged cache, codebooks), from a seed
  run()         one pass
  work()        bytes and operations a pass cannot do without
  tolerance()   how far two correct implementations may be apart

A workload's "kind" names the path:
  append      compress_and_scatter: new K/V of a step, or of a prefill, into the paged cache
  decode      paged_decode_attention over a filled cache
  step        both, as one layer of a decode step: append each sequence's new token, then attend
  attention   packed_attention on contiguous [BH, Sk] packed K/V
  pack        compress_k_permuted + compress_v: the producer side of `attention`
  polar       polarquant_compress with unpacked outputs

K/V are N(0, 1) with four outlier channels x10 per head, as in bench.py.
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.abspath("turboquant-amd_b200"))   # imported with the repository's root as working folder

from turboquant.core import PolarQuantConfig, make_codebook, make_wht_matrix, polarquant_compress  # noqa: E402
from turboquant.kernels.packed_attention import packed_attention  # noqa: E402
from turboquant.kernels.packed_compress import compress_k_permuted, compress_v  # noqa: E402
from turboquant.kernels.paged import (CacheFormat, Codebooks, allocate_cache, compress_and_scatter,  # noqa: E402
                                      paged_decode_attention)

DEV = "cuda:0"
D = 128
OUTLIER_CHANNELS = [5, 50, 90, 127]
DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16, "fp32": torch.float32}
ITEM = {"fp16": 2, "bf16": 2, "fp32": 4}
FORMATS = {"turbo2": (2, 2, True), "turbo3": (3, 3, True), "turbo4": (4, 4, False)}
CORR = math.sqrt(math.pi / 2) / D


def _paged(kind, fmt, **more):
    kb, vb, qjl = FORMATS[fmt]
    return dict(kind=kind, k_bits=kb, v_bits=vb, qjl=qjl, **more)


def listed():
    return [
        # The new tokens of one decode step of 64 sequences: the smallest call, made once per layer and step.
        dict(_paged("append", "turbo3", tokens=64, kv_heads=8, q_heads=64, block_size=16, dtype="fp16"),
             name="append turbo3 64"),
        # A chunked prefill of a ragged length; K and V are slices of the fused qkv projection, blocks of 32 tokens.
        dict(_paged("append", "turbo4", tokens=3001, kv_heads=8, q_heads=32, block_size=32, dtype="bf16"),
             name="append turbo4 3001 bf16"),
        # Bulk ingest of long documents: the throughput end of compression.
        dict(_paged("append", "turbo2", tokens=1 << 20, kv_heads=8, q_heads=0, block_size=16, dtype="fp16"),
             name="append turbo2 1M"),
        # One interactive user with a 4096-token context: latency.
        dict(_paged("decode", "turbo4", batch=1, lens="fixed:4096", q_heads=32, kv_heads=8, block_size=16, dtype="fp16",
                    rotate=True, sparse=False), name="decode turbo4 1x4096"),
        # Batched serving at a common length: the shape of the default benchmark.
        dict(_paged("decode", "turbo3", batch=64, lens="fixed:8192", q_heads=64, kv_heads=8, block_size=16, dtype="fp16",
                    rotate=True, sparse=False), name="decode turbo3 64x8192"),
        # Long contexts under high concurrency with the Sparse-V rule on; projections carry the rotation.
        dict(_paged("decode", "turbo3", batch=64, lens="uniform:16384:32768", q_heads=64, kv_heads=8, block_size=16,
                    dtype="fp16", rotate=False, sparse=True), name="sparse-v turbo3 64x16k-32k"),
        # A serving batch of mixed lengths: few very long sequences, many short ones.
        dict(_paged("decode", "turbo2", batch=256, lens="lognormal:4096:1.0:128:65536", q_heads=32, kv_heads=8,
                    block_size=16, dtype="fp16", rotate=True, sparse=False), name="decode turbo2 256 mixed"),
        # One layer of an engine's decode step in bf16: cache update, then attention, block tables as wide as the model length.
        dict(_paged("step", "turbo4", batch=32, lens="uniform:300:5000", q_heads=32, kv_heads=8, block_size=16, dtype="bf16",
                    rotate=True, sparse=False), name="step turbo4 32x300-5000 bf16"),
        # Contiguous attention, one query per K/V stream: a long-context batch, and a short ragged one.
        dict(kind="attention", bits=3, streams=64, tokens=32768, name="attention 3-bit 64x32768"),
        dict(kind="attention", bits=4, streams=32, tokens=1000, name="attention 4-bit 32x1000"),
        # The producer of contiguous attention: K and V of 32 heads x 32768 tokens.
        dict(kind="pack", bits=3, rows=1 << 20, dtype="fp16", name="pack 3-bit 1M"),
        # Unpacked compression for calibration and quality studies, fp32 rows as in the reference's round trip.
        dict(kind="polar", bits=3, rows=65537, qjl=True, dtype="fp32", name="polar 3-bit 65537"),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def _format(rng):
    # mostly the named formats, sometimes a wider K than V
    kb, vb, qjl = rng.choice([(2, 2, True), (3, 3, True), (3, 3, True), (4, 4, False), (4, 4, False), (4, 3, False)])
    return dict(k_bits=kb, v_bits=vb, qjl=qjl)


def draw(rng):
    kind = rng.choice(["append", "append", "decode", "decode", "decode", "step", "attention", "pack", "polar"])
    if kind == "append":
        return dict(kind=kind, **_format(rng), tokens=_log(rng, 1, 1 << 20), kv_heads=rng.choice([1, 2, 4, 8]),
                    q_heads=rng.choice([0, 32, 64]), block_size=rng.choice([16, 16, 32]), dtype=rng.choice(["fp16", "bf16"]))
    if kind in ("decode", "step"):
        kv = rng.choice([1, 2, 4, 8, 8])
        batch = _log(rng, 1, 256)
        mean = _log(rng, 64, max(64, min(32768, (12 << 20) // (batch * kv))))
        lens = rng.choice(["fixed:%d" % mean, "uniform:%d:%d" % (max(1, mean // 2), mean + mean // 2),
                           "lognormal:%d:0.7:%d:%d" % (max(1, mean * 3 // 4), max(1, mean // 16), 4 * mean)])
        return dict(kind=kind, **_format(rng), batch=batch, lens=lens, q_heads=kv * rng.choice([1, 2, 4, 6, 8, 8]), kv_heads=kv,
                    block_size=rng.choice([16, 16, 32]), dtype=rng.choice(["fp16", "bf16"]), rotate=rng.random() < 0.7,
                    sparse=kind == "decode" and rng.random() < 0.2)
    if kind == "attention":
        streams = _log(rng, 1, 256)
        return dict(kind=kind, bits=rng.choice([2, 3, 3, 4]), streams=streams,
                    tokens=_log(rng, 100, min(65536, (2 << 20) // streams)))
    if kind == "pack":
        return dict(kind=kind, bits=rng.choice([2, 3, 3, 4]), rows=_log(rng, 64, 1 << 20), dtype=rng.choice(["fp16", "bf16"]))
    return dict(kind=kind, bits=rng.choice([2, 3, 4]), rows=_log(rng, 256, 1 << 19), qjl=rng.random() < 0.7,
                dtype=rng.choice(["fp32", "fp32", "fp16"]))


# ---- inputs ------------------------------------------------------------------------------------
def _lengths(case):
    """Sequence lengths of a batch: a property of the workload, the same for every seed."""
    kind, *a = case["lens"].split(":")
    n, g = case["batch"], torch.Generator().manual_seed(1234)
    if kind == "fixed":
        return torch.full((n,), int(a[0]), dtype=torch.int64)
    if kind == "uniform":
        return torch.randint(int(a[0]), int(a[1]) + 1, (n,), generator=g, dtype=torch.int64)
    z = torch.randn(n, generator=g) * float(a[1]) + math.log(float(a[0]))
    return z.exp().clamp(float(a[2]), float(a[3])).to(torch.int64)


def _vectors(g, dtype, *shape):
    x = torch.randn(*shape, D, generator=g, device=DEV, dtype=DTYPES[dtype])
    for ch in OUTLIER_CHANNELS:
        x[..., ch] *= 10
    return x


def _format_of(case):
    return CacheFormat(case["k_bits"], case["v_bits"], case["qjl"])


def _prepare_append(case, g):
    T, H, hq, bs = case["tokens"], case["kv_heads"], case["q_heads"], case["block_size"]
    fmt = _format_of(case)
    blocks = -(-T // bs)
    if hq:      # views of one [T, (Hq + 2 Hkv) * 128] projection output, as a model's attention layer has them
        qkv = _vectors(g, case["dtype"], T, hq + 2 * H)
        k, v = qkv[:, hq:hq + H], qkv[:, hq + H:]
    else:
        k, v = _vectors(g, case["dtype"], T, H), _vectors(g, case["dtype"], T, H)
    perm = torch.randperm(blocks, generator=g, device=DEV)
    pos = torch.arange(T, device=DEV)
    return dict(key=k, value=v, cache=allocate_cache(blocks, bs, H, fmt, DEV), slots=perm[pos // bs] * bs + pos % bs,
                books=Codebooks(fmt, DEV), block_size=bs)


def _prepare_paged(case, g):
    lens, H, bs = _lengths(case), case["kv_heads"], case["block_size"]
    fmt = _format_of(case)
    books = Codebooks(fmt, DEV)
    blocks = (lens + bs - 1) // bs
    n, total = int(blocks.sum()), int(lens.sum())
    start = torch.cumsum(blocks, 0) - blocks
    perm = torch.randperm(n, generator=g, device=DEV)
    # a step's tables are as wide as the engine's longest allowed sequence; otherwise as the longest one present
    width = max(int(blocks.max()), 32768 // bs) if case["kind"] == "step" else int(blocks.max())
    col = torch.arange(width, device=DEV)
    at = start.to(DEV)[:, None] + col
    tables = torch.where(col < blocks.to(DEV)[:, None], perm[at.clamp(max=n - 1)], 0).to(torch.int32)
    seq = torch.repeat_interleave(torch.arange(case["batch"], device=DEV), lens.to(DEV), output_size=total)
    pos = torch.arange(total, device=DEV) - (torch.cumsum(lens, 0) - lens).to(DEV)[seq]
    slots = tables[seq, pos // bs].to(torch.int64) * bs + pos % bs
    cache = allocate_cache(n, bs, H, fmt, DEV)
    for a in range(0, total, 1 << 16):
        m = min(1 << 16, total - a)
        compress_and_scatter(_vectors(g, case["dtype"], m, H), _vectors(g, case["dtype"], m, H), cache, slots[a:a + m], books, bs)
    s = dict(q=torch.randn(case["batch"], case["q_heads"], D, generator=g, device=DEV, dtype=DTYPES[case["dtype"]]), cache=cache,
             tables=tables, lens=lens.to(DEV, torch.int32), books=books, block_size=bs,
             flags=dict(rotate_q=case["rotate"], derotate_out=case["rotate"], sparse_thresh=1e-6 if case["sparse"] else 0.0))
    if case["kind"] == "step":
        last = (lens - 1).to(DEV)
        s["slots"] = tables.gather(1, (last // bs)[:, None])[:, 0].to(torch.int64) * bs + last % bs
        s["key"], s["value"] = (_vectors(g, case["dtype"], case["batch"], H) for _ in range(2))
        s["flags"]["max_seq_len"] = int(lens.max())
    return s


def _prepare_attention(case, g):
    bits, n, sk = case["bits"], case["streams"], case["tokens"]
    c, b = make_codebook(D, bits, device=DEV)
    h = make_wht_matrix(D, device=DEV)
    k = compress_k_permuted(_vectors(g, "fp16", n * sk), h, None, c, b)
    v = compress_v(_vectors(g, "fp16", n * sk), h, c, b)
    q = (torch.randn(n, D, generator=g, device=DEV) * D ** -0.5 @ h).half()
    return dict(q=q, packed=[t.view(n, sk, *t.shape[1:]) for t in (*k, *v)], centroids=c)


def prepare(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    kind = case["kind"]
    if kind == "append":
        s = _prepare_append(case, g)
    elif kind in ("decode", "step"):
        s = _prepare_paged(case, g)
    elif kind == "attention":
        s = _prepare_attention(case, g)
    else:
        c, b = make_codebook(D, case["bits"], device=DEV)
        s = dict(x=_vectors(g, case["dtype"], case["rows"]), wht=make_wht_matrix(D, device=DEV), centroids=c, boundaries=b)
        if kind == "pack":
            s["v"] = _vectors(g, case["dtype"], case["rows"])
        else:
            s["config"] = PolarQuantConfig(bits=case["bits"], use_qjl=case["qjl"])
    return dict(s, kind=kind)


# ---- one pass ----------------------------------------------------------------------------------
def run(s):
    kind = s["kind"]
    if kind in ("append", "step"):
        compress_and_scatter(s["key"], s["value"], s["cache"], s["slots"], s["books"], s["block_size"])
        if kind == "append":
            return s["cache"]
    if kind in ("decode", "step"):
        out = paged_decode_attention(s["q"], s["cache"], s["tables"], s["lens"], s["books"], s["block_size"], **s["flags"])
        return out if kind == "decode" else (out, s["cache"])
    if kind == "attention":
        return packed_attention(s["q"], s["q"], *s["packed"], s["centroids"], CORR)
    if kind == "pack":
        return (compress_k_permuted(s["x"], s["wht"], None, s["centroids"], s["boundaries"]),
                compress_v(s["v"], s["wht"], s["centroids"], s["boundaries"]))
    return polarquant_compress(s["x"], s["centroids"], s["boundaries"], s["config"], s["wht"])


def work(case):
    kind = case["kind"]
    if kind in ("append", "decode", "step"):
        per_token = case["kv_heads"] * _format_of(case).bytes_per_token
        item = ITEM[case["dtype"]]
        new = case["tokens"] if kind == "append" else case["batch"] if kind == "step" else 0
        # in: K, V and the slots; out: packed records.  Rotation (7 adds a value), norm, quantisation, residual.
        bytes_ = new * (2 * case["kv_heads"] * D * item + 8 + per_token)
        flops = new * 2 * case["kv_heads"] * D * 16
        if kind != "append":
            tokens = int(_lengths(case).sum())
            rows = case["batch"] * case["q_heads"]
            bytes_ += tokens * per_token + 2 * rows * D * item + tokens // case["block_size"] * 4
            flops += 2 * tokens * case["q_heads"] * D * (3 if case["qjl"] else 2)
        return {"bytes": bytes_, "flops": flops}
    if kind == "attention":
        n = case["streams"] * case["tokens"]
        return {"bytes": n * (32 * case["bits"] + 16 + 6) + case["streams"] * D * 6, "flops": 2 * n * D * 3}
    n, item = case["rows"], ITEM[case["dtype"]]
    if kind == "pack":
        return {"bytes": n * (2 * D * item + 32 * case["bits"] + 16 + 6), "flops": n * 2 * D * 16}
    return {"bytes": n * (D * item + D * (8 + 4) + 4 + (D * 4 + 4 if case["qjl"] else 0)), "flops": n * D * 16}


def tolerance(case):
    kind = case["kind"]
    if kind in ("decode", "step"):
        # The softmax weights and the output are rounded to 11 (fp16) or, the output, to 8 (bf16) significant bits.
        return {"rel": 2e-3 if case["dtype"] == "fp16" else 1e-2, "differ": 5e-4}
    if kind == "attention":
        return {"rel": 2e-3}
    # Rotating in another order of summation moves a coordinate across a centroid boundary in at most 1e-4 of the
    # cases (a packed byte holds two to four coordinates), and an fp16 norm to its neighbour.
    if kind == "polar":
        return {"rel": 2e-3, "max": 0.99, "differ": 1e-4}
    return {"rel": 1e-3, "max": 1e-3, "differ": 5e-4}
