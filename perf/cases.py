"""The attention work whose speed is followed: what a program that uses this library has it do.

Four kinds of call, each through the public entry points:

* "cache"   a step of a serving engine over its paged KV cache: the new tokens' K/V rows are written into
            their pages (`low.kvcache_append`), then every new token attends to its sequence's cache
            (`high.flash_attn_with_kvcache`). One new token per sequence is decoding, a few are the check of
            speculated tokens, hundreds are a chunk of a long prompt.
* "packed"  sequences of different lengths packed back to back (`high.flash_attn_varlen_func`): whole prompts
            over contiguous K/V, or the mixed batch of a continuously batching engine (chunks of prompts next
            to decoding sequences) over the paged cache.
* "dense"   batched tensors of one length (`high.flash_attn_func`): prefill with or without the log-sum-exp
            output, right-padded prompts with their key-padding mask (`low.flash_attn`), and decoding over a
            contiguous cache (`start_pos`).
* "softmax" the row softmax of the math path (`low.softmax_last_dim`).

Sizes are those of the benchmark and the tests: head layouts 32/8, 32/32, 64/8, 8/8, 8/2; head sizes 128, 64 and
32; contexts up to 32768 tokens; pages of 16 tokens in the main. Lengths of the sequences of one batch are spread
evenly between `lo` and `hi` and dealt out in an order that the seed decides, so that a case's work is fixed.
"""
import math

import torch

from luma_b200 import high, low

DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}
BYTES = {"bf16": 2, "f16": 2, "f32": 4}


def _cache(name, seqs, new, lo, hi, max_len, hq=32, hkv=8, d=128, page=16, dtype="bf16"):
    return dict(name=name, kind="cache", seqs=seqs, new=new, lo=lo, hi=hi, max_len=max_len, hq=hq, hkv=hkv, d=d, page=page, dtype=dtype)


def _packed(name, seqs, ones, chunk, lo, hi, hq=32, hkv=8, d=128, page=0, dtype="bf16"):
    return dict(name=name, kind="packed", seqs=seqs, ones=ones, chunk=chunk, lo=lo, hi=hi, hq=hq, hkv=hkv, d=d, page=page, dtype=dtype)


def _dense(name, batch, s, kv, hq, hkv, d, dtype="bf16", lse=False, padded=False):
    return dict(name=name, kind="dense", batch=batch, s=s, kv=kv, hq=hq, hkv=hkv, d=d, dtype=dtype, lse=lse, padded=padded)


def listed():
    return [
        # one conversation, one token after the other: nothing but latency and launches (the table is as wide as the model's longest context)
        _cache("decode_one", 1, 1, 777, 777, 4096),
        # the decode benchmark: 64 sequences of 512 to 8192 tokens
        _cache("decode_batch", 64, 1, 512, 8192, 8192),
        # a few long documents, the wide head layout of the large model
        _cache("decode_long", 4, 1, 8192, 32768, 32768, hq=64),
        # decoding by a program that keeps its cache as contiguous tensors
        _dense("decode_contiguous", 8, 1, 4000, 32, 8, 128, dtype="f16"),
        # four speculated tokens per sequence checked at once
        _cache("speculate", 16, 4, 512, 8192, 8192),
        # 512-token chunks of four long prompts
        _cache("chunked_prefill", 4, 512, 1024, 8192, 8192),
        # one step of a continuously batching engine: chunks of four prompts next to 32 decoding sequences
        _packed("serve_mixed", 36, 32, 512, 512, 8192, page=16),
        # the small f32 problem that the CPU reference is quoted on
        _dense("prefill_f32", 1, 256, 256, 8, 8, 64, dtype="f32"),
        # the prefill benchmarks: MHA with the log-sum-exp output, and GQA at 8192 tokens
        _dense("prefill_mha_lse", 4, 2048, 2048, 32, 32, 128, lse=True),
        _dense("prefill_gqa", 2, 8192, 8192, 32, 8, 128),
        # whole prompts of very different lengths packed together, small heads
        _packed("prompts_packed", 24, 0, 0, 17, 2000, d=64, dtype="f16"),
        # the scores of a head group on the math path
        dict(name="softmax_rows", kind="softmax", rows=131072, n=4096, dtype="bf16"),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def _draw(rng):
    hq, hkv = rng.choice([(32, 8), (32, 8), (32, 32), (64, 8), (8, 8), (8, 2)])
    d = rng.choice([128, 128, 64])
    dtype = rng.choice(["bf16", "bf16", "f16"])
    kind = rng.choice(["decode", "decode", "speculate", "chunk", "mixed", "prompts", "prefill", "prefill", "contiguous", "f32", "softmax"])
    if kind in ("decode", "speculate", "chunk"):
        new = {"decode": 1, "speculate": rng.randint(2, 8), "chunk": _log(rng, 64, 1024)}[kind]
        hi = max(new, _log(rng, 64, 32768))
        seqs = _log(rng, 1, {"decode": 256, "speculate": 64, "chunk": 16}[kind])
        lo = max(new, hi // rng.choice([1, 4, 16]))
        max_len = (1 << (hi - 1).bit_length()) * rng.choice([1, 1, 2, 4])
        return _cache("", seqs, new, lo, hi, max_len, hq, hkv, d, rng.choice([16, 16, 16, 32, 64, 8]), dtype)
    if kind == "mixed":
        hi = _log(rng, 64, 8192)
        prompts = rng.randint(1, 6)
        ones = _log(rng, 1, 128)
        return _packed("", prompts + ones, ones, _log(rng, 64, 1024), max(1, hi // 16), hi, hq, hkv, d, rng.choice([16, 16, 32]), dtype)
    if kind == "prompts":
        hi = _log(rng, 64, 8192)
        return _packed("", _log(rng, 1, 48), 0, 0, max(1, hi // rng.choice([4, 16, 100])), hi, hq, hkv, d, 0, dtype)
    if kind == "prefill":
        s = _log(rng, 64, 8192)
        padded = rng.random() < 0.25
        return _dense("", _log(rng, 1, 8), s, s, hq, hkv, rng.choice([d, d, d, 32]), dtype, not padded and rng.random() < 0.3, padded)
    if kind == "contiguous":
        s = rng.choice([1, 1, 1, 4])
        return _dense("", _log(rng, 1, 64), s, _log(rng, 64, 8192), hq, hkv, d, dtype)
    if kind == "f32":
        s = _log(rng, 64, 1024)
        hq, hkv = rng.choice([(8, 8), (8, 2), (16, 4)])
        return _dense("", _log(rng, 1, 4), s, s, hq, hkv, rng.choice([32, 64, 128]), "f32")
    n = _log(rng, 128, 16384)
    return dict(kind="softmax", rows=_log(rng, 256, 131072), n=n, dtype=rng.choice(["bf16", "f16", "f32"]))


# No draw costs more than the largest listed case (1.1e12 operations, 2.1e9 bytes); f32 storage has no 16-bit
# tensor operations to count on, so its share is smaller.
_MOST_FLOPS, _MOST_FLOPS_F32, _MOST_BYTES = 1.0e12, 4.5e9, 2.1e9


def draw(rng):
    while True:
        c = _draw(rng)
        w = work(c)
        if w["bytes"] <= _MOST_BYTES and w["flops"] <= (_MOST_FLOPS_F32 if c["dtype"] == "f32" and c["kind"] == "dense" else _MOST_FLOPS):
            c.pop("name", None)
            return c


def _spread(n, lo, hi):
    """n lengths from lo to hi, evenly spread, hi among them."""
    return [hi] if n == 1 else [lo + (hi - lo) * i // (n - 1) for i in range(n)]


def _lengths(case):
    """(new tokens, tokens seen in all) of each sequence, in no particular order."""
    if case["kind"] == "cache":
        return [(case["new"], n) for n in _spread(case["seqs"], case["lo"], case["hi"])]
    if case["kind"] == "packed":
        prompts = _spread(case["seqs"] - case["ones"], case["lo"], case["hi"])
        got = [(min(n, case["chunk"]) if case["chunk"] else n, n) for n in prompts]
        return got + ([(1, n) for n in _spread(case["ones"], case["lo"], case["hi"])] if case["ones"] else [])
    if case["padded"]:
        return [(n, n) for n in _spread(case["batch"], case["s"] // 2 + 1, case["s"])]
    return [(case["s"], case["kv"])] * case["batch"]


def work(case):
    size = BYTES[case["dtype"]]
    if case["kind"] == "softmax":
        return {"bytes": 2 * case["rows"] * case["n"] * size, "flops": 4 * case["rows"] * case["n"]}
    hq, hkv, d = case["hq"], case["hkv"], case["d"]
    lens = _lengths(case)
    q_rows = sum(a for a, _ in lens)
    kv_rows = sum(b for _, b in lens)
    seen = sum(a * (b - a) + a * (a + 1) // 2 for a, b in lens)   # the last of a sequence's tokens sees all of it
    nbytes = (2 * q_rows * hq * d + 2 * kv_rows * hkv * d) * size
    if case["kind"] == "cache":
        nbytes += 4 * q_rows * hkv * d * size                       # the new rows, read and written into their pages
    if case.get("page"):
        nbytes += sum(4 * -(-b // case["page"]) + 4 for _, b in lens)
    if case["kind"] == "dense" and case["padded"]:
        nbytes = (2 * case["batch"] * case["s"] * hq * d + 2 * kv_rows * hkv * d) * size + case["batch"] * case["kv"]
    if case.get("lse"):
        nbytes += 4 * q_rows * hq
    return {"bytes": nbytes, "flops": 4 * d * hq * seen}


def tolerance(case):
    """Results are rounded to the storage type once, and so are the attention weights on the way."""
    return {"rel": {"bf16": 1e-2, "f16": 2e-3, "f32": 1e-5}[case["dtype"]]}


def _normal(shape, dtype, g):
    return torch.randn(shape, generator=g, device="cuda", dtype=dtype)


def _pages(lens, page, width, g):
    """A pool with one part in eight to spare and a table of `width` pages per sequence into a permutation of it."""
    need = [-(-n // page) for n in lens]
    pool = sum(need) + sum(need) // 8 + 1
    perm = torch.randperm(pool, generator=g, device="cuda").to(torch.int32)
    table = torch.full((len(lens), width), -1, dtype=torch.int32, device="cuda")
    at = 0
    for i, n in enumerate(need):
        table[i, :n] = perm[at:at + n]
        at += n
    return pool, table


def prepare(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    dt = DTYPES[case["dtype"]]
    if case["kind"] == "softmax":
        return {"case": case, "x": _normal((case["rows"], case["n"]), dt, g) * 2}
    hq, hkv, d = case["hq"], case["hkv"], case["d"]
    lens = _lengths(case)
    order = torch.randperm(len(lens), generator=torch.Generator().manual_seed(seed)).tolist()
    lens = [lens[i] for i in order]
    st = {"case": case}
    if case["kind"] == "cache":
        seqs, new, page = case["seqs"], case["new"], case["page"]
        pool, st["table"] = _pages([b for _, b in lens], page, -(-case["max_len"] // page), g)
        st["lens"] = torch.tensor([b for _, b in lens], dtype=torch.int32, device="cuda")
        st["k"], st["v"] = _normal((pool, page, hkv, d), dt, g), _normal((pool, page, hkv, d), dt, g)
        st["k_new"], st["v_new"] = _normal((seqs, new, hkv, d), dt, g), _normal((seqs, new, hkv, d), dt, g)
        st["q"] = _normal((seqs, new, hq, d), dt, g)
    elif case["kind"] == "packed":
        q_lens, k_lens = [a for a, _ in lens], [b for _, b in lens]
        st["cu_q"] = torch.tensor([sum(q_lens[:i]) for i in range(len(lens) + 1)], dtype=torch.int32, device="cuda")
        st["cu_k"] = torch.tensor([sum(k_lens[:i]) for i in range(len(lens) + 1)], dtype=torch.int32, device="cuda")
        st["max_q"], st["max_k"] = max(q_lens), max(k_lens)
        st["q"] = _normal((sum(q_lens), hq, d), dt, g)
        rows, st["table"] = (sum(k_lens),), None
        if case["page"]:
            pool, st["table"] = _pages(k_lens, case["page"], -(-st["max_k"] // case["page"]), g)
            rows = (pool, case["page"])
        st["k"], st["v"] = _normal((*rows, hkv, d), dt, g), _normal((*rows, hkv, d), dt, g)
    else:
        b, s, kv = case["batch"], case["s"], case["kv"]
        st["q"] = _normal((b, s, hq, d), dt, g)
        st["k"], st["v"] = _normal((b, kv, hkv, d), dt, g), _normal((b, kv, hkv, d), dt, g)
        if case["padded"]:
            real = torch.tensor([n for n, _ in lens], device="cuda").unsqueeze(1)
            st["mask"] = (torch.arange(kv, device="cuda").unsqueeze(0) < real).to(torch.uint8)
    return st


def run(st):
    case = st["case"]
    if case["kind"] == "softmax":
        return low.softmax_last_dim(st["x"])
    q, k, v = st["q"], st["k"], st["v"]
    if case["kind"] == "cache":
        table, lens = st["table"], st["lens"]
        low.kvcache_append(st["k_new"], st["v_new"], k, v, table, lens, case["seqs"], case["new"], case["hkv"], case["d"], case["page"],
                           table.shape[1])
        return {"o": high.flash_attn_with_kvcache(q, k, v, lens, table), "k": k, "v": v}
    if case["kind"] == "packed":
        return high.flash_attn_varlen_func(q, k, v, st["cu_q"], st["cu_k"], st["max_q"], st["max_k"], block_table=st["table"])
    if case["padded"]:
        o = torch.empty_like(q)
        low.flash_attn(q, k, v, o, case["batch"], case["s"], case["kv"], case["hq"], case["hkv"], case["d"], 0, 1.0 / math.sqrt(case["d"]),
                       st["mask"])
        return o
    return high.flash_attn_func(q, k, v, start_pos=case["kv"] - case["s"], return_lse=case["lse"])
