"""The calls this framework is used for, with their sizes, for timing programs.

A case is one call (or one short sequence of calls) of the public API at one size. `listed()` are the fixed ones, `draw()`
gives further cases from the ranges that the listed ones stand for. Five operations:

  decode      `decode` on a paged NVFP4 cache: one layer's attention of one decode step
  step        `quantize_append_paged_mla_kv_cache` of one new token per request, then `decode`: what a serving engine does
              per layer and step
  verify      `serving.decode_multi_token`: several query tokens per request (speculative / MTP verification)
  append      `quantize_append_paged_mla_kv_cache` of whole prompts: what follows a prefill
  dequantize  `dequantize` of a whole cache, for consumers that need it in BF16 or FP32
  pool        `serving.PagedLatentCache`: requests are admitted (pages handed out, prompts appended), decoded once and
              released

Inputs are the distributions of the project's tests and benchmark: N(0, 1) queries and latent rows, written into a page
pool in shuffled order, with global scales as a calibration would give them.
"""
import math
import random

import torch

import nvfp4_mla_b200 as mla
from nvfp4_mla_b200 import serving

CKV, KPE, TOKEN_BYTES = 512, 64, 352
SM_SCALE = (128 + KPE) ** -0.5
CKV_SCALE, KPE_SCALE = 6.5 / (6 * 448), 6.5 / 448  # amax / (6 * 448) and amax / 448 of N(0, 1) data
MAX_TOKENS, MAX_TOKEN_HEADS = 64 * 65536, 128 * 2 * 1048576  # the largest listed cases
CHUNK = 1 << 18  # rows generated at a time


def listed():
    return [
        # one user, a short context, on a tensor-parallel shard: latency and launches
        dict(name="decode_h16_b1_2k", op="decode", heads=16, batch=1, lo=2048, hi=2048, page_size=64, precision="bf16"),
        # a small chat batch per layer and step: the new token's row is appended, then decoded; short ragged contexts, small pages
        dict(name="step_h16_b24_short", op="step", heads=16, batch=24, lo=1, hi=1000, page_size=16, precision="bf16"),
        # DeepSeek-V3 on eight tensor-parallel GPUs, ordinary batch and context
        dict(name="decode_h16_b32_8k", op="decode", heads=16, batch=32, lo=8192, hi=8192, page_size=64, precision="bf16"),
        # the headline shape: large batch, long contexts, bandwidth-bound
        dict(name="decode_h16_b64_64k", op="decode", heads=16, batch=64, lo=65536, hi=65536, page_size=64, precision="bf16"),
        # the same shard in the 8-bit mode at a middle context length
        dict(name="decode_h16_b64_16k_fp8", op="decode", heads=16, batch=64, lo=16384, hi=16384, page_size=64, precision="fp8"),
        # data-parallel attention with all 128 heads on one GPU, ragged batch, 8-bit mode: compute-bound
        dict(name="decode_h128_b64_ragged_fp8", op="decode", heads=128, batch=64, lo=1024, hi=32768, page_size=64, precision="fp8"),
        # two million-token contexts with all heads, 16-bit mode
        dict(name="decode_h128_b2_1m", op="decode", heads=128, batch=2, lo=1048576, hi=1048576, page_size=64, precision="bf16"),
        # two tensor-parallel GPUs (64 heads each), ragged batch, 16-bit mode
        dict(name="decode_h64_b32_ragged", op="decode", heads=64, batch=32, lo=500, hi=16000, page_size=64, precision="bf16"),
        # speculative decoding: one new and three drafted tokens per request are verified together
        dict(name="verify_q4_h16_b16_8k", op="verify", heads=16, batch=16, lo=4000, hi=12000, q_len=4, page_size=64, precision="bf16"),
        # the latent rows of prefilled prompts go into the cache
        dict(name="append_b64_16k", op="append", batch=64, lo=1000, hi=16384, page_size=64),
        # a whole cache in BF16
        dict(name="dequantize_512k", op="dequantize", tokens=524288, page_size=64, dtype="bf16"),
        # requests come and go: prompts of a few hundred tokens admitted to the pool, decoded once, released
        dict(name="pool_h16_b8", op="pool", heads=16, batch=8, lo=50, hi=600, page_size=64, precision="bf16"),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    op = rng.choice(["decode"] * 10 + ["step"] * 2 + ["verify"] * 2 + ["append", "dequantize", "pool"])
    case = dict(op=op, page_size=rng.choice([16, 32, 64, 64, 64, 64, 128]))
    if op == "dequantize":
        return dict(case, tokens=case["page_size"] * _log_int(rng, 8, 1048576 // case["page_size"]), dtype=rng.choice(["bf16", "bf16", "fp32"]))
    if op == "append":
        batch = _log_int(rng, 1, 128)
        hi = _log_int(rng, 1, min(32768, 1048576 // batch))
        return dict(case, batch=batch, lo=max(1, hi // rng.choice([1, 2, 16])), hi=hi)
    if op == "pool":
        batch, hi = _log_int(rng, 1, 32), _log_int(rng, 8, 2000)
        return dict(case, heads=rng.choice([16, 32]), batch=batch, lo=max(1, hi // 10), hi=hi, precision="bf16")
    case.update(heads=rng.choice([16, 16, 16, 32, 64, 128]), precision=rng.choice(["bf16", "bf16", "bf16", "fp8"]))
    if op == "verify":
        case.update(q_len=rng.randint(2, 4))
    # log-uniform batch and length, within what the largest listed cases read and multiply
    q_len = case.get("q_len", 1)
    batch = _log_int(rng, 1, 256 // q_len)
    hi = _log_int(rng, 128, min(262144, MAX_TOKENS // batch // q_len, MAX_TOKEN_HEADS // (case["heads"] * batch * q_len)))
    lo = max(q_len, hi // rng.choice([1, 1, 2, 16, hi]))
    return dict(case, batch=batch, lo=lo, hi=hi)


def _lens(case):
    """Tokens per request, uniform in [lo, hi]: part of the case, the same for every seed."""
    r = random.Random(case["batch"] * 1000003 + case["lo"] * 101 + case["hi"])
    return [r.randint(case["lo"], case["hi"]) for _ in range(case["batch"])]


def _rows(g, n):
    return (torch.randn(n, CKV, generator=g, device="cuda", dtype=torch.bfloat16),
            torch.randn(n, KPE, generator=g, device="cuda", dtype=torch.bfloat16))


def _pages(case, lens, g):
    """An empty cache for `lens`, its page list in shuffled order (as kv_indices, kv_indptr) and as a page table."""
    ps = case["page_size"]
    need = [-(-n // ps) for n in lens]
    total, width = sum(need), max(need)
    cache = (torch.zeros(total, ps, CKV // 2, dtype=torch.uint8, device="cuda"),
             torch.zeros(total, ps, CKV // 16, dtype=torch.uint8, device="cuda").view(torch.float8_e4m3fn),
             torch.zeros(total, ps, KPE, dtype=torch.uint8, device="cuda").view(torch.float8_e4m3fn))
    kv_indices = torch.randperm(total, generator=g, device="cuda").int()
    counts = torch.tensor(need, device="cuda")
    kv_indptr = torch.cat([counts.new_zeros(1), counts.cumsum(0)]).int()
    column = torch.arange(width, device="cuda")
    at = (kv_indptr[:-1, None].long() + column).clamp_(max=total - 1)
    page_table = torch.where(column < counts[:, None], kv_indices[at], 0).int().contiguous()
    return cache, kv_indices, kv_indptr, page_table


def _token_list(lens):
    """(batch_indices, positions) of every token of every request."""
    n = torch.tensor(lens, device="cuda")
    indptr = torch.cat([n.new_zeros(1), n.cumsum(0)])
    return mla.get_batch_indices_positions(indptr, n, int(indptr[-1]))


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    op = case["op"]
    if op == "dequantize":
        ps = case["page_size"]
        pages = case["tokens"] // ps
        cache, kv_indices, kv_indptr, _ = _pages(dict(page_size=ps), [case["tokens"]], g)
        b, pos = _token_list([case["tokens"]])
        for i in range(0, case["tokens"], CHUNK):
            ckv, kpe = _rows(g, min(CHUNK, case["tokens"] - i))
            mla.quantize_append_paged_mla_kv_cache(ckv, kpe, b[i:i + CHUNK], pos[i:i + CHUNK], *cache, kv_indices, kv_indptr, None,
                                                   CKV_SCALE, KPE_SCALE)
        return dict(op=op, cache=cache, dtype=torch.bfloat16 if case["dtype"] == "bf16" else torch.float32, pages=pages)
    lens = _lens(case)
    if op == "pool":
        need = sum(-(-n // case["page_size"]) for n in lens)
        width = -(-case["hi"] // case["page_size"])
        pool = serving.PagedLatentCache(need + 8, case["page_size"], case["batch"], width, CKV_SCALE, KPE_SCALE)
        ckv, kpe = _rows(g, sum(lens))
        return dict(op=op, pool=pool, requests=list(enumerate(lens)), ckv=ckv, kpe=kpe, precision=case["precision"], **_queries(g, (case["batch"], case["heads"])))
    cache, kv_indices, kv_indptr, page_table = _pages(case, lens, g)
    b, pos = _token_list(lens)
    if op == "append":
        ckv, kpe = _rows(g, sum(lens))
        return dict(op=op, ckv=ckv, kpe=kpe, batch_indices=b, positions=pos, cache=cache, kv_indices=kv_indices, kv_indptr=kv_indptr)
    for i in range(0, sum(lens), CHUNK):
        ckv, kpe = _rows(g, min(CHUNK, sum(lens) - i))
        mla.quantize_append_paged_mla_kv_cache(ckv, kpe, b[i:i + CHUNK], pos[i:i + CHUNK], *cache, kv_indices, kv_indptr, None, CKV_SCALE, KPE_SCALE)
    shape = (case["batch"], case["q_len"], case["heads"]) if op == "verify" else (case["batch"], case["heads"])
    state = dict(op=op, cache=cache, page_table=page_table, kv_lens=torch.tensor(lens, dtype=torch.int32, device="cuda"), max_kv_len=max(lens),
                 precision=case["precision"], **_queries(g, shape))
    if op == "step":  # the newest token of every request
        ckv, kpe = _rows(g, case["batch"])
        state.update(ckv=ckv, kpe=kpe, batch_indices=torch.arange(case["batch"], dtype=torch.int32, device="cuda"),
                     positions=state["kv_lens"] - 1, kv_indices=kv_indices, kv_indptr=kv_indptr)
    return state


def _queries(g, shape):
    return dict(q_nope=torch.randn(*shape, CKV, generator=g, device="cuda", dtype=torch.bfloat16),
                q_pe=torch.randn(*shape, KPE, generator=g, device="cuda", dtype=torch.bfloat16))


def run(s):
    op = s["op"]
    if op == "dequantize":
        return mla.dequantize(*s["cache"], CKV_SCALE, KPE_SCALE, dtype=s["dtype"])
    if op == "pool":
        pool, requests = s["pool"], [r for r, _ in s["requests"]]
        pool.append(s["requests"], s["ckv"], s["kpe"])
        out = pool.decode(requests, s["q_nope"], s["q_pe"], SM_SCALE, precision=s["precision"])
        for r in requests:
            pool.release(r)
        return out
    if op in ("append", "step"):
        mla.quantize_append_paged_mla_kv_cache(s["ckv"], s["kpe"], s["batch_indices"], s["positions"], *s["cache"], s["kv_indices"],
                                               s["kv_indptr"], None, CKV_SCALE, KPE_SCALE)
        if op == "append":
            return s["cache"]
    call = serving.decode_multi_token if op == "verify" else mla.decode
    return call(s["q_nope"], s["q_pe"], *s["cache"], s["page_table"], s["kv_lens"], SM_SCALE, CKV_SCALE, KPE_SCALE, max_kv_len=s["max_kv_len"],
                precision=s["precision"])


def work(case):
    """Cached tokens are read once per request (all heads and query tokens share them): 352 bytes each; queries in, outputs
    out in BF16. 2176 operations per head and token: 576 channels in QK^T, 512 in PV."""
    op = case["op"]
    if op == "dequantize":
        return dict(bytes=case["tokens"] * (TOKEN_BYTES + (CKV + KPE) * (2 if case["dtype"] == "bf16" else 4)), flops=0)
    lens = _lens(case)
    tokens, written = sum(lens), dict(append=sum(lens), pool=sum(lens), step=case["batch"]).get(op, 0)
    append_bytes = written * (2 * (CKV + KPE) + TOKEN_BYTES + 8)
    if op == "append":
        return dict(bytes=append_bytes, flops=0)
    q_len = case.get("q_len", 1)
    queries = case["batch"] * q_len * case["heads"]
    pages = sum(-(-n // case["page_size"]) for n in lens)
    return dict(bytes=TOKEN_BYTES * tokens + queries * 2 * (CKV + KPE + CKV) + 4 * pages + append_bytes, flops=2176 * case["heads"] * q_len * tokens)


def tolerance(case):
    if case["op"] in ("append", "dequantize"):
        return "exact"
    if case["precision"] == "fp8":  # E4M3 query, KV and probabilities (three bits of mantissa): 0.045 against the same in 64 bits
        return {"rel": 0.03, "max": 0.5}
    # 16-bit operands and a BF16 result: 1.7e-3 and 0.0045 against the same in 64 bits
    return {"rel": 7e-3, "max": 0.02}
