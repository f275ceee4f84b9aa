"""The work that users of this framework have it do, as measurable cases.

A case is a plain dict.  `kind` names the entry point:
  "dense"    flash_mla_with_kvcache on a paged bf16 / fp16 cache (one decode step of one layer)
  "sparse"   flash_mla_with_kvcache on FP8 token records gathered by index
  "prefill"  flash_mla_sparse_fwd, every query token with its own list of keys
  "write"    the FP8 cache writers of flashmla_b200.kvcache, the step before sparse decode

A decode step runs the same schedule through every layer of a model: its first layer makes it, the others reuse it.  `fresh`
says which of the two a case is (True: the pass makes its schedule).
"""
import math

import torch

from flashmla_b200 import flash_mla_sparse_fwd, flash_mla_with_kvcache, get_mla_metadata
from flashmla_b200.kvcache import quantize_fp8_kvcache, quantize_fp8_kvcache_model1

D_V = 512
PAGE = 64


def _dense(b, s_q, h_q, lengths, typical, spread, lo, hi, dtype="bf16", fresh=False):
    return dict(kind="dense", b=b, s_q=s_q, h_q=h_q, lengths=lengths, typical=typical, spread=spread, lo=lo, hi=hi,
                dtype=dtype, fresh=fresh)


def _sparse(width, b, s_q, h_q, s_kv, topk, page=64, extra_topk=0, extra_page=0, ragged=False, sink=False,
            padded=False, fresh=False):
    return dict(kind="sparse", width=width, b=b, s_q=s_q, h_q=h_q, s_kv=s_kv, topk=topk, page=page, extra_topk=extra_topk,
                extra_page=extra_page, ragged=ragged, sink=sink, padded=padded, fresh=fresh)


def _prefill(width, s_q, h_q, s_kv, topk, ragged=False, sink=False):
    return dict(kind="prefill", width=width, s_q=s_q, h_q=h_q, s_kv=s_kv, topk=topk, ragged=ragged, sink=sink)


def _write(width, pages, page, pow2):
    return dict(kind="write", width=width, pages=pages, page=page, pow2=pow2)


def listed():
    named = [
        # a handful of short chats on a tensor-parallel rank with 16 heads: nothing but latency
        ("dense_small", _dense(4, 1, 16, "uniform", 0, 0, 64, 512)),
        # the serving shape: a full batch of ordinary conversations, all 128 heads on one GPU
        ("dense_serving", _dense(128, 1, 128, "normal", 4096, 512, 1, 8192)),
        # the same with a speculated second token (causal between the two)
        ("dense_mtp", _dense(128, 2, 128, "normal", 4096, 512, 1, 8192)),
        # a tensor-parallel rank: 16 of the 128 heads against the whole cache, fp16
        ("dense_few_heads_fp16", _dense(61, 1, 16, "normal", 4096, 512, 1, 8192, dtype="fp16")),
        # a single very long document: one request has to fill the GPU
        ("dense_one_long", _dense(1, 1, 128, "uniform", 0, 0, 100003, 100003, fresh=True)),
        # one GPU's share of the long-context sweep: lengths over two and a half decades
        ("dense_long_mix", _dense(128, 1, 128, "lognormal", 8192, 1.0, 256, 131072, fresh=True)),
        # token-sparse decode, a full batch at the usual top-k; the last 5 % of every list are padding (-1)
        ("sparse_batch", _sparse(576, 64, 1, 128, 32768, 2048, padded=True)),
        # token-sparse decode, two users with a speculated token on a rank with 64 heads; attention sink, lists of different lengths
        ("sparse_small", _sparse(576, 2, 2, 64, 8192, 2048, ragged=True, sink=True, fresh=True)),
        # 512-wide records with a second (compressed) cache beside the window
        ("sparse_512_extra", _sparse(512, 74, 1, 128, 16384, 512, extra_topk=1024, extra_page=32, ragged=True, sink=True)),
        # a chunk of a long prompt
        ("prefill_chunk", _prefill(576, 4096, 128, 32768, 2048)),
        # the ragged last chunk of a short prompt, 512-wide, on a rank with 64 heads
        ("prefill_tail_512", _prefill(512, 117, 64, 5003, 640, ragged=True, sink=True)),
        # a prefilled prompt goes into the FP8 cache
        ("write_records", _write(576, 1031, 64, False)),
    ]
    return [dict(case, name=name) for name, case in named]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["dense", "dense", "dense", "sparse", "sparse", "prefill", "prefill", "write"])
    if kind == "dense":
        b, s_q, h_q = _log(rng, 1, 160), rng.choice([1, 1, 1, 2, 3]), rng.choice([8, 16, 32, 64, 96, 128, 128])
        most = min(131072, 1_200_000 // (b * s_q))          # tokens of the whole batch, times query tokens
        typical = _log(rng, 64, max(64, most // 2))
        lengths = rng.choice(["normal", "lognormal", "uniform"])
        spread = {"normal": round(typical * rng.uniform(0.05, 0.3), 1), "lognormal": round(rng.uniform(0.3, 1.0), 3), "uniform": 0}[lengths]
        lo, hi = (max(1, typical // 2), typical * 3 // 2) if lengths == "uniform" else (1, min(typical * 8, most))
        return _dense(b, s_q, h_q, lengths, typical, spread, lo, hi, dtype=rng.choice(["bf16", "bf16", "fp16"]),
                      fresh=rng.random() < 0.25)
    if kind == "sparse":
        width, s_q = rng.choice([576, 576, 512]), rng.choice([1, 1, 1, 2])
        topk = rng.choice([128, 256, 512, 1024, 2048, 2048, 64 * rng.randint(2, 32)])
        extra = rng.random() < 0.3
        b = _log(rng, 1, min(160, 400_000 // (s_q * topk)))
        return _sparse(width, b, s_q, rng.choice([16, 64, 64, 128, 128]), rng.randint(topk, 32768), topk,
                       page=rng.choice([64, 64, 32, 256]), extra_topk=64 * rng.randint(1, 16) if extra else 0,
                       extra_page=rng.choice([2, 32, 64]) if extra else 0, ragged=rng.random() < 0.4, sink=rng.random() < 0.4,
                       padded=rng.random() < 0.4, fresh=rng.random() < 0.25)
    if kind == "prefill":
        topk = rng.choice([128, 512, 1024, 2048, 2048, 64 * rng.randint(2, 32)])
        return _prefill(rng.choice([576, 576, 512]), _log(rng, 16, min(4096, 6_000_000 // topk)), rng.choice([64, 128, 128]),
                        rng.randint(topk // 2, 32768), topk, ragged=rng.random() < 0.4, sink=rng.random() < 0.4)
    return _write(rng.choice([576, 512]), _log(rng, 1, 4000), 64, rng.random() < 0.5)


# ---- inputs ---------------------------------------------------------------------------------------------------------

def _lengths(case):
    """The batch's lengths in ascending order: the quantiles of its distribution (the seed only says which request has which)."""
    at = torch.arange(case["b"], dtype=torch.float64).add(0.5).div(case["b"])
    if case["lengths"] == "normal":
        x = case["typical"] + case["spread"] * math.sqrt(2) * torch.erfinv(2 * at - 1)
    elif case["lengths"] == "lognormal":
        x = case["typical"] * torch.exp(case["spread"] * math.sqrt(2) * torch.erfinv(2 * at - 1))
    else:
        x = case["lo"] + (case["hi"] - case["lo"]) * at
    return x.round().clamp(case["lo"], case["hi"]).to(torch.int32)


def _list_lengths(n, most):
    """Lengths of n index lists of at most `most` keys: from a quarter full to full (all full where there is one list)."""
    return torch.linspace(most / 4, most, n).round().to(torch.int32) if n > 1 else torch.tensor([most], dtype=torch.int32)


def _normal(shape, gen, dtype=torch.bfloat16):
    """N(0, 1), a piece at a time (a cache may take gigabytes)."""
    out = torch.empty(shape, dtype=dtype, device="cuda")
    flat, step = out.view(-1), 1 << 27
    for i in range(0, flat.numel(), step):
        n = min(step, flat.numel() - i)
        flat[i:i + n] = torch.randn(n, generator=gen, device="cuda")
    return out


def _chosen(rows, limit, topk, gen):
    """[rows, topk] keys without repetition: row i chooses from [0, limit[i]); -1 where there are fewer keys than topk."""
    out = torch.empty(rows, topk, dtype=torch.int64, device="cuda")
    width = int(limit.max())
    for i in range(0, rows, 512):
        lim = limit[i:i + 512].cuda().unsqueeze(1)
        rank = torch.rand(lim.shape[0], max(width, topk), generator=gen, device="cuda")
        rank[torch.arange(rank.shape[1], device="cuda").unsqueeze(0) >= lim] = -1.0
        best = rank.topk(topk, dim=-1)
        out[i:i + 512] = torch.where(best.values < 0, -1, best.indices)
    return out


def _records(case, b, s_kv, page, gen):
    """An FP8 cache of s_kv tokens for each of b requests, and its block table."""
    per = -(-s_kv // page)
    table = torch.randperm(b * per, generator=gen, device="cuda").view(b, per)
    write = quantize_fp8_kvcache if case["width"] == 576 else quantize_fp8_kvcache_model1
    return write(_normal((b * per, page, 1, case["width"]), gen)), table


def _slots(keys, table, page):
    """Keys [b, s_q, topk] of each request -> positions in the paged cache (-1 stays -1)."""
    b, s_q, topk = keys.shape
    key = keys.clamp_min(0).view(b, -1)
    return torch.where(keys < 0, -1, (table.gather(1, key // page) * page + key % page).view(b, s_q, topk)).to(torch.int32)


def _prefill_limits(case):
    """How many keys each query token of the chunk can see (the chunk is the end of the sequence)."""
    return (torch.arange(case["s_q"]) + max(case["s_kv"] - case["s_q"], 0) + 1).clamp_max(case["s_kv"])


def _valid(case, topk):
    """Keys in a list of topk entries that are not padding."""
    return topk - topk // 20 if case["padded"] else topk


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    state = dict(case=case)
    if case["kind"] == "write":
        state["kv"] = _normal((case["pages"], case["page"], 1, case["width"]), gen)
        return state
    if case["kind"] == "prefill":
        state["q"] = _normal((case["s_q"], case["h_q"], case["width"]), gen)
        state["kv"] = _normal((case["s_kv"], 1, case["width"]), gen)
        state["indices"] = _chosen(case["s_q"], _prefill_limits(case), case["topk"], gen).to(torch.int32).unsqueeze(1)
        state["sink"] = torch.randn(case["h_q"], generator=gen, device="cuda") if case["sink"] else None
        state["lengths"] = None
        if case["ragged"]:
            lengths = _list_lengths(case["s_q"], case["topk"]).cuda()
            state["lengths"] = lengths[torch.randperm(case["s_q"], generator=gen, device="cuda")].contiguous()
        return state
    b, s_q = case["b"], case["s_q"]
    state["sched"] = get_mla_metadata()[0]
    if case["kind"] == "dense":
        dtype = torch.float16 if case["dtype"] == "fp16" else torch.bfloat16
        lengths = _lengths(case)
        width = -(-int(lengths.max()) // PAGE)
        lengths = lengths.cuda()[torch.randperm(b, generator=gen, device="cuda")].contiguous()
        pages = (lengths.long() + PAGE - 1) // PAGE
        total = int(pages.sum())
        # pages in random order; table entries behind a request's last page point at page 0 and are not read
        order = torch.randperm(total, generator=gen, device="cuda").to(torch.int32)
        table = torch.zeros(b, width, dtype=torch.int32, device="cuda")
        table[torch.arange(width, device="cuda").unsqueeze(0) < pages.unsqueeze(1)] = order
        state.update(q=_normal((b, s_q, case["h_q"], 576), gen, dtype), cache=_normal((total, PAGE, 1, 576), gen, dtype),
                     table=table, lengths=lengths)
        return state
    state["q"] = _normal((b, s_q, case["h_q"], case["width"]), gen)
    state["sink"] = torch.randn(case["h_q"], generator=gen, device="cuda") if case["sink"] else None
    for name, topk, page, s_kv in (("", case["topk"], case["page"], case["s_kv"]),
                                   ("extra_", case["extra_topk"], case["extra_page"], max(case["extra_topk"], case["s_kv"] // 4))):
        state[name + "cache"] = state[name + "indices"] = state[name + "lengths"] = None
        if not topk:
            continue
        state[name + "cache"], table = _records(case, b, s_kv, page, gen)
        keys = _chosen(b * s_q, torch.full((b * s_q,), s_kv), topk, gen).view(b, s_q, topk)
        keys[..., _valid(case, topk):] = -1
        state[name + "indices"] = _slots(keys, table, page)
        if case["ragged"]:
            lengths = _list_lengths(b, topk).cuda()
            state[name + "lengths"] = lengths[torch.randperm(b, generator=gen, device="cuda")].contiguous()
    return state


# ---- one pass -------------------------------------------------------------------------------------------------------

def run(state):
    case = state["case"]
    if case["kind"] == "write":
        if case["width"] == 576:
            return quantize_fp8_kvcache(state["kv"], case["pow2"]).view(torch.uint8)
        return quantize_fp8_kvcache_model1(state["kv"]).view(torch.uint8)
    if case["kind"] == "prefill":
        return flash_mla_sparse_fwd(state["q"], state["kv"], state["indices"], case["width"] ** -0.5, D_V,
                                    attn_sink=state["sink"], topk_length=state["lengths"])
    if case["fresh"]:
        state["sched"] = get_mla_metadata()[0]
    if case["kind"] == "dense":
        return flash_mla_with_kvcache(state["q"], state["cache"], state["table"], state["lengths"], D_V, state["sched"],
                                      softmax_scale=576 ** -0.5, causal=True)
    return flash_mla_with_kvcache(state["q"], state["cache"], None, None, D_V, state["sched"], softmax_scale=case["width"] ** -0.5,
                                  is_fp8_kvcache=True, indices=state["indices"], attn_sink=state["sink"],
                                  extra_k_cache=state["extra_cache"], extra_indices_in_kvcache=state["extra_indices"],
                                  topk_length=state["lengths"], extra_topk_length=state["extra_lengths"])


# ---- what a pass cannot do without ------------------------------------------------------------------------------------

def work(case):
    if case["kind"] == "write":
        return {"bytes": case["pages"] * case["page"] * (2 * case["width"] + (656 if case["width"] == 576 else 584)), "flops": 0}
    h_q, s_q = case["h_q"], case["s_q"]
    if case["kind"] == "prefill":
        lists = _list_lengths(s_q, case["topk"]) if case["ragged"] else torch.full((s_q,), case["topk"])
        keys = int(torch.minimum(lists, _prefill_limits(case)).sum())
        return {"bytes": min(keys, case["s_kv"]) * case["width"] * 2 + keys * 4 + s_q * h_q * ((case["width"] + D_V) * 2 + 8),
                "flops": 2 * keys * h_q * (case["width"] + D_V)}
    b = case["b"]
    if case["kind"] == "dense":
        tokens = int(_lengths(case).sum())
        return {"bytes": tokens * 1152 + b * s_q * h_q * (1152 + D_V * 2 + 4), "flops": 2 * tokens * s_q * h_q * (576 + D_V)}
    keys = unique = 0
    for topk, s_kv in ((case["topk"], case["s_kv"]), (case["extra_topk"], max(case["extra_topk"], case["s_kv"] // 4))):
        for n in (_list_lengths(b, topk) if case["ragged"] else torch.full((b,), topk)).tolist():
            n = min(n, _valid(case, topk))
            keys += s_q * n
            unique += min(s_q * n, s_kv)
    record = 656 if case["width"] == 576 else 584
    return {"bytes": unique * record + keys * 4 + b * s_q * h_q * ((case["width"] + D_V) * 2 + 4),
            "flops": 2 * keys * h_q * (case["width"] + D_V)}


def tolerance(case):
    # written records are whole bytes.  Attention: probabilities and outputs are rounded to 16 bits (2^-9 each, a few of
    # them on one value), sums are fp32
    return "exact" if case["kind"] == "write" else {"rel": 1e-2, "max": 5e-2}
