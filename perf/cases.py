"""The workloads whose speed matters, through the public entry points of the package.

Three kinds of case: ``dense`` (batches of equal lengths: ``flash_attn_func`` and its packed-input variants), ``varlen``
(sequences packed end to end: ``flash_attn_varlen_*``) and ``kvcache`` (``flash_attn_with_kvcache``: decode steps and
chunked prefill on contiguous and paged caches).  Everything is fp16, the only type the operator takes; queries, keys,
values and output gradients are N(0, 1), as in the benchmark configurations and the tests.  Dense and varlen cases are either a
training step (forward + gradients of every input) or a forward alone.
"""
import math
import random

import torch

from flash_attention_turing_b200 import (
    flash_attn_func,
    flash_attn_kvpacked_func,
    flash_attn_qkvpacked_func,
    flash_attn_varlen_func,
    flash_attn_varlen_kvpacked_func,
    flash_attn_varlen_qkvpacked_func,
    flash_attn_with_kvcache,
)


def _dense(name, batch, seqlen_q, seqlen_k, heads, heads_k, head_dim, causal, backward, layout="separate"):
    return dict(name=name, kind="dense", layout=layout, batch=batch, seqlen_q=seqlen_q, seqlen_k=seqlen_k, heads=heads,
                heads_k=heads_k, head_dim=head_dim, causal=causal, backward=backward)


def _varlen(name, batch, shortest, longest, most_tokens, lengths_seed, heads, heads_k, head_dim, causal, backward,
            layout="separate"):
    return dict(name=name, kind="varlen", layout=layout, batch=batch, shortest=shortest, longest=longest,
                most_tokens=most_tokens, lengths_seed=lengths_seed, heads=heads, heads_k=heads_k, head_dim=head_dim,
                causal=causal, backward=backward)


def _kvcache(name, batch, new_tokens, shortest, longest, lengths_seed, capacity, page, heads, heads_k, head_dim,
             num_splits):
    return dict(name=name, kind="kvcache", batch=batch, new_tokens=new_tokens, shortest=shortest, longest=longest,
                lengths_seed=lengths_seed, capacity=capacity, page=page, heads=heads, heads_k=heads_k, head_dim=head_dim,
                num_splits=num_splits)


def listed():
    return [
        # One small batch through an encoder layer: the launch and the host path are most of it.
        _dense("forward_small", 2, 512, 512, 8, 8, 64, False, False),
        # A training step of a small model on a short odd length, packed qkv projection: eight launches or so, none of them long.
        _dense("train_small_odd", 3, 197, 197, 12, 12, 64, False, True, "qkvpacked"),
        # The prompt of one user, grouped heads, a length that no tile divides.
        _dense("prefill_odd_gqa", 1, 3001, 3001, 32, 8, 128, True, False),
        # Decoder over encoder states: more keys than queries, both odd, packed kv projection.
        _dense("train_cross", 4, 333, 2047, 16, 16, 64, False, True, "kvpacked"),
        # Pre-training at the two usual context lengths.
        _dense("train_4k", 4, 4096, 4096, 32, 32, 128, True, True),
        _dense("train_8k", 4, 8192, 8192, 32, 32, 128, True, True),
        # Long-context training, one sequence, small head size.
        _dense("train_64k", 1, 65536, 65536, 16, 16, 64, True, True),
        # A language-model batch of many short texts, without padding.
        _varlen("train_short_texts", 64, 130, 640, 32768, 1, 16, 16, 64, True, True, "qkvpacked"),
        # Fine-tuning on packed documents with grouped heads.
        _varlen("train_documents_gqa", 16, 256, 4096, 32768, 2, 32, 8, 128, True, True),
        # One user's next token: a contiguous cache that is partly filled.
        _kvcache("decode_one", 1, 1, 1500, 1500, 3, 4096, 0, 32, 8, 128, 0),
        # The next token of a full serving batch: paged cache, lengths far apart.
        _kvcache("decode_batch_paged", 64, 1, 1024, 32768, 4, 33024, 256, 32, 8, 128, 0),
        # Chunks of four prompts on top of what the cache already holds.
        _kvcache("prefill_chunk_paged", 4, 512, 1024, 16384, 5, 16896, 256, 32, 8, 128, 0),
    ]


def _log_between(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _length(rng, low, high):
    """A length: half of them as they come (mostly odd), half multiples of 64."""
    n = _log_between(rng, low, high)
    return n if rng.random() < 0.5 else min(high, max(low, n // 64 * 64))


MOST_FLOPS = 8e12
MOST_BYTES = 3e9
MOST_ELEMENTS = 3e8  # of one tensor of queries


def draw(rng):
    while True:
        head_dim = rng.choice((64, 128))
        heads_k = rng.choice((1, 2, 4, 8, 12, 16, 32))
        heads = heads_k * rng.choice((1, 1, 2, 4)) if heads_k <= 8 else heads_k
        kind = rng.choice(("dense", "dense", "dense", "varlen", "varlen", "kvcache", "kvcache", "kvcache"))
        if kind == "dense":
            seqlen_q = _length(rng, 64, 16384)
            layout = rng.choice(("separate", "separate", "kvpacked", "qkvpacked"))
            if layout == "qkvpacked":
                heads = heads_k
            cross = layout != "qkvpacked" and rng.random() < 0.25
            seqlen_k = _length(rng, 64, 16384) if cross else seqlen_q
            case = _dense("", _log_between(rng, 1, 16), seqlen_q, seqlen_k, heads, heads_k, head_dim,
                          not cross and rng.random() < 0.6, rng.random() < 0.65, layout)
        elif kind == "varlen":
            layout = rng.choice(("separate", "kvpacked", "qkvpacked"))
            if layout == "qkvpacked":
                heads = heads_k
            causal, backward = rng.random() < 0.6, rng.random() < 0.65
            # training texts have more than 128 tokens, and bidirectional ones more than 512; a forward takes any length
            least = (130 if causal else 520) if backward else 1
            longest = _log_between(rng, max(128, least + least // 2), 8192)
            shortest = max(least, int(longest * rng.uniform(0.05, 0.8)))
            batch = min(_log_between(rng, 2, 64), 65536 // longest)
            case = _varlen("", batch, shortest, longest, batch * longest, rng.randrange(1 << 30), heads, heads_k, head_dim,
                           causal, backward, layout)
        else:
            longest = _log_between(rng, 64, 32768)
            page = rng.choice((0, 256, 512))
            new_tokens = rng.choice((1, 1, 1, 2, 4, _length(rng, 64, 1024)))
            capacity = longest + new_tokens + rng.randrange(256)
            if page:
                capacity = -(-capacity // page) * page
            case = _kvcache("", _log_between(rng, 1, 128), new_tokens, max(1, int(longest * rng.uniform(0.05, 1.0))),
                            longest, rng.randrange(1 << 30), capacity, page, heads, heads_k, head_dim,
                            rng.choice((0, 0, 0, 1, 4)))
        del case["name"]
        w = work(case)
        queries = case["batch"] * case.get("seqlen_q", case.get("longest", 0)) * case["heads"] * head_dim
        if kind == "kvcache":
            queries = case["batch"] * case["capacity"] * case["heads_k"] * head_dim
        if w["flops"] <= MOST_FLOPS and w["bytes"] <= MOST_BYTES and queries <= MOST_ELEMENTS:
            return case


def _lengths(case):
    """The sequence lengths of a varlen or kvcache case, from the case alone."""
    rng = random.Random(case["lengths_seed"])
    lengths = [rng.randint(case["shortest"], case["longest"]) for _ in range(case["batch"])]
    if "most_tokens" in case and sum(lengths) > case["most_tokens"]:
        lengths = [max(1, n * case["most_tokens"] // sum(lengths)) for n in lengths]
    return lengths


def _normal(generator, *shape):
    return torch.randn(*shape, generator=generator, device="cuda", dtype=torch.float16)


def _qkv(case, generator, rows_q, rows_k):
    """The inputs in the layout of the case; rows_*: the leading dimensions."""
    h, h_k, d = case["heads"], case["heads_k"], case["head_dim"]
    if case["layout"] == "qkvpacked":
        return [_normal(generator, *rows_q, 3, h, d)]
    if case["layout"] == "kvpacked":
        return [_normal(generator, *rows_q, h, d), _normal(generator, *rows_k, 2, h_k, d)]
    return [_normal(generator, *rows_q, h, d), _normal(generator, *rows_k, h_k, d), _normal(generator, *rows_k, h_k, d)]


def prepare(case, seed):
    generator = torch.Generator(device="cuda").manual_seed(seed)
    state = {"case": case}
    if case["kind"] == "kvcache":
        b, h, h_k, d, new, page = (case[k] for k in ("batch", "heads", "heads_k", "head_dim", "new_tokens", "page"))
        state["q"] = _normal(generator, b, new, h, d)
        state["k"], state["v"] = _normal(generator, b, new, h_k, d), _normal(generator, b, new, h_k, d)
        rows = (b * (case["capacity"] // page), page) if page else (b, case["capacity"])
        state["k_cache"], state["v_cache"] = _normal(generator, *rows, h_k, d), _normal(generator, *rows, h_k, d)
        state["cache_seqlens"] = torch.tensor(_lengths(case), dtype=torch.int32, device="cuda")
        state["block_table"] = None
        if page:
            order = torch.randperm(rows[0], generator=generator, device="cuda", dtype=torch.int64)
            state["block_table"] = order.to(torch.int32).view(b, -1)
        return state
    h, d = case["heads"], case["head_dim"]
    if case["kind"] == "dense":
        rows_q, rows_k = (case["batch"], case["seqlen_q"]), (case["batch"], case["seqlen_k"])
    else:
        lengths = _lengths(case)
        rows_q = rows_k = (sum(lengths),)
        ends = torch.tensor([0] + lengths, dtype=torch.int32).cumsum(0, dtype=torch.int32)
        state["cu_seqlens"], state["max_seqlen"] = ends.cuda(), max(lengths)
    state["inputs"] = _qkv(case, generator, rows_q, rows_k)
    if case["backward"]:
        for t in state["inputs"]:
            t.requires_grad_(True)
        state["dout"] = _normal(generator, *rows_q, h, d)
    return state


_DENSE = {"separate": flash_attn_func, "kvpacked": flash_attn_kvpacked_func, "qkvpacked": flash_attn_qkvpacked_func}


def _forward(state):
    case, inputs = state["case"], state["inputs"]
    if case["kind"] == "dense":
        return _DENSE[case["layout"]](*inputs, causal=case["causal"])
    cu, longest = state["cu_seqlens"], state["max_seqlen"]
    if case["layout"] == "qkvpacked":
        return flash_attn_varlen_qkvpacked_func(*inputs, cu, longest, causal=case["causal"])
    fn = flash_attn_varlen_kvpacked_func if case["layout"] == "kvpacked" else flash_attn_varlen_func
    return fn(*inputs, cu, cu, longest, longest, causal=case["causal"])


def run(state):
    case = state["case"]
    if case["kind"] == "kvcache":
        out, lse = flash_attn_with_kvcache(
            state["q"], state["k_cache"], state["v_cache"], state["k"], state["v"], cache_seqlens=state["cache_seqlens"],
            block_table=state["block_table"], causal=True, num_splits=case["num_splits"], return_softmax_lse=True)
        return out, lse, state["k_cache"], state["v_cache"]
    if not case["backward"]:
        with torch.no_grad():
            return _forward(state)
    out = _forward(state)
    return (out.detach(), *torch.autograd.grad(out, state["inputs"], state["dout"]))


def _pairs(rows, keys, causal):
    """Visible (query, key) pairs of one head; causal masks are aligned at the bottom right."""
    if not causal:
        return rows * keys
    seen = min(rows, keys)
    return rows * keys - rows * (rows - 1) // 2 if keys >= rows else seen * (seen + 1) // 2


def work(case):
    """Products over the visible pairs: two in the forward, five more in the backward.  Bytes: inputs once, outputs once."""
    h, h_k, d = case["heads"], case["heads_k"], case["head_dim"]
    if case["kind"] == "kvcache":
        new, lengths = case["new_tokens"], _lengths(case)
        pairs = sum(_pairs(new, n + new, True) for n in lengths)
        tokens = case["batch"] * new
        moved = 2 * 2 * h_k * d * (sum(lengths) + 2 * tokens)  # cached k, v read; new k, v read and stored
        return {"bytes": moved + 2 * 2 * tokens * h * d + 4 * tokens * h, "flops": 4.0 * pairs * h * d}
    if case["kind"] == "dense":
        pairs = case["batch"] * _pairs(case["seqlen_q"], case["seqlen_k"], case["causal"])
        tokens, tokens_k = case["batch"] * case["seqlen_q"], case["batch"] * case["seqlen_k"]
    else:
        pairs = sum(_pairs(n, n, case["causal"]) for n in _lengths(case))
        tokens = tokens_k = sum(_lengths(case))
    q_bytes, kv_bytes = 2 * tokens * h * d, 2 * 2 * tokens_k * h_k * d
    if not case["backward"]:
        return {"bytes": 2 * q_bytes + kv_bytes, "flops": 4.0 * pairs * h * d}
    return {"bytes": 4 * q_bytes + 2 * kv_bytes, "flops": 14.0 * pairs * h * d}


def tolerance(case):
    """fp16 keeps 11 bits: probabilities, their gradients and the results are each rounded to it, 2e-3 together.  In the
    backward the normalised probabilities of a long row lie below fp16's normal range and keep fewer bits."""
    return {"rel": 5e-3 if case.get("backward") else 2e-3}
