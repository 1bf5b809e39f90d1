"""The work a user of this library has it do, as cases that can be timed one by one.

Every case is one call (or the two calls of a vocabulary-sharded step) through the public Python API on
synthetic inputs made on the GPU from a seed.  A program that decodes keeps one context for its lifetime and
its output buffers from step to step; so do the cases.  Sizes are those of pulsatrix_b200/workloads.py and of
bench.py where one of them fits, and generic otherwise.
"""
from __future__ import annotations

import math

import torch

import pulsatrix_b200 as psx

# Decoding settings of the cases; a case overrides what it needs.
SETTINGS = {"do_sample": True, "temperature": 1.0, "top_k": 0, "top_p": 1.0, "min_p": 0.0, "penalty": 1.0, "history": 0,
            "sigma": 2.5, "zeta": 1.2}

LARGEST_CACHE_BYTES = 2 * 64 * 8 * 4096 * 128 * 4  # "attention-grouped": what a drawn attention case may reach
LARGEST_HEAD = 64 * 2048 * 151936                  # multiply-adds of "head-64-rows"


def listed():
    def sample(name, rows, vocab, kind="sample", **settings):
        return {"name": name, "kind": kind, "rows": rows, "vocab": vocab, **SETTINGS, **settings}

    return [
        # One sequence being decoded, its logits on the GPU: the smallest call there is, latency and launches.
        sample("one-row", 1, 49152, sigma=2.0, zeta=1.2, history=64, penalty=1.1, temperature=0.8, top_k=50, top_p=0.9),
        # A server's decoding step: top-k and top-p over a batch of a large vocabulary.
        sample("top-k-64-rows", 64, 151936, sigma=3.0, zeta=1.0, history=256, penalty=1.05, temperature=0.7, top_k=20,
               top_p=0.8),
        # Nucleus sampling without a top-k: the cut depends on the whole row.
        sample("nucleus-256-rows", 256, 128256, sigma=2.5, zeta=1.5, history=512, penalty=1.2, top_p=0.95),
        # Greedy decoding of a large batch (evaluation), with the log-probabilities of the chosen tokens.
        sample("greedy-1024-rows", 1024, 49152, do_sample=False, sigma=4.0, zeta=0.0),
        # Sampling from the whole distribution, as rollouts and perplexity-matched generation do: temperature alone,
        # rows of an odd length.
        sample("unfiltered-100-rows", 100, 50021, temperature=0.9),
        # One GPU's share of a vocabulary-sharded step over eight: its columns of every row, its eighth of the rows.
        sample("one-shard-of-8", 512, 262144, kind="shard", shards=8, sigma=3.0, zeta=1.3, history=1024, penalty=1.1,
               temperature=0.9, top_k=64, top_p=0.9),
        # A model that runs elsewhere hands one row of logits over in host memory, token after token.
        sample("one-row-from-host", 1, 128256, kind="host", sigma=2.0, zeta=1.2, history=200, penalty=1.1, temperature=0.8,
               top_k=50, top_p=0.9),
        # The selection primitive by itself (beam search, routing, retrieval).
        {"name": "select-64-of-16384", "kind": "top_k", "rows": 4096, "cols": 16384, "k": 64, "largest": True},
        # Head and sampling of one sequence: the weights are the traffic.
        sample("head-one-row", 1, 151936, kind="head", d=2048, tied=True, history=64, penalty=1.1, temperature=0.8, top_k=50,
               top_p=0.9),
        # The same for a full decoding batch: the largest call, arithmetic rather than traffic.
        sample("head-64-rows", 64, 151936, kind="head", d=2048, tied=True, history=64, penalty=1.1, temperature=0.8, top_k=50,
               top_p=0.9),
        # One new position per sequence over a cache with grouped query heads, the cache not quite full.
        {"name": "attention-grouped", "kind": "attention", "batch": 64, "heads": 32, "kv_heads": 8, "q_len": 1, "head_dim": 128,
         "cached": 4000, "max_len": 4096, "window": 0, "padded": False},
        # Row-wise softmax of scores.
        {"name": "softmax-4096", "kind": "row_op", "op": "softmax", "rows": 8192, "cols": 4096},
    ]


def _log_uniform(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _vocab(rng, low=16000, high=262144):
    """A vocabulary size: padded to a multiple of 64 as often as not."""
    v = _log_uniform(rng, low, high)
    return max(low, v // 64 * 64) if rng.random() < 0.5 else v


def _decoding(rng, kinds):
    """Settings of one request class, over the ranges people use."""
    s = dict(SETTINGS)
    kind = rng.choice(kinds)
    s["sigma"] = round(rng.uniform(2.0, 4.0), 2)
    s["zeta"] = round(rng.uniform(0.8, 1.5), 2)
    if rng.random() < 0.7:
        s["penalty"] = round(rng.uniform(1.02, 1.3), 2)
        s["history"] = _log_uniform(rng, 8, 2048)
    if kind == "greedy":
        s["do_sample"] = False
        return s
    s["temperature"] = round(rng.uniform(0.5, 1.2), 2)
    if kind == "top_k":
        s["top_k"] = _log_uniform(rng, 2, 100)
        s["top_p"] = rng.choice([1.0, 0.8, 0.9, 0.95])
    elif kind == "nucleus":
        s["top_p"] = round(rng.uniform(0.5, 0.95), 2)
    elif kind == "min_p":
        s["min_p"] = round(rng.uniform(0.02, 0.2), 2)
    return s


def draw(rng):
    kind = rng.choice(["sample", "sample", "sample", "sample", "unfiltered", "shard", "host", "top_k", "head", "attention", "row_op"])
    if kind == "sample":
        vocab = _vocab(rng)
        rows = _log_uniform(rng, 1, min(1024, 50_331_648 // vocab))
        return {"kind": "sample", "rows": rows, "vocab": vocab, **_decoding(rng, ["top_k", "top_k", "nucleus", "greedy", "min_p"])}
    if kind == "unfiltered":
        vocab = _vocab(rng)
        rows = _log_uniform(rng, 1, max(1, 16_777_216 // vocab))
        return {"kind": "sample", "rows": rows, "vocab": vocab, **_decoding(rng, ["unfiltered"])}
    if kind == "shard":
        shards = rng.choice([2, 4, 8])
        vocab = _vocab(rng, 64000) // shards * shards
        rows = _log_uniform(rng, 16, 512)
        return {"kind": "shard", "rows": rows, "vocab": vocab, "shards": shards, **_decoding(rng, ["top_k", "top_k", "greedy"])}
    if kind == "host":
        return {"kind": "host", "rows": _log_uniform(rng, 1, 8), "vocab": _vocab(rng), **_decoding(rng, ["top_k", "nucleus", "greedy"])}
    if kind == "top_k":
        cols = _log_uniform(rng, 512, 262144)
        rows = _log_uniform(rng, 1, min(16384, 67_108_864 // cols))
        return {"kind": "top_k", "rows": rows, "cols": cols, "k": _log_uniform(rng, 1, min(1024, cols)), "largest": rng.random() < 0.9}
    if kind == "head":
        d = _log_uniform(rng, 512, 4096)
        d = max(64, d // 64 * 64) if rng.random() < 0.8 else d
        vocab = _vocab(rng, 16000, min(151936, 311_164_928 // d))
        rows = _log_uniform(rng, 1, min(64, LARGEST_HEAD // (d * vocab)))
        return {"kind": "head", "rows": rows, "vocab": vocab, "d": d, "tied": rng.random() < 0.7,
                **_decoding(rng, ["top_k", "top_k", "greedy"])}
    if kind == "attention":
        head_dim = rng.choice([64, 96, 128, 128, 128, 256])
        kv_heads, group, q_len = rng.choice([1, 2, 4, 8, 8, 16]), rng.choice([1, 2, 4, 4, 8]), rng.choice([1, 1, 1, 2, 4])
        q_len = min(q_len, 8 // group)
        cached = _log_uniform(rng, 64, 32768)
        most = max(1, LARGEST_CACHE_BYTES // (8 * kv_heads * (cached + 64) * head_dim))
        return {"kind": "attention", "batch": _log_uniform(rng, 1, min(256, most)), "heads": kv_heads * group, "kv_heads": kv_heads,
                "q_len": q_len, "head_dim": head_dim, "cached": cached, "max_len": cached + q_len + rng.randrange(0, 60),
                "window": rng.choice([0, 0, 0, 1024]), "padded": rng.random() < 0.25}
    cols = _log_uniform(rng, 100, 262144)
    return {"kind": "row_op", "op": rng.choice(["softmax", "softmax", "logsumexp"]), "rows": _log_uniform(rng, 1, min(65536, 67_108_864 // cols)),
            "cols": cols}


_context = None


def _ctx():
    """The context a program keeps (its scratch belongs to it)."""
    global _context
    if _context is None:
        _context = psx.Context(0)
    return _context


def _config(case):
    return psx.SamplingConfig.make(do_sample=case["do_sample"], temperature=case["temperature"], top_k=case["top_k"],
                                   top_p=case["top_p"], min_p=case["min_p"], repetition_penalty=case["penalty"])


def _logits(gen, rows, cols, case):
    """N(0, sigma) plus a Zipf bias over random ranks; without the bias one row in a hundred has a tie at its maximum."""
    x = torch.randn((rows, cols), generator=gen, device="cuda").mul_(case["sigma"])
    if case["zeta"] > 0:
        x -= torch.rand((rows, cols), generator=gen, device="cuda").mul_(case["vocab"]).floor_().add_(1.0).log_().mul_(case["zeta"])
    else:
        n = max(1, rows // 100)
        at = torch.randint(0, cols, (n, 2), generator=gen, device="cuda")
        x[:n].scatter_(1, at, x[:n].max(dim=1, keepdim=True).values.expand(n, 2))
    return x


def _history(gen, case):
    rows, n = case["rows"], case["history"]
    if n == 0:
        return None, None
    ids = torch.randint(0, case["vocab"], (rows * n,), generator=gen, device="cuda", dtype=torch.int64)
    return ids, torch.arange(rows + 1, device="cuda", dtype=torch.int64) * n


def prepare(case, seed):
    ctx = _ctx()
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    kind, s = case["kind"], {"kind": case["kind"], "ctx": ctx}
    if kind == "top_k":
        s.update(x=torch.randn((case["rows"], case["cols"]), generator=gen, device="cuda"), k=case["k"], largest=case["largest"])
        return s
    if kind == "row_op":
        s.update(x=torch.randn((case["rows"], case["cols"]), generator=gen, device="cuda").mul_(3.0), op=case["op"])
        return s
    if kind == "attention":
        cache = (case["batch"], case["kv_heads"], case["max_len"], case["head_dim"])
        s.update(q=torch.randn((case["batch"], case["heads"], case["q_len"], case["head_dim"]), generator=gen, device="cuda"),
                 keys=torch.randn(cache, generator=gen, device="cuda"), values=torch.randn(cache, generator=gen, device="cuda"),
                 cached=case["cached"], window=case["window"], keep=None)
        if case["padded"]:  # a batch of prompts of different lengths, padded on the left
            total = case["cached"] + case["q_len"]
            pads = torch.randint(0, case["cached"] // 2, (case["batch"], 1), generator=gen, device="cuda")
            s["keep"] = (torch.arange(total, device="cuda")[None, :] >= pads).to(torch.float32).contiguous()
        return s
    rows, vocab = case["rows"], case["vocab"]
    s["config"] = _config(case)
    s["ids"], s["offsets"] = _history(gen, case)
    s["uniforms"] = torch.rand(rows, generator=gen, device="cuda", dtype=torch.float64)
    if kind == "head":
        shape = (vocab, case["d"]) if case["tied"] else (case["d"], vocab)
        s.update(weight=torch.randn(shape, generator=gen, device="cuda").mul_(3.0 / math.sqrt(case["d"])), tied=case["tied"],
                 hidden=torch.randn((rows, case["d"]), generator=gen, device="cuda"), out=ctx.alloc_outputs(rows, with_diag=False))
    elif kind == "shard":
        shards, cols = case["shards"], vocab // case["shards"]
        rank, share = seed % shards, -(-rows // shards)
        gathered = torch.zeros((shards, rows * ctx.shard_record_bytes(s["config"])), dtype=torch.uint8, device="cuda")
        for other in range(shards):  # the other GPUs' records, as the all-gather leaves them here
            logits = _logits(gen, rows, cols, case)
            if other == rank:
                s["logits"] = logits
            ctx.shard_scan(logits, other * cols, vocab, s["ids"], s["offsets"], s["config"], gathered[other])
        begin = min(rank * share, rows)
        count = min(share, rows - begin)
        s.update(gathered=gathered, own=gathered[rank], shards=shards, rows=rows, shard_begin=rank * cols, vocab=vocab,
                 row_begin=begin, row_count=count, out=ctx.alloc_outputs(count, with_diag=False))
    elif kind == "host":
        s.update(logits=_logits(gen, rows, vocab, case).cpu().numpy(), uniforms=s["uniforms"].cpu().numpy(),
                 ids=None if s["ids"] is None else s["ids"].cpu().numpy(),
                 offsets=None if s["offsets"] is None else s["offsets"].cpu().numpy())
    else:
        s.update(logits=_logits(gen, rows, vocab, case), out=ctx.alloc_outputs(rows, with_diag=False))
    return s


def run(s):
    ctx, kind = s["ctx"], s["kind"]
    if kind == "top_k":
        return ctx.top_k_rows(s["x"], s["k"], largest=s["largest"])
    if kind == "row_op":
        return ctx.softmax_rows(s["x"]) if s["op"] == "softmax" else ctx.logsumexp_rows(s["x"])
    if kind == "attention":
        return ctx.decode_attention(s["q"], s["keys"], s["values"], s["cached"], window=s["window"], key_keep=s["keep"])
    if kind == "host":
        tokens, log_probs, status, _ = ctx.sample_rows_host(s["logits"], s["ids"], s["offsets"], s["config"], s["uniforms"])
        return {"tokens": tokens, "log_probs": log_probs, "status": status}
    if kind == "head":
        out = ctx.lm_head_sample_rows(s["hidden"], s["weight"], s["ids"], s["offsets"], s["config"], s["uniforms"],
                                      vocab_by_d=s["tied"], out=s["out"])
    elif kind == "shard":
        ctx.shard_scan(s["logits"], s["shard_begin"], s["vocab"], s["ids"], s["offsets"], s["config"], s["own"])
        out = ctx.shard_merge(s["gathered"], s["shards"], s["rows"], s["vocab"], s["config"], s["uniforms"], out=s["out"],
                              row_begin=s["row_begin"], row_count=s["row_count"])
    else:
        out = ctx.sample_rows(s["logits"], s["ids"], s["offsets"], s["config"], s["uniforms"], out=s["out"])
    return {"tokens": out["tokens"], "log_probs": out["log_probs"], "status": out["status"]}


def work(case):
    """Inputs read once, outputs written once; the arithmetic that the results are made of."""
    kind = case["kind"]
    if kind == "top_k":
        n = case["rows"] * case["cols"]
        return {"bytes": 4 * n + 8 * case["rows"] * case["k"], "flops": n}
    if kind == "row_op":
        n = case["rows"] * case["cols"]
        return {"bytes": 8 * n if case["op"] == "softmax" else 4 * n + 4 * case["rows"], "flops": 4 * n}
    if kind == "attention":
        total = case["cached"] + case["q_len"]
        seen = min(total, case["window"] + case["q_len"] - 1) if case["window"] else total
        queries = case["batch"] * case["heads"] * case["q_len"] * case["head_dim"]
        return {"bytes": 8 * case["batch"] * case["kv_heads"] * seen * case["head_dim"] + 8 * queries, "flops": 4 * queries * seen}
    rows, vocab = case["rows"], case["vocab"]
    around = rows * (8 * case["history"] + 8 + 16)  # history ids, the uniform, (token, log-prob, status)
    if kind == "head":
        return {"bytes": 4 * case["d"] * (vocab + rows) + around, "flops": 2 * rows * case["d"] * vocab}
    if kind == "shard":
        cols, kept = vocab // case["shards"], max(1, case["top_k"])
        return {"bytes": 4 * rows * cols + around + 8 * kept * (rows + -(-rows // case["shards"]) * case["shards"]),
                "flops": 4 * rows * cols}
    return {"bytes": 4 * rows * vocab + around, "flops": 4 * rows * vocab}


def tolerance(case):
    """Token ids, statuses and top_k's values and columns are the same bit for bit; a log-probability, a softmax and an
    attention output are float results of 32-bit sums."""
    return "exact" if case["kind"] == "top_k" else {"rel": 1e-5}
