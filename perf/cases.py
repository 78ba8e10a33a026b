"""Performance cases: what users of this package have it do, through its public entry points.

A case is a dict of plain values; ``path`` names the entry points and the other values their sizes and options:

  prefill   attention of the prompts of one step in one layer (``ops.prefill_attn`` with the step's work list, as the executor builds it)
  decode    attention of one decode step in one layer over the paged cache (``ops.decode_plan`` and ``ops.decode_attn``)
  delta     the gated delta rule of one layer (``ops.gated_delta``), prompts or one token per sequence
  mlstm     the matrix memory of one layer (``ops.mlstm``)
  scan      the selective scan of one layer (``ops.selective_scan``)
  space     the state-space recurrence of one layer (``ops.state_space``)
  experts   a mixture of experts and the residual update behind it (``ops.moe_sort``, two ``ops.moe_gemm``, ``ops.residual_norm_pair``)
  sample    next tokens of a step (``ops.sample``)
  steps     a whole small decoder through ``Engine.replay_step``: one step over the prompts, then single tokens

Sizes are those of the repository's shapes: 16 query heads of 128 with 8 KV heads (or 4 of 256 with one), width 1024 or 2048, KV blocks
of 256 tokens.  A case's sequence lengths follow from its own numbers, its values from the seed.  ``exact`` restates every path in plain
64-bit torch.
"""
from __future__ import annotations

import math
import random

import torch

from mini_vllm_b200 import ops
from mini_vllm_b200.config import Config, qwen3_shape
from mini_vllm_b200.engine.engine import Engine
from mini_vllm_b200.engine.request import Request

BF, F32, F64 = torch.bfloat16, torch.float32, torch.float64
BLOCK = 256
EPS = 1e-6


def listed() -> list[dict]:
    attention = {"heads": 16, "kv": 8, "dim": 128, "window": 0, "cap": 0.0, "prefix": 0}
    return [
        # the prompts that join one step of a server: ragged, every other one behind an instruction of 512 tokens found in the cache
        {"name": "prefill_ragged", "path": "prefill", "seqs": 16, "low": 100, "high": 2048, **attention, "prefix": 512},
        # long documents
        {"name": "prefill_long", "path": "prefill", "seqs": 4, "low": 8192, "high": 8192, **attention},
        # layers with a window of 1024 keys and a cap on the scores, as the hybrid decoders have them
        {"name": "prefill_capped", "path": "prefill", "seqs": 8, "low": 1024, "high": 4096, **attention, "window": 1024, "cap": 30.0},
        # a decode step of many conversations
        {"name": "decode_ragged", "path": "decode", "seqs": 240, "low": 128, "high": 4096, "heads": 16, "kv": 8, "dim": 128, "window": 0},
        # the delta rule over prompts, and over one new token of each of many sequences
        {"name": "delta_prompts", "path": "delta", "decode": False, "seqs": 4, "low": 2048, "high": 2048, "heads": 16, "dim": 128},
        {"name": "delta_decode", "path": "delta", "decode": True, "seqs": 256, "low": 1, "high": 1, "heads": 16, "dim": 128},
        # matrix memory over ragged prompts
        {"name": "mlstm_prompts", "path": "mlstm", "decode": False, "seqs": 6, "low": 500, "high": 2500, "heads": 16, "dim": 128},
        # selective scan over prompts
        {"name": "scan_prompts", "path": "scan", "decode": False, "seqs": 4, "low": 2048, "high": 2048, "channels": 4096, "states": 16},
        # state-space layers over ragged prompts
        {"name": "space_prompts", "path": "space", "decode": False, "seqs": 6, "low": 500, "high": 2500, "heads": 64, "dim": 64, "groups": 8,
         "states": 128},
        # the experts of a layer over a step of prompts
        {"name": "experts_prompts", "path": "experts", "rows": 8192, "width": 2048, "inner": 1536, "experts": 16, "top": 2},
        # top-k / top-p sampling for a decode step: the smallest call
        {"name": "sample_rows", "path": "sample", "rows": 64, "vocab": 151936, "top_k": 50},
        # offline scoring with a whole (four-layer) decoder: all prompts in one step, then four single tokens of each
        {"name": "score_prompts", "path": "steps", "seqs": 32, "low": 32, "high": 2048, "layers": 4},
    ]


def _log(rng, low, high) -> int:
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng) -> dict:
    path = rng.choice(["prefill", "prefill", "decode", "delta", "mlstm", "scan", "space", "experts", "sample", "steps"])
    if path == "prefill":
        heads, kv, dim = rng.choice([(16, 8, 128), (16, 8, 128), (32, 8, 128), (4, 1, 256)])
        seqs = _log(rng, 1, 32)
        high = _log(rng, 64, min(8192, 16384 // seqs))
        options = rng.choice([(0, 0.0), (0, 0.0), (1024, 0.0), (1024, 30.0)])
        return {"path": path, "seqs": seqs, "low": _log(rng, 16, high), "high": high, "heads": heads, "kv": kv, "dim": dim,
                "window": options[0], "cap": options[1], "prefix": rng.choice([0, 0, 512])}
    if path == "decode":
        heads, kv, dim = rng.choice([(16, 8, 128), (16, 8, 128), (32, 8, 128), (4, 1, 256)])
        high = _log(rng, 64, 4096)
        return {"path": path, "seqs": _log(rng, 1, 256), "low": _log(rng, 16, high), "high": high, "heads": heads, "kv": kv, "dim": dim,
                "window": rng.choice([0, 0, 512])}
    if path in ("delta", "mlstm", "scan", "space"):
        decode = rng.random() < 0.4
        seqs = _log(rng, 1, 256 if decode else 16)
        high = 1 if decode else _log(rng, 64, min(8192, 10000 // seqs))
        case = {"path": path, "decode": decode, "seqs": seqs, "low": 1 if decode else _log(rng, 16, high), "high": high}
        if path == "scan":
            return {**case, "channels": rng.choice([2048, 4096]), "states": 16}
        if path == "space":
            heads, dim, groups = rng.choice([(64, 64, 8), (32, 64, 8), (16, 128, 16)])
            return {**case, "heads": heads, "dim": dim, "groups": groups, "states": 128}
        return {**case, "heads": rng.choice([8, 16, 32 if decode else 16]), "dim": rng.choice([64, 128, 128])}
    if path == "experts":
        return {"path": path, "rows": _log(rng, 16, 8192), "width": rng.choice([1024, 2048]), "inner": rng.choice([768, 1536]),
                "experts": 16, "top": 2}
    if path == "sample":
        return {"path": path, "rows": _log(rng, 1, 512), "vocab": rng.choice([32768, 151936, 262144]), "top_k": rng.choice([0, 20, 50])}
    seqs = _log(rng, 1, 32)
    high = _log(rng, 48, 2048)
    return {"path": path, "seqs": seqs, "low": _log(rng, 16, high), "high": high, "layers": rng.choice([2, 4])}


# ---- what follows from a case alone ----------------------------------------------------------------------------
def lengths(case) -> list[int]:
    """Tokens that each sequence brings (prompts) or has (decode steps of attention), the longest first."""
    rng = random.Random(case["seqs"] * 1000003 + case["low"] * 10007 + case["high"])
    spread = [_log(rng, case["low"], case["high"]) for _ in range(case["seqs"] - 1)]
    return [case["high"]] + spread


def prefixes(case) -> list[int]:
    """Cached tokens in front of each prompt."""
    return [case["prefix"] if i % 2 == 0 else 0 for i in range(case["seqs"])]


def _pairs(new: int, cached: int, window: int) -> int:
    reach = window or cached + new
    full = min(max(reach - cached, 0), new)            # queries that still see every key before them
    return full * cached + full * (full + 1) // 2 + (new - full) * reach


def work(case) -> dict:
    path = case["path"]
    if path == "prefill":
        lens, before, d, h, g = lengths(case), prefixes(case), case["dim"], case["heads"], case["kv"]
        pairs = sum(_pairs(n, c, case["window"]) for n, c in zip(lens, before))
        return {"bytes": 2 * (2 * sum(lens) * h * d + 2 * (sum(lens) + sum(before)) * g * d), "flops": 4 * h * d * pairs}
    if path == "decode":
        d, h, g = case["dim"], case["heads"], case["kv"]
        seen = sum(min(n, case["window"] or n) for n in lengths(case))
        return {"bytes": 2 * (2 * seen * g * d + 2 * case["seqs"] * h * d), "flops": 4 * h * d * seen}
    if path in ("delta", "mlstm", "scan", "space"):
        tokens, seqs, states = sum(lengths(case)), case["seqs"], 2 if case["decode"] else 1      # states are read as well when decoding
        if path == "scan":
            c, n = case["channels"], case["states"]
            return {"bytes": 2 * tokens * (4 * c + 2 * n) + 4 * states * seqs * c * n, "flops": 7 * tokens * c * n}
        h, d = case["heads"], case["dim"]
        if path == "space":
            n = case["states"]
            return {"bytes": 2 * tokens * (2 * h * d + 2 * case["groups"] * n + h) + 4 * states * seqs * h * n * d,
                    "flops": 5 * tokens * h * d * n}
        rows = 6 if path == "delta" else 5
        return {"bytes": 2 * tokens * (rows * h * d + h) + 4 * states * seqs * h * d * d, "flops": (7 if path == "delta" else 5) * tokens * h * d * d}
    if path == "experts":
        r, w, i, e, t = (case[k] for k in ("rows", "width", "inner", "experts", "top"))
        return {"bytes": 2 * 3 * min(e, r * t) * w * i + 4 * r * e + r * w * (2 + 2 + 2 + 8), "flops": 6 * r * t * w * i}
    if path == "sample":
        return {"bytes": 2 * case["rows"] * case["vocab"], "flops": 2 * case["rows"] * case["vocab"]}
    lens, layers = lengths(case), case["layers"]
    weights = layers * WIDTH * (2 * 16 * 128 + 2 * 8 * 128 + 3 * FF)
    rows = (1 + FED) * len(lens)
    pairs = sum(_pairs(n + FED, 0, 0) for n in lens)
    return {"bytes": (1 + FED) * 2 * (weights + VOCAB * WIDTH) + 4 * rows * VOCAB + 4 * layers * 8 * 128 * sum(n + FED * (n + FED) for n in lens),
            "flops": 2 * weights * sum(n + FED for n in lens) + 2 * VOCAB * WIDTH * rows + 4 * layers * 16 * 128 * pairs}


def tolerance(case):
    if case["path"] == "sample":
        return "exact"
    # four to five times what the outputs differ from exact() by, which is their rounding to bf16 and that of probabilities, expert inputs
    # or a decoder's activations: 2.3e-3 for the attention kernels, 1.7e-3 for the recurrences, 2.1e-3 for experts, 1.5e-2 for the decoder
    return {"rel": 6e-2 if case["path"] == "steps" else 1e-2}


# ---- inputs ----------------------------------------------------------------------------------------------------
def _gen(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(seed)


def _bf(g, *shape, scale=1.0):
    return (torch.randn(*shape, generator=g, device="cuda") * scale).to(BF)


def _ends(lens) -> torch.Tensor:
    return torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32, device="cuda")


def _pages(g, lens):
    """A block table for these lengths: a permutation of the pool's blocks, -1 behind a sequence's last."""
    per = [-(-n // BLOCK) for n in lens]
    order = torch.randperm(sum(per), generator=g, device="cuda").to(torch.int32)
    table = torch.full((len(lens), max(per)), -1, dtype=torch.int32, device="cuda")
    at = 0
    for i, n in enumerate(per):
        table[i, :n] = order[at:at + n]
        at += n
    return table, sum(per)


def _attention_inputs(case, seed):
    g, lens, before = _gen(seed), lengths(case), prefixes(case)
    h, kv, d = case["heads"], case["kv"], case["dim"]
    q = _bf(g, sum(lens), h, d)
    total = [n + c for n, c in zip(lens, before)]
    if any(before):
        table, blocks = _pages(g, total)
        k, v = _bf(g, blocks, BLOCK, kv, d), _bf(g, blocks, BLOCK, kv, d)
    else:
        table, k, v = None, _bf(g, sum(lens), kv, d), _bf(g, sum(lens), kv, d)
    return {"q": q, "k": k, "v": v, "table": table}


def _prepare_prefill(case, seed):
    s, lens = _attention_inputs(case, seed), lengths(case)
    total = [n + c for n, c in zip(lens, prefixes(case))]
    rows = ops.prefill_item_rows(case["heads"], case["kv"], case["dim"])
    items = torch.from_numpy(ops.build_prefill_items(lens, total, rows)).cuda()
    return {**s, "items": items, "cu_q": _ends(lens), "cu_k": _ends(total), "longest": max(lens), "status": ops.new_status("cuda")}


def _prepare_decode(case, seed):
    g, lens = _gen(seed), lengths(case)
    h, kv, d = case["heads"], case["kv"], case["dim"]
    table, blocks = _pages(g, lens)
    return {"q": _bf(g, len(lens), h, d), "k": _bf(g, blocks, BLOCK, kv, d), "v": _bf(g, blocks, BLOCK, kv, d), "table": table,
            "lens": torch.tensor(lens, dtype=torch.int32, device="cuda"), "ws": ops.decode_workspace(len(lens), h, d, "cuda"),
            "status": ops.new_status("cuda")}


def _recurrent(case, g) -> dict:
    """Slots, row boundaries and positions of a recurrence: prompts start at position 0, decoded tokens far behind it."""
    lens = lengths(case)
    rows = {"slots": torch.randperm(len(lens), generator=g, device="cuda").to(torch.int32), "status": ops.new_status("cuda")}
    if case["decode"]:
        return {**rows, "cu": None, "pos": torch.full((len(lens),), 1199, device="cuda")}
    return {**rows, "cu": _ends(lens), "pos": torch.cat([torch.arange(n, device="cuda") for n in lens])}


def _prepare_delta(case, seed):
    g, t, n, h, d = _gen(seed), sum(lengths(case)), case["seqs"], case["heads"], case["dim"]
    s = _recurrent(case, g)
    for name in ("q", "k", "v", "gate"):
        s[name] = _bf(g, t, h, d)
    s["a"], s["b"] = _bf(g, t, h * d), _bf(g, t, h)
    s["exp_a"] = torch.rand(h, generator=g, device="cuda") * 8 + 1
    s["bias"] = torch.full((h * d,), -4.0, device="cuda")
    s["norm"] = torch.rand(d, generator=g, device="cuda") + 0.5
    s["state"] = torch.randn(n, h, d, d, generator=g, device="cuda") * 0.1
    return s


def _prepare_mlstm(case, seed):
    g, t, n, h, d = _gen(seed), sum(lengths(case)), case["seqs"], case["heads"], case["dim"]
    s = _recurrent(case, g)
    for name in ("q", "k", "v", "gate"):
        s[name] = _bf(g, t, h, d)
    s["f"], s["i"] = _bf(g, t, h), _bf(g, t, h)
    s["f_bias"], s["i_bias"] = torch.full((h,), 4.0, device="cuda"), torch.full((h,), -2.0, device="cuda")
    s["norm"] = torch.rand(h * d, generator=g, device="cuda") + 0.5
    s["states"] = (torch.randn(n, h, d, d, generator=g, device="cuda"), torch.randn(n, h, d, generator=g, device="cuda"),
                   torch.rand(n, h, generator=g, device="cuda"))
    return s


def _prepare_scan(case, seed):
    g, t, n, c, m = _gen(seed), sum(lengths(case)), case["seqs"], case["channels"], case["states"]
    s = _recurrent(case, g)
    for name in ("u", "dt", "z"):
        s[name] = _bf(g, t, c)
    s["bc"] = _bf(g, t, 2 * m)
    s["bias"], s["skip"] = torch.full((c,), -4.0, device="cuda"), torch.rand(c, generator=g, device="cuda") + 0.5
    rate = torch.arange(1, m + 1, device="cuda").float() * (0.8 + 0.4 * torch.rand(c, 1, generator=g, device="cuda"))
    s["a"] = -rate / math.log(2.0)
    s["state"] = torch.randn(n, c, m, generator=g, device="cuda") * 0.1
    return s


def _prepare_space(case, seed):
    g, t, n, h, d = _gen(seed), sum(lengths(case)), case["seqs"], case["heads"], case["dim"]
    keys = case["groups"] * case["states"]
    s = _recurrent(case, g)
    s["xbc"], s["dt"] = _bf(g, t, h * d + 2 * keys), _bf(g, t, h)
    s["bias"], s["skip"] = torch.full((h,), -4.0, device="cuda"), torch.rand(h, generator=g, device="cuda") + 0.5
    s["a"] = -(torch.rand(h, generator=g, device="cuda") * 8 + 1) / math.log(2.0)
    s["state"] = torch.randn(n, h, case["states"], d, generator=g, device="cuda") * 0.1
    s["longest"] = 0 if case["decode"] else max(lengths(case))
    return s


def _prepare_experts(case, seed):
    g = _gen(seed)
    r, w, i, e = (case[k] for k in ("rows", "width", "inner", "experts"))
    return {"h": _bf(g, r, w), "logits": torch.randn(r, e, generator=g, device="cuda"), "up": _bf(g, e, 2, i, w, scale=w ** -0.5),
            "down": _bf(g, e, w, i, scale=i ** -0.5), "x": torch.randn(r, w, generator=g, device="cuda"), "y": _bf(g, r, w),
            "norm": (torch.rand(w, generator=g, device="cuda") + 0.5).to(BF),
            "counters": torch.zeros(e + 1, dtype=torch.int32, device="cuda"), "status": ops.new_status("cuda")}


def _prepare_sample(case, seed):
    g, r = _gen(seed), case["rows"]
    return {"logits": _bf(g, r, case["vocab"], scale=3.0), "temperature": torch.full((r,), 0.8, device="cuda"),
            "top_k": torch.full((r,), case["top_k"], dtype=torch.int32, device="cuda"), "top_p": torch.full((r,), 0.9, device="cuda"), "seed": seed}


WIDTH, FF, VOCAB, FED = 1024, 3072, 32768, 4      # the decoder of "steps"; FED: single tokens after the prompts


def _decoder(case, seed):
    """Checkpoint tensors and tokens."""
    g, w = _gen(seed), {}
    w["embed_tokens.weight"] = _bf(g, VOCAB, WIDTH, scale=0.02)
    gain = lambda n: (torch.rand(n, generator=g, device="cuda") + 0.5).to(BF)
    w["norm.weight"] = gain(WIDTH)
    for i in range(case["layers"]):
        p = f"layers.{i}."
        w[p + "self_attn.qkv_proj.weight"] = _bf(g, 32 * 128, WIDTH, scale=WIDTH ** -0.5)
        w[p + "self_attn.o_proj.weight"] = _bf(g, WIDTH, 16 * 128, scale=0.02)
        w[p + "mlp.gate_up_proj.weight"] = _bf(g, 2 * FF, WIDTH, scale=WIDTH ** -0.5)
        w[p + "mlp.down_proj.weight"] = _bf(g, WIDTH, FF, scale=0.02)
        for name, size in (("self_attn.q_norm", 128), ("self_attn.k_norm", 128), ("input_layernorm", WIDTH), ("post_attention_layernorm", WIDTH)):
            w[p + name + ".weight"] = gain(size)
    tokens = [torch.randint(VOCAB, (n + FED,), generator=g, device="cuda").tolist() for n in lengths(case)]
    return w, tokens


def _prepare_steps(case, seed):
    w, tokens = _decoder(case, seed)
    blocks = sum(-(-len(t) // BLOCK) for t in tokens) + 8
    shape = qwen3_shape(num_hidden_layers=case["layers"], hidden_size=WIDTH, intermediate_size=FF, vocab_size=VOCAB, max_position_embeddings=4096)
    engine = Engine(Config(hf_config=shape, kv_cache_num_blocks=blocks, max_num_batched_seqs=32, max_graph_batch_size=32))
    engine.executor.model.load_weights(w.items())
    return {"engine": engine, "prompts": [t[:-FED] for t in tokens], "fed": [t[-FED:] for t in tokens]}


def prepare(case, seed):
    state = {"prefill": _prepare_prefill, "decode": _prepare_decode, "delta": _prepare_delta, "mlstm": _prepare_mlstm, "scan": _prepare_scan,
             "space": _prepare_space, "experts": _prepare_experts, "sample": _prepare_sample, "steps": _prepare_steps}[case["path"]](case, seed)
    return {**state, "case": case}


# ---- the calls -------------------------------------------------------------------------------------------------
def _run_prefill(s, c):
    return ops.prefill_attn(s["q"], s["k"], s["v"], s["cu_q"], s["cu_k"], s["longest"], c["dim"] ** -0.5, c["window"] - 1, block_table=s["table"],
                            items=s["items"], softcap=c["cap"], status=s["status"])


def _run_decode(s, c):
    left = c["window"] - 1
    ops.decode_plan(s["lens"], left, c["heads"], c["kv"], c["dim"], s["ws"], block_table=s["table"], block_size=BLOCK)
    return ops.decode_attn(s["q"], s["k"], s["v"], s["lens"], s["table"], c["dim"] ** -0.5, left, s["ws"], status=s["status"])


def _run_delta(s, c):
    out = torch.empty_like(s["v"])
    ops.gated_delta(s["q"], s["k"], s["v"], s["a"], s["b"], s["gate"].flatten(1), s["exp_a"], s["bias"], s["norm"], out, s["state"], s["slots"],
                    s["cu"], s["pos"], c["dim"] ** -0.5, EPS, status=s["status"])
    return {"out": out, "state": s["state"]}


def _run_mlstm(s, c):
    out = torch.empty_like(s["v"])
    ops.mlstm(s["q"], s["k"], s["v"], s["f"], s["f_bias"], s["i"], s["i_bias"], 15.0, s["gate"].flatten(1), s["norm"], out, s["states"], s["slots"],
              s["cu"], s["pos"], c["dim"] ** -0.5, EPS, status=s["status"])
    return {"out": out, "states": list(s["states"])}


def _run_scan(s, c):
    out, m = torch.empty_like(s["u"]), c["states"]
    ops.selective_scan(s["u"], s["dt"], s["z"], s["bc"][:, :m], s["bc"][:, m:], s["bias"], s["a"], s["skip"], out, s["state"], s["slots"], s["cu"],
                       s["pos"], status=s["status"])
    return {"out": out, "state": s["state"]}


def _space_parts(s, c):
    keys = c["groups"] * c["states"]
    x, b, q = s["xbc"].split([c["heads"] * c["dim"], keys, keys], dim=1)
    return x.unflatten(1, (c["heads"], c["dim"])), b.unflatten(1, (c["groups"], c["states"])), q.unflatten(1, (c["groups"], c["states"]))


def _run_space(s, c):
    x, b, q = _space_parts(s, c)
    out = torch.empty(x.shape, dtype=BF, device="cuda")
    ops.state_space(x, b, q, s["dt"], s["bias"], s["a"], s["skip"], out, s["state"], s["slots"], s["cu"], s["pos"], longest=s["longest"],
                    status=s["status"])
    return {"out": out, "state": s["state"]}


def _run_experts(s, c):
    rows, sorted_by = ops.moe_sort(s["h"], s["logits"], c["top"], s["counters"])
    act = ops.moe_gemm(rows, s["up"], sorted_by, c["width"], gated=(7.0, 1.702, 1.0), status=s["status"])
    back = ops.moe_gemm(act, s["down"], sorted_by, c["inner"], status=s["status"])
    out, _ = ops.residual_norm_pair(s["x"], s["y"], s["norm"], None, EPS, extra=back, extra_index=sorted_by.slots, status=s["status"])
    return {"out": out, "x": s["x"]}


def _run_sample(s, c):
    if c["top_k"] == 0:
        return ops.sample(s["logits"])
    return ops.sample(s["logits"], s["temperature"], s["top_k"], s["seed"], 0, top_p=s["top_p"])


def _run_steps(s, c):
    engine = s["engine"]
    reqs = [Request([]) for _ in s["prompts"]]
    logits = [engine.replay_step([(r, t, [len(t) - 1]) for r, t in zip(reqs, s["prompts"])])]
    for j in range(FED):
        logits.append(engine.replay_step([(r, [t[j]], [0]) for r, t in zip(reqs, s["fed"])]))
    for r in reqs:
        engine.release(r)
    return logits


_RUN = {"prefill": _run_prefill, "decode": _run_decode, "delta": _run_delta, "mlstm": _run_mlstm, "scan": _run_scan, "space": _run_space,
        "experts": _run_experts, "sample": _run_sample, "steps": _run_steps}


def run(state):
    return _RUN[state["case"]["path"]](state, state["case"])


# ---- the same in plain 64-bit torch ------------------------------------------------------------------------------
def _attend(q, k, v, scale, window=0, cap=0.0):
    """q [n, heads, d] behind k, v [m, kv, d] whose last n rows are the queries' own -> [n, heads, d]."""
    n, m, per = q.shape[0], k.shape[0], q.shape[1] // k.shape[1]
    out = torch.empty(q.shape, dtype=F64, device=q.device)
    behind = torch.arange(m, device=q.device)[None, :] - torch.arange(m - n, m, device=q.device)[:, None]
    hidden = behind > 0
    if window:
        hidden |= behind <= -window
    for h in range(q.shape[1]):
        s = q[:, h].double() @ k[:, h // per].double().T * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        out[:, h] = torch.softmax(s.masked_fill_(hidden, -math.inf), dim=-1) @ v[:, h // per].double()
    return out


def _rows_of(pool, table, n):
    return pool[table[: -(-n // BLOCK)].long()].flatten(0, 1)[:n]


def _exact_prefill(case, seed):
    s, at, outs = _attention_inputs(case, seed), 0, []
    for i, (n, c) in enumerate(zip(lengths(case), prefixes(case))):
        q = s["q"][at:at + n]
        k, v = (s[x][at:at + n] if s["table"] is None else _rows_of(s[x], s["table"][i], n + c) for x in ("k", "v"))
        outs.append(_attend(q, k, v, case["dim"] ** -0.5, case["window"], case["cap"]))
        at += n
    return torch.cat(outs)


def _exact_decode(case, seed):
    s = _prepare_decode(case, seed)
    return torch.cat([_attend(s["q"][i:i + 1], *(_rows_of(s[x], s["table"][i], n) for x in ("k", "v")), case["dim"] ** -0.5, case["window"])
                      for i, n in enumerate(lengths(case))])


def _walk(case, s, state, step, **rows):
    """Walks all sequences at once, token by token: ``step(state, row tensors, rows that still run) -> (output rows, state)``; the rows are
    [sequences, ...].  ``state``: a list of tensors by slot, in place; returns the packed outputs."""
    lens = lengths(case)
    first = [0] + torch.tensor(lens).cumsum(0).tolist()
    slots = s["slots"].long()
    now = [t.double()[slots] if case["decode"] else torch.zeros(t.shape, dtype=F64, device="cuda") for t in state]
    order = sorted(range(len(lens)), key=lambda i: -lens[i])
    outs = None
    base = torch.tensor([first[i] for i in order], device="cuda")
    perm = torch.tensor(order, device="cuda")
    now = [t[perm] for t in now]
    for t in range(max(lens)):
        live = sum(lens[i] > t for i in order)
        at = base[:live] + t
        part = [x[:live] for x in now]
        o, part = step(part, {k: v[at].double() for k, v in rows.items()})
        for x, y in zip(now, part):
            x[:live] = y
        if outs is None:
            outs = torch.empty(first[-1], *o.shape[1:], dtype=F64, device="cuda")
        outs[at] = o
    final = []
    for t, x in zip(state, now):
        y = torch.empty_like(x)
        y[slots[perm]] = x
        final.append(y)
    return outs, final


def _headed_norm(o, gate, weight):
    return o / torch.sqrt((o * o).mean(-1, keepdim=True) + EPS) * weight * torch.sigmoid(gate.double())


def _exact_delta(case, seed):
    s, (h, d) = _prepare_delta(case, seed), (case["heads"], case["dim"])
    unit = lambda x: x.double() / torch.sqrt((x.double() ** 2).sum(-1, keepdim=True) + 1e-6)
    decay = torch.exp(-s["exp_a"].double()[:, None] * torch.nn.functional.softplus(s["a"].double() + s["bias"].double()).unflatten(1, (h, d)))

    def step(state, r):
        S = r["g"].unsqueeze(-1) * state[0]
        e = r["beta"].unsqueeze(-1) * (r["v"] - torch.einsum("nhkv,nhk->nhv", S, r["k"]))
        S = S + r["k"].unsqueeze(-1) * e.unsqueeze(-2)
        return torch.einsum("nhkv,nhk->nhv", S, r["q"]), [S]

    o, (state,) = _walk(case, s, [s["state"]], step, q=unit(s["q"]) * d ** -0.5, k=unit(s["k"]), v=s["v"], g=decay, beta=torch.sigmoid(s["b"].double()))
    return {"out": _headed_norm(o, s["gate"], s["norm"].double()), "state": state}


def _exact_mlstm(case, seed):
    s, (h, d) = _prepare_mlstm(case, seed), (case["heads"], case["dim"])
    capped = lambda x, bias: 15.0 * torch.tanh((x.double() + bias.double()) / 15.0)

    def step(state, r):
        S, n, m = state
        new = torch.maximum(r["f"] + m, r["i"])
        keep, take = torch.exp(r["f"] + m - new).unsqueeze(-1), torch.exp(r["i"] - new).unsqueeze(-1)
        S = keep.unsqueeze(-1) * S + (take * r["k"]).unsqueeze(-1) * r["v"].unsqueeze(-2)
        n = keep * n + take * r["k"]
        low = torch.maximum((n * r["q"]).sum(-1).abs(), torch.exp(-new)) + 1e-6
        return torch.einsum("nhkv,nhk->nhv", S, r["q"]) / low.unsqueeze(-1), [S, n, new]

    o, states = _walk(case, s, list(s["states"]), step, q=s["q"].double() * d ** -0.5, k=s["k"], v=s["v"],
                      f=torch.nn.functional.logsigmoid(capped(s["f"], s["f_bias"])), i=capped(s["i"], s["i_bias"]))
    return {"out": _headed_norm(o, s["gate"], s["norm"].double().view(h, d)), "states": states}


def _exact_scan(case, seed):
    s, m = _prepare_scan(case, seed), case["states"]
    a, skip = s["a"].double() * math.log(2.0), s["skip"].double()

    def step(state, r):
        S = torch.exp(r["dt"].unsqueeze(-1) * a) * state[0] + (r["dt"] * r["u"]).unsqueeze(-1) * r["b"].unsqueeze(1)
        y = torch.einsum("ncm,nm->nc", S, r["c"]) + skip * r["u"]
        return y * torch.nn.functional.silu(r["z"]), [S]

    o, (state,) = _walk(case, s, [s["state"]], step, u=s["u"], dt=torch.nn.functional.softplus(s["dt"].double() + s["bias"].double()), z=s["z"],
                        b=s["bc"][:, :m], c=s["bc"][:, m:])
    return {"out": o, "state": state}


def _exact_space(case, seed):
    s = _prepare_space(case, seed)
    x, b, q = _space_parts(s, case)
    per = case["heads"] // case["groups"]
    a, skip = s["a"].double() * math.log(2.0), s["skip"].double()

    def step(state, r):
        b, q = r["b"].repeat_interleave(per, 1), r["q"].repeat_interleave(per, 1)
        S = torch.exp(r["dt"] * a)[..., None, None] * state[0] + (r["dt"].unsqueeze(-1) * b).unsqueeze(-1) * r["x"].unsqueeze(-2)
        return torch.einsum("nhkv,nhk->nhv", S, q) + skip[:, None] * r["x"], [S]

    o, (state,) = _walk(case, s, [s["state"]], step, x=x, b=b, q=q, dt=torch.nn.functional.softplus(s["dt"].double() + s["bias"].double()))
    return {"out": o, "state": state}


def _exact_experts(case, seed):
    s = _prepare_experts(case, seed)
    x = s["x"].double() + s["y"].double()
    score, pick = torch.topk(s["logits"].double(), case["top"], dim=-1)
    score, h = torch.sigmoid(score), s["h"].double()
    for e in range(case["experts"]):
        token, place = torch.nonzero(pick == e, as_tuple=True)
        if token.numel():
            up = s["up"][e].double()
            rows = h[token] * score[token, place].unsqueeze(-1)
            g, u = (rows @ up[0].T).clamp(max=7.0), (rows @ up[1].T).clamp(-7.0, 7.0)
            x.index_add_(0, token, (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ s["down"][e].double().T)
    return {"out": x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS) * s["norm"].double(), "x": x}


def _exact_steps(case, seed):
    w, tokens = _decoder(case, seed)
    w = {k: v.double() for k, v in w.items()}
    rms = lambda x, weight: x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS) * weight
    logits = [[] for _ in range(1 + FED)]
    for seq in tokens:
        n = len(seq)
        angle = torch.arange(n, device="cuda", dtype=F64)[:, None] * 1e6 ** (-torch.arange(64, device="cuda", dtype=F64) / 64)
        cos, sin = torch.cos(angle)[:, None, :], torch.sin(angle)[:, None, :]

        def turn(t):
            a, b = t.chunk(2, dim=-1)
            return torch.cat([a * cos - b * sin, b * cos + a * sin], dim=-1)

        x = w["embed_tokens.weight"][torch.tensor(seq, device="cuda")]
        for i in range(case["layers"]):
            p = f"layers.{i}."
            qkv = rms(x, w[p + "input_layernorm.weight"]) @ w[p + "self_attn.qkv_proj.weight"].T
            q, k, v = (t.unflatten(1, (-1, 128)) for t in qkv.split([16 * 128, 8 * 128, 8 * 128], dim=1))
            q, k = turn(rms(q, w[p + "self_attn.q_norm.weight"])), turn(rms(k, w[p + "self_attn.k_norm.weight"]))
            x = x + _attend(q, k, v, 128 ** -0.5).flatten(1) @ w[p + "self_attn.o_proj.weight"].T
            gate, up = (rms(x, w[p + "post_attention_layernorm.weight"]) @ w[p + "mlp.gate_up_proj.weight"].T).chunk(2, dim=1)
            x = x + (torch.nn.functional.silu(gate) * up) @ w[p + "mlp.down_proj.weight"].T
        last = rms(x[-1 - FED:], w["norm.weight"]) @ w["embed_tokens.weight"].T
        for j in range(1 + FED):
            logits[j].append(last[j])
    return [torch.stack(rows) for rows in logits]


def exact(case, seed):
    if case["path"] == "sample":      # which of the likely tokens comes out follows from the generator's stream
        return None
    return {"prefill": _exact_prefill, "decode": _exact_decode, "delta": _exact_delta, "mlstm": _exact_mlstm, "scan": _exact_scan,
            "space": _exact_space, "experts": _exact_experts, "steps": _exact_steps}[case["path"]](case, seed)
