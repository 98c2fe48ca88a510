"""What a user of the engine has it do, as cases that can be timed and compared.

Two cases are whole steps through ``ModelRunner.step`` (they return logits); the others are single layers as a program
that builds a decoder from the parts calls them: ``build_part(...)``, ``part.forward(ctx, rows, cache, ...)``.  Decode
layers run inside a CUDA graph, as the engine's own decode steps do; prompt steps are launched one by one, as the
engine's are.  Layer sizes are those of the benchmark configuration (7b), of the two workloads (14b), of the design
comparison's small size (1.5b) and of the model the reference was validated with (0.5b).

Every input comes from a seed through plain torch; ``exact`` computes the same outputs in 64 bits without the package.
"""
from __future__ import annotations

import math
import random

import torch
import torch.nn.functional as F

import tessweave_engine_b200 as tw
from tessweave_engine_b200.parts.base import Runtime, StepContext, Workspace, build_part, dense_delta

DEVICE = "cuda:0"
PAGE = 16
VOCAB = 152064
THETA = 1000000.0
EPS = 1e-6

# hidden, query heads, key/value heads, head size, feed-forward size
SIZES = {
    "0.5b": (896, 14, 2, 64, 4864),
    "1.5b": (1536, 12, 2, 128, 8960),
    "7b": (3584, 28, 4, 128, 18944),
    "14b": (5120, 40, 8, 128, 13824),
}


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed() -> list[dict]:
    return [
        # generation at the benchmark's point: eight requests in the middle of their answers, a whole decode step
        # (embedding, layers, logits) of a decoder cut to four layers
        {"name": "decode_step_7b_b8_ctx4096", "kind": "step", "size": "7b", "layers": 4, "singles": 8, "least": 4096,
         "most": 4096, "portions": "", "prefixes": ""},
        # continuous batching: two prompt portions (one a continuation) share a step with thirty generating requests
        {"name": "mixed_step_14b", "kind": "step", "size": "14b", "layers": 4, "singles": 30, "least": 130, "most": 2200,
         "portions": "301,182", "prefixes": "512,0"},
        # reading a prompt: the attention layer of one 2,048-token prompt (projections, rotation, cache, attention)
        {"name": "attention_prompt_7b_2048", "kind": "attention", "size": "7b", "dtype": "bfloat16", "portions": "2048",
         "prefixes": "0", "singles": 0, "least": 0, "most": 0},
        # a large batch generating at uneven lengths: the attention layer of 64 requests
        {"name": "attention_decode_7b_b64", "kind": "attention", "size": "7b", "dtype": "bfloat16", "portions": "",
         "prefixes": "", "singles": 64, "least": 300, "most": 8000},
        # one chat on a small model: the smallest call there is
        {"name": "attention_decode_1.5b_b1", "kind": "attention", "size": "1.5b", "dtype": "bfloat16", "portions": "",
         "prefixes": "", "singles": 1, "least": 700, "most": 700},
        # replaying recorded requests in 32 bits (what the engine is validated with): prompts of odd lengths
        {"name": "attention_prompt_0.5b_fp32", "kind": "attention", "size": "0.5b", "dtype": "float32",
         "portions": "777,1000,37", "prefixes": "0,0,0", "singles": 0, "least": 0, "most": 0},
        # the dense feed-forward of a 2,048-token prompt
        {"name": "mlp_prompt_7b_2048", "kind": "mlp", "size": "7b", "dtype": "bfloat16", "rows": 2048},
        # a matrix memory over a whole prompt (Sapatar's mLSTM)
        {"name": "mlstm_prompt_2048", "kind": "recurrent", "rule": "mlstm", "hidden": 3584, "heads": 14, "dim": 128,
         "portions": "2048"},
        # the gated delta rule (Nufatar) over three prompts of odd lengths in one step
        {"name": "delta_prompts_ragged", "kind": "recurrent", "rule": "gated_delta", "hidden": 3584, "heads": 14, "dim": 128,
         "portions": "777,1024,201"},
        # eight experts, two chosen, and a shared one (Sapatar, Varivik): a prompt, and eight generating requests
        {"name": "experts_prompt_2048", "kind": "experts", "hidden": 3584, "experts": 8, "top": 2, "ff": 4736, "rows": 2048},
        {"name": "experts_decode_b8", "kind": "experts", "hidden": 3584, "experts": 8, "top": 2, "ff": 4736, "rows": 8},
        # attention over low-rank latents (Dugudra, Bavetar): eight generating requests
        {"name": "latent_decode_b8_ctx4096", "kind": "latent", "hidden": 3584, "heads": 28, "dim": 128, "rot": 64,
         "q_rank": 1536, "kv_rank": 192, "singles": 8, "least": 4096, "most": 4096},
    ]


def _log(rng: random.Random, low: int, high: int) -> int:
    return max(low, min(high, round(math.exp(rng.uniform(math.log(low), math.log(high))))))


def _cut(rng: random.Random, total: int) -> str:
    """``total`` tokens as one to three portions."""
    parts = rng.randint(1, 3) if total >= 64 else 1
    at = sorted(rng.sample(range(1, total), parts - 1)) + [total]
    return ",".join(str(b - a) for a, b in zip([0] + at, at))


def _draw(rng: random.Random) -> dict:
    kind = rng.choice(["step", "mixed", "attention_prompt", "attention_prompt", "attention_decode", "attention_decode",
                       "attention_fp32", "mlp", "recurrent", "recurrent", "recurrent", "experts_prompt", "experts_decode", "latent"])
    if kind == "step":
        least = _log(rng, 128, 3000)
        return {"kind": "step", "size": rng.choice(["0.5b", "1.5b", "7b", "14b"]), "layers": rng.randint(1, 4),
                "singles": _log(rng, 1, 64), "least": least, "most": _log(rng, least, 4096), "portions": "", "prefixes": ""}
    if kind == "mixed":
        portions = _cut(rng, _log(rng, 64, 512))
        return {"kind": "step", "size": rng.choice(["0.5b", "1.5b", "7b", "14b"]), "layers": rng.randint(1, 4),
                "singles": rng.randint(0, 31), "least": 64, "most": _log(rng, 256, 2200), "portions": portions,
                "prefixes": ",".join(str(rng.choice([0, 0, 512, 1030])) for _ in portions.split(","))}
    if kind == "attention_prompt":
        portions = _cut(rng, _log(rng, 128, 2048))
        return {"kind": "attention", "size": rng.choice(["0.5b", "1.5b", "7b", "14b"]), "dtype": "bfloat16", "portions": portions,
                "prefixes": ",".join(str(rng.choice([0, 0, 512, 1030])) for _ in portions.split(",")), "singles": 0, "least": 0,
                "most": 0}
    if kind == "attention_decode":
        least = _log(rng, 100, 4000)
        return {"kind": "attention", "size": rng.choice(["0.5b", "1.5b", "7b", "14b"]), "dtype": "bfloat16", "portions": "",
                "prefixes": "", "singles": _log(rng, 1, 64), "least": least, "most": _log(rng, least, 8000)}
    if kind == "attention_fp32":
        portions = _cut(rng, _log(rng, 64, 1814))
        return {"kind": "attention", "size": rng.choice(["0.5b", "1.5b"]), "dtype": "float32", "portions": portions,
                "prefixes": ",".join(str(rng.choice([0, 0, 300])) for _ in portions.split(",")), "singles": 0, "least": 0, "most": 0}
    if kind == "mlp":
        return {"kind": "mlp", "size": rng.choice(["0.5b", "1.5b", "7b", "14b"]), "dtype": "bfloat16", "rows": _log(rng, 128, 2048)}
    if kind == "recurrent":
        return {"kind": "recurrent", "rule": rng.choice(["mlstm", "retention", "gla", "gated_delta"]),
                "hidden": rng.choice([1536, 3584]), "heads": rng.choice([6, 8, 14]), "dim": rng.choice([64, 128]),
                "portions": _cut(rng, _log(rng, 128, 2048))}
    if kind == "experts_prompt":
        return {"kind": "experts", "hidden": rng.choice([1536, 3584]), "experts": 8, "top": rng.choice([2, 3]),
                "ff": rng.choice([2240, 4736]), "rows": _log(rng, 128, 2048)}
    if kind == "experts_decode":
        return {"kind": "experts", "hidden": rng.choice([1536, 3584]), "experts": 8, "top": rng.choice([2, 3]),
                "ff": rng.choice([2240, 4736]), "rows": _log(rng, 1, 64)}
    least = _log(rng, 100, 4000)
    return {"kind": "latent", "hidden": rng.choice([1536, 3584]), "heads": rng.choice([12, 28]), "dim": 128, "rot": 64,
            "q_rank": 1536, "kv_rank": 192, "singles": _log(rng, 1, 32), "least": least, "most": _log(rng, least, 4096)}


def _cost(case: dict) -> float:
    """What a case costs at least, in seconds of a B200."""
    w = work(case)
    rate = 7e13 if case.get("dtype") == "float32" else 1.6e15
    return max(w["bytes"] / 6.5e12, w["flops"] / rate)


def draw(rng: random.Random) -> dict:
    limits: dict[str, float] = {}
    for case in listed():
        limits[case["kind"]] = max(limits.get(case["kind"], 0.0), _cost(case))
    while True:
        case = _draw(rng)
        if _cost(case) <= limits[case["kind"]]:
            return case


# ---------------------------------------------------------------------------
# requests of a step
# ---------------------------------------------------------------------------
def _numbers(text: str) -> list[int]:
    return [int(t) for t in text.split(",")] if text else []


def _requests(case: dict) -> tuple[list[int], list[int]]:
    """(tokens each request brings, tokens it already holds): the portions first, then the single tokens."""
    lens = _numbers(case.get("portions", ""))
    held = _numbers(case.get("prefixes", "")) or [0] * len(lens)
    n = case.get("singles", 0)
    for i in range(n):       # total lengths spread evenly from `least` to `most`, the longest neither first nor last
        k = (i * 7 + 3) % n if math.gcd(7, n) == 1 else i
        total = case["least"] + (case["most"] - case["least"]) * k // max(1, n - 1)
        lens.append(1)
        held.append(max(0, total - 1))
    return lens, held


def _generator(seed: int) -> torch.Generator:
    return torch.Generator(device=DEVICE).manual_seed(int(seed) * 1000003 + 17)


def _draw_tensors(decls, gen: torch.Generator, dtype: torch.dtype) -> dict[str, torch.Tensor]:
    """Weights by name.  decls: (name, shape, rule); matrices in the run's type, vectors in 32 bits."""
    out = {}
    for name, shape, rule in decls:
        t = torch.randn(shape, generator=gen, device=DEVICE, dtype=torch.float32)
        if rule == "matrix":
            out[name] = (0.02 * t).to(dtype)
        elif rule == "vector":
            out[name] = 0.02 * t
        elif rule == "norm":
            out[name] = 1.0 + 0.1 * t
        elif rule == "wide":
            out[name] = 0.4 * t
        elif rule == "forget":          # a forget gate's bias: memories of some tens to hundreds of tokens
            out[name] = 4.0 + t
        elif rule == "router":
            out[name] = (0.1 * t).to(dtype)
    return out


def _rows(gen: torch.Generator, n: int, width: int, dtype: torch.dtype) -> torch.Tensor:
    """Rows as a norm leaves them: unit scale."""
    return torch.randn((n, width), generator=gen, device=DEVICE, dtype=torch.float32).to(dtype)


def _dtype(case: dict) -> torch.dtype:
    return torch.float32 if case.get("dtype") == "float32" else torch.bfloat16


# ---------------------------------------------------------------------------
# weights and held keys of each kind, in plain torch
# ---------------------------------------------------------------------------
def _attention_decls(hidden, heads, kv, dim, prefix=""):
    return [(prefix + "q_proj.weight", (heads * dim, hidden), "matrix"), (prefix + "k_proj.weight", (kv * dim, hidden), "matrix"),
            (prefix + "v_proj.weight", (kv * dim, hidden), "matrix"), (prefix + "q_proj.bias", (heads * dim,), "vector"),
            (prefix + "k_proj.bias", (kv * dim,), "vector"), (prefix + "v_proj.bias", (kv * dim,), "vector"),
            (prefix + "o_proj.weight", (hidden, heads * dim), "matrix")]


def _mlp_decls(hidden, ff, prefix=""):
    return [(prefix + "gate_proj.weight", (ff, hidden), "matrix"), (prefix + "up_proj.weight", (ff, hidden), "matrix"),
            (prefix + "down_proj.weight", (hidden, ff), "matrix")]


def _layer_decls(case):
    hidden, heads, kv, dim, ff = SIZES[case["size"]]
    decls = [("model.embed_tokens.weight", (VOCAB, hidden), "matrix")]
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        decls += [(p + "input_layernorm.weight", (hidden,), "norm"), (p + "post_attention_layernorm.weight", (hidden,), "norm")]
        decls += _attention_decls(hidden, heads, kv, dim, p + "self_attn.") + _mlp_decls(hidden, ff, p + "mlp.")
    return decls + [("model.norm.weight", (hidden,), "norm"), ("lm_head.weight", (VOCAB, hidden), "matrix")]


def _recurrent_decls(case):
    hid, H, D = case["hidden"], case["heads"], case["dim"]
    a = H * D
    if case["rule"] == "gated_delta":
        q = (H // 2) * D
        return [("q", (q, hid), "matrix"), ("k", (q, hid), "matrix"), ("v", (a, hid), "matrix"), ("q.conv", (q, 4), "wide"),
                ("k.conv", (q, 4), "wide"), ("v.conv", (a, 4), "wide"), ("b", (H, hid), "matrix"), ("a", (H, hid), "matrix"),
                ("A_log", (H,), "vector"), ("dt_bias", (H,), "vector"), ("norm", (D,), "norm"), ("g", (a, hid), "matrix"),
                ("o", (hid, a), "matrix")]
    decls = [("q", (a, hid), "matrix"), ("k", (a, hid), "matrix"), ("v", (a, hid), "matrix"), ("g", (a, hid), "matrix"),
             ("o", (hid, a), "matrix")]
    if case["rule"] == "mlstm":
        decls += [("i", (H, hid), "matrix"), ("i.b", (H,), "vector"), ("f", (H, hid), "matrix"), ("f.b", (H,), "forget"),
                  ("norm", (a,), "norm")]
    if case["rule"] == "gla":
        decls += [("a1", (64, hid), "matrix"), ("a2", (a, 64), "matrix"), ("a2.b", (a,), "wide"), ("norm", (D,), "norm")]
    return decls


def _recurrent_spec(case):
    hid, H, D = case["hidden"], case["heads"], case["dim"]
    if case["rule"] == "gated_delta":
        return tw.PartSpec("gated_delta", {"hidden": hid, "n_heads": H, "n_qk_heads": H // 2, "key_dim": D, "value_dim": D,
                                           "conv_taps": 4, "eps": EPS})
    params = {"hidden": hid, "n_heads": H, "key_dim": D, "value_dim": D, "eps": EPS}
    if case["rule"] == "mlstm":
        params["gate_cap"] = 15.0
    if case["rule"] == "gla":
        params.update(decay_rank=64, tau=16.0)
    if case["rule"] == "retention":
        params.update(decay=tuple(_retention_decay(h) for h in range(H)), position=tw.PartSpec("rope", {"theta": THETA, "dims": D}))
    return tw.PartSpec(case["rule"], params)


def _retention_decay(h: int) -> float:
    return 1.0 - 2.0 ** -(5 + h % 8)


def _experts_decls(case):
    hid, ff, E = case["hidden"], case["ff"], case["experts"]
    decls = [("router", (E, hid), "router"), ("router.b", (E,), "vector")]
    for e in range(E):
        decls += [(f"e{e}.gate", (ff, hid), "matrix"), (f"e{e}.up", (ff, hid), "matrix"), (f"e{e}.down", (hid, ff), "matrix")]
    return decls + [("shared.gate", (ff, hid), "matrix"), ("shared.up", (ff, hid), "matrix"), ("shared.down", (hid, ff), "matrix"),
                    ("shared.sg", (1, hid), "matrix")]


def _latent_decls(case):
    hid, H, D, R, C, Q = (case[k] for k in ("hidden", "heads", "dim", "rot", "kv_rank", "q_rank"))
    return [("dq", (Q, hid), "matrix"), ("dq.norm", (Q,), "norm"), ("uq", (H * (D + R), Q), "matrix"), ("dkv", (C + R, hid), "matrix"),
            ("dkv.norm", (C,), "norm"), ("uk", (H * D, C), "matrix"), ("uv", (H * D, C), "matrix"), ("g", (H, hid), "matrix"),
            ("sink", (H,), "wide"), ("o", (hid, H * D), "matrix")]


def _held(case, gen, heads, dim, layers=1):
    """Keys and values each request already holds, by layer: lists of [tokens, heads, dim] (keys as cached: rotated)."""
    _, held = _requests(case)
    dt = _dtype(case)
    make = lambda n: torch.randn((n, heads, dim), generator=gen, device=DEVICE, dtype=torch.float32).to(dt)   # noqa: E731
    return [[(make(n), make(n)) for n in held] for _ in range(layers)]


def _inputs(case: dict, seed: int) -> dict:
    """Everything random in a case, in plain torch: weights by name, rows or token ids, held keys and values."""
    gen, dt, kind = _generator(seed), _dtype(case), case["kind"]
    if kind == "step":
        hidden, heads, kv, dim, _ = SIZES[case["size"]]
        lens, _ = _requests(case)
        return {"weights": _draw_tensors(_layer_decls(case), gen, dt), "held": _held(case, gen, kv, dim, case["layers"]),
                "tokens": torch.randint(0, VOCAB, (sum(lens),), generator=gen, device=DEVICE)}
    if kind == "attention":
        hidden, heads, kv, dim, _ = SIZES[case["size"]]
        return {"weights": _draw_tensors(_attention_decls(hidden, heads, kv, dim), gen, dt), "held": _held(case, gen, kv, dim),
                "rows": _rows(gen, sum(_requests(case)[0]), hidden, dt)}
    if kind == "mlp":
        hidden, _, _, _, ff = SIZES[case["size"]]
        return {"weights": _draw_tensors(_mlp_decls(hidden, ff), gen, dt), "rows": _rows(gen, case["rows"], hidden, dt)}
    if kind == "recurrent":
        return {"weights": _draw_tensors(_recurrent_decls(case), gen, dt),
                "rows": _rows(gen, sum(_requests(case)[0]), case["hidden"], dt)}
    if kind == "experts":
        return {"weights": _draw_tensors(_experts_decls(case), gen, dt), "rows": _rows(gen, case["rows"], case["hidden"], dt)}
    if kind == "latent":
        weights = _draw_tensors(_latent_decls(case), gen, dt)
        return {"weights": weights, "held": _held(case, gen, 1, case["kv_rank"] + case["rot"]),
                "rows": _rows(gen, case["singles"], case["hidden"], dt)}
    raise ValueError(f"unknown kind {kind!r}")


# ---------------------------------------------------------------------------
# prepare and run: the package's public entry points
# ---------------------------------------------------------------------------
def _fill(decls, weights: dict[str, torch.Tensor]) -> None:
    for name, decl in decls:
        decl.dest.copy_(weights[name].view(decl.dest.shape))


def _context(rt: Runtime, lens: list[int], held: list[int], fixed: bool) -> StepContext:
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=rt.device)    # noqa: E731
    starts = [sum(lens[:i]) for i in range(len(lens))]
    slots = list(range(len(lens)))
    kv = [a + b for a, b in zip(lens, held)]
    return StepContext(
        runtime=rt, workspace=Workspace(rt.device), n_tokens=sum(lens), n_seqs=len(lens), token_ids=i32([0] * sum(lens)),
        positions=i32([h + t for n, h in zip(lens, held) for t in range(n)]),
        seq_of_token=i32([i for i, n in enumerate(lens) for _ in range(n)]), seq_slot=i32(slots), seq_q_start=i32(starts),
        seq_q_len=i32(lens), seq_kv_len=i32(kv), status=torch.zeros(1, dtype=torch.int32, device=rt.device), host_slot=slots,
        host_q_start=starts, host_q_len=list(lens), host_kv_len=kv, max_q_len=max(lens), max_kv_len=max(kv),
        decode_only=all(n == 1 for n in lens), fixed_shape=fixed)


def _cache(needs, rt: Runtime, lens: list[int], held: list[int], keys_values) -> tw.CacheManager:
    """A cache whose requests hold ``keys_values`` (by layer and request) and have room for the step's tokens."""
    total = [a + b for a, b in zip(lens, held)]
    cache = tw.CacheManager(needs, PAGE, sum(-(-t // PAGE) for t in total), len(lens), max(total), rt.dtype, rt.device,
                            prefix_cache=False)
    leases = [cache.admit(None) for _ in lens]
    for lease, t in zip(leases, total):
        cache.ensure(lease, t)
    cache.sync_tables()
    assert [lease.slot for lease in leases] == list(range(len(lens)))
    for layer, requests in enumerate(keys_values or []):
        view = cache.view(layer)
        for lease, (k, v) in zip(leases, requests):
            n = k.shape[0]
            if not n:
                continue
            pages = torch.tensor(lease.tables[0][:-(-n // PAGE)], dtype=torch.long, device=rt.device)
            for dest, rows in ((view.k_pages, k), (view.v_pages, v)):
                if dest is view.v_pages and dest.data_ptr() == view.k_pages.data_ptr():
                    continue             # one set of pages is both
                full = F.pad(rows, (0, 0, 0, 0, 0, len(pages) * PAGE - n)).view(len(pages), PAGE, *rows.shape[1:])
                dest[pages] = full.transpose(1, 2).to(dest.dtype)
    return cache


def _captured(call):
    """``call`` as a CUDA graph, as the engine runs its decode steps; returns the graph and the call's outputs."""
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(2):
            call()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = call()
    return graph, out


@torch.inference_mode()
def prepare(case: dict, seed: int) -> dict:
    given, dt, kind = _inputs(case, seed), _dtype(case), case["kind"]
    rt = Runtime(torch.device(DEVICE), dt)
    if kind == "step":
        hidden, heads, kv, dim, ff = SIZES[case["size"]]
        config = {"architectures": ["Qwen2ForCausalLM"], "model_type": "qwen2", "vocab_size": VOCAB, "hidden_size": hidden,
                  "intermediate_size": ff, "num_hidden_layers": case["layers"], "num_attention_heads": heads,
                  "num_key_value_heads": kv, "head_dim": dim, "rope_theta": THETA, "rms_norm_eps": EPS,
                  "max_position_embeddings": 32768, "tie_word_embeddings": False, "use_sliding_window": False,
                  "hidden_act": "silu", "initializer_range": 0.02}
        cfg, spec = tw.resolve(config)
        model = tw.Model(spec, rt, config=cfg)
        _fill(model.weight_decls().items(), given["weights"])
        model.finalize()
        lens, held = _requests(case)
        cache = _cache(model.cache_needs(), rt, lens, held, given["held"])
        runner = tw.ModelRunner(model, cache, max_step_tokens=max(sum(lens), len(lens)), max_step_seqs=len(lens),
                                max_logit_rows=len(lens))
        ids, entries = given["tokens"].tolist(), []
        for i, (n, h) in enumerate(zip(lens, held)):
            at = sum(lens[:i])
            entries.append(tw.StepEntry(i, ids[at:at + n], h, [n - 1]))
        if all(n == 1 for n in lens):
            runner.step(entries)         # an engine that generates has captured its decode graphs
        return {"kind": kind, "runner": runner, "entries": entries}
    rows = given["rows"]
    if kind in ("mlp", "experts"):
        if kind == "mlp":
            hidden, _, _, _, ff = SIZES[case["size"]]
            spec = tw.PartSpec("swiglu", {"hidden": hidden, "intermediate": ff})
        else:
            spec = tw.PartSpec("routed_experts", {
                "hidden": case["hidden"], "experts": case["experts"], "top": case["top"], "intermediate": case["ff"],
                "shared": tw.PartSpec("swiglu", {"hidden": case["hidden"], "intermediate": case["ff"], "names": ("gate", "up", "down")}),
                "shared_gate": True})
        part = build_part("feed_forward", spec, rt)
        decode = case["rows"] <= 64
        ctx = _context(rt, [1] * case["rows"] if decode else [case["rows"]], [100] * case["rows"] if decode else [0], decode)
        call = lambda: dense_delta(ctx, part.forward(ctx, rows), dt)        # noqa: E731
        cache = None
    else:
        lens, held = _requests(case)
        if kind == "attention":
            hidden, heads, kv, dim, _ = SIZES[case["size"]]
            spec = tw.PartSpec("gqa_attention", {"hidden": hidden, "n_heads": heads, "n_kv_heads": kv, "head_dim": dim, "qkv_bias": True,
                                                 "position": tw.PartSpec("rope", {"theta": THETA})})
        elif kind == "recurrent":
            spec = _recurrent_spec(case)
        else:
            spec = tw.PartSpec("latent_attention", {
                "hidden": case["hidden"], "n_heads": case["heads"], "head_dim": case["dim"], "rot_dim": case["rot"],
                "v_head_dim": case["dim"], "q_rank": case["q_rank"], "kv_rank": case["kv_rank"],
                "scale": (case["dim"] + case["rot"]) ** -0.5, "eps": EPS, "gate": "heads", "sink": "sink",
                "position": tw.PartSpec("rope_interleaved", {"theta": THETA, "dims": case["rot"]})})
        part = build_part("mixer", spec, rt)
        cache = _cache([(part.cache_need(), None)], rt, lens, held, given.get("held"))
        decode = all(n == 1 for n in lens)
        ctx = _context(rt, lens, held, decode)
        view = cache.view(0)
        if kind == "recurrent":
            def call():
                view.state.zero_()       # new prompts: admission gives them a zeroed state
                return dense_delta(ctx, part.forward(ctx, rows, view, True), dt), view.state
        else:
            call = lambda: dense_delta(ctx, part.forward(ctx, rows, view, True), dt)       # noqa: E731
    _fill([(d.name, d) for d in part.weights()], given["weights"])
    part.finalize()
    state = {"kind": kind, "call": call, "keep": (part, ctx, cache, rows), "graph": None}
    if decode:
        state["graph"], state["out"] = _captured(call)
    return state


@torch.inference_mode()
def run(state: dict):
    if state["kind"] == "step":
        return state["runner"].step(state["entries"])
    if state["graph"] is not None:
        state["graph"].replay()
        return state["out"]
    return state["call"]()


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _attention_work(case, hidden, heads, kv, dim, element):
    lens, held = _requests(case)
    rows = sum(lens)
    pairs = sum(n * h + n * (n + 1) // 2 for n, h in zip(lens, held))
    weights = (2 * heads + 2 * kv) * dim * hidden
    return {"bytes": element * (weights + 2 * kv * dim * (sum(held) + rows)),
            "flops": 2 * rows * weights + 4 * heads * dim * pairs}, rows


def work(case: dict) -> dict:
    kind = case["kind"]
    e = 4 if case.get("dtype") == "float32" else 2
    if kind == "step":
        hidden, heads, kv, dim, ff = SIZES[case["size"]]
        a, rows = _attention_work(case, hidden, heads, kv, dim, e)
        lens, _ = _requests(case)
        mlp = 3 * hidden * ff
        return {"bytes": case["layers"] * (a["bytes"] + e * mlp) + e * hidden * (VOCAB + rows) + 4 * len(lens) * VOCAB,
                "flops": case["layers"] * (a["flops"] + 2 * rows * mlp) + 2 * len(lens) * VOCAB * hidden}
    if kind == "attention":
        hidden, heads, kv, dim, _ = SIZES[case["size"]]
        a, rows = _attention_work(case, hidden, heads, kv, dim, e)
        return {"bytes": a["bytes"] + 2 * e * rows * hidden, "flops": a["flops"]}
    if kind == "mlp":
        hidden, _, _, _, ff = SIZES[case["size"]]
        return {"bytes": e * (3 * hidden * ff + 2 * case["rows"] * hidden), "flops": 6 * case["rows"] * hidden * ff}
    if kind == "recurrent":
        hid, H, D = case["hidden"], case["heads"], case["dim"]
        lens, _ = _requests(case)
        weights = sum(math.prod(shape) for _, shape, rule in _recurrent_decls(case) if rule == "matrix")
        return {"bytes": e * (weights + 2 * sum(lens) * hid) + 4 * len(lens) * H * D * D,
                "flops": 2 * sum(lens) * weights + 4 * sum(lens) * H * D * D}
    if kind == "experts":
        hid, ff, rows = case["hidden"], case["ff"], case["rows"]
        touched = min(case["experts"], rows * case["top"]) + 1
        return {"bytes": e * (touched * 3 * hid * ff + 2 * rows * hid), "flops": 6 * rows * (case["top"] + 1) * hid * ff}
    hid, H, D, R, C, Q = (case[k] for k in ("hidden", "heads", "dim", "rot", "kv_rank", "q_rank"))
    weights = sum(math.prod(shape) for _, shape, rule in _latent_decls(case) if rule == "matrix")
    _, held = _requests(case)
    keys = sum(held) + len(held)
    return {"bytes": e * (weights + keys * (C + R) + 2 * len(held) * hid),
            "flops": 2 * len(held) * weights + 2 * H * keys * (2 * C + R)}


def tolerance(case: dict) -> dict:
    """bfloat16: a change in the order of a sum moves roundings of 2^-9 in the projections, the attention's operands and
    the result; 32 bits: sums of up to some thousand products."""
    if case.get("dtype") == "float32":
        return {"rel": 1e-5}
    if case["kind"] == "step":
        return {"rel": 4e-2}         # four layers: 0.010 to 0.015 from 64 bits
    if case["kind"] == "mlp":
        return {"rel": 1e-2}         # 0.0023 from 64 bits
    return {"rel": 2e-2}             # 0.003 to 0.007 from 64 bits


# ---------------------------------------------------------------------------
# the same in 64 bits, without the package
# ---------------------------------------------------------------------------
def _rms(x: torch.Tensor) -> torch.Tensor:
    return x / torch.sqrt(x.square().mean(-1, keepdim=True) + EPS)


def _rotate(x: torch.Tensor, positions: torch.Tensor, dims: int, neighbours: bool = False) -> torch.Tensor:
    """x [..., tokens, heads, dims]: pairs (i, i + dims / 2), or (2 i, 2 i + 1)."""
    inv = THETA ** (-torch.arange(0, dims, 2, dtype=torch.float64, device=x.device) / dims)
    ang = positions.double()[:, None] * inv
    c, s = ang.cos()[:, None], ang.sin()[:, None]
    if neighbours:
        a, b = x[..., 0::2], x[..., 1::2]
        return torch.stack((a * c - b * s, b * c + a * s), -1).flatten(-2)
    a, b = x[..., :dims // 2], x[..., dims // 2:]
    return torch.cat((a * c - b * s, b * c + a * s), -1)


def _attend(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, first: int, scale: float, sink=None) -> torch.Tensor:
    """q [n, H, D] at positions first ...; k, v [m, G, D]; softmax over the keys at and before a query."""
    n, H, _ = q.shape
    m, G, _ = k.shape
    at = first + torch.arange(n, device=q.device)
    hidden = torch.arange(m, device=q.device)[None, :] > at[:, None]
    out = torch.empty(n, H, v.shape[-1], dtype=q.dtype, device=q.device)
    for h in range(H):
        g = h // (H // G)
        s = (q[:, h] @ k[:, g].T * scale).masked_fill(hidden, float("-inf"))
        if sink is None:
            p = torch.softmax(s, -1)
        else:
            top = torch.clamp_min(s.amax(-1, keepdim=True), float(sink[h]))
            e = torch.exp(s - top)
            p = e / (e.sum(-1, keepdim=True) + torch.exp(sink[h] - top))
        out[:, h] = p @ v[:, g]
    return out


def _exact_attention(case, w, prefix, x, held):
    _, heads, kv, dim, _ = SIZES[case["size"]]
    lens, had = _requests(case)
    proj = lambda n, g: (x @ w[f"{prefix}{n}_proj.weight"].double().T + w[f"{prefix}{n}_proj.bias"].double()).view(-1, g, dim)  # noqa: E731
    q, k, v = proj("q", heads), proj("k", kv), proj("v", kv)
    outs, at = [], 0
    for n, h, (kh, vh) in zip(lens, had, held):
        pos = h + torch.arange(n, device=x.device)
        qr, kr = (_rotate(t[at:at + n], pos, dim) for t in (q, k))
        outs.append(_attend(qr, torch.cat((kh.double(), kr)), torch.cat((vh.double(), v[at:at + n])), h, dim ** -0.5))
        at += n
    return torch.cat(outs).flatten(1) @ w[prefix + "o_proj.weight"].double().T


def _exact_mlp(w, x, names):
    g, u, d = (w[n].double() for n in names)
    return (F.silu(x @ g.T) * (x @ u.T)) @ d.T


def _head_rms(o: torch.Tensor) -> torch.Tensor:
    return _rms(o).flatten(1)


def _exact_recurrent(case, w, x):
    H, D, rule = case["heads"], case["dim"], case["rule"]
    w = {n: t.double() for n, t in w.items()}
    lens, _ = _requests(case)
    heads = lambda n: (x @ w[n].T).view(-1, H, D)          # noqa: E731
    g = x @ w["g"].T
    outs, states, at = [], [], 0
    if rule == "gated_delta":
        qkv = [x @ w[n].T for n in "qkv"]
        beta = torch.sigmoid(x @ w["b"].T)
        keep = torch.exp(-torch.exp(w["A_log"]) * F.softplus(x @ w["a"].T + w["dt_bias"], threshold=700.0))
    else:
        q, k, v = heads("q"), heads("k"), heads("v")
        if rule == "mlstm":
            cap = 15.0
            gi = cap * torch.tanh((x @ w["i"].T + w["i.b"]) / cap)
            gf = F.logsigmoid(cap * torch.tanh((x @ w["f"].T + w["f.b"]) / cap))
        elif rule == "gla":
            keep = torch.exp(F.logsigmoid(x @ w["a1"].T @ w["a2"].T + w["a2.b"]) / 16.0).view(-1, H, D, 1)
        else:
            keep = torch.tensor([_retention_decay(h) for h in range(H)], dtype=torch.float64, device=x.device).view(H, 1, 1)
    for n in lens:
        S = torch.zeros(H, D, D, dtype=torch.float64, device=x.device)
        span = slice(at, at + n)
        o = torch.empty(n, H, D, dtype=torch.float64, device=x.device)
        if rule == "gated_delta":
            mixed = []
            for name, t in zip("qkv", qkv):
                pad = F.pad(t[span], (0, 0, 3, 0))
                mixed.append(F.silu(sum(pad[j:j + n] * w[name + ".conv"][:, j] for j in range(4))))
            unit = lambda t: t / torch.sqrt(t.square().sum(-1, keepdim=True) + 1e-6)       # noqa: E731
            qq, kk = (unit(t.view(n, H // 2, D)).repeat_interleave(2, 1) for t in mixed[:2])
            qq, vv, b, a = qq * D ** -0.5, mixed[2].view(n, H, D), beta[span, :, None], keep[span, :, None, None]
            for t in range(n):
                S = a[t] * S
                u = b[t] * (vv[t] - torch.einsum("hij,hi->hj", S, kk[t]))
                S = S + kk[t][:, :, None] * u[:, None, :]
                o[t] = torch.einsum("hij,hi->hj", S, qq[t])
            tail = F.pad(torch.cat(qkv, 1)[span], (0, 0, 3, 0))[-3:].T
            states.append(torch.cat((S.flatten(), tail.flatten())))
        elif rule == "mlstm":
            qq, kk, vv = q[span] * D ** -0.5, k[span], v[span]
            nn, m = torch.zeros(H, D, dtype=torch.float64, device=x.device), torch.zeros(H, dtype=torch.float64, device=x.device)
            for t in range(n):
                fi, ff = gi[at + t], gf[at + t]
                new = torch.maximum(ff + m, fi)
                a, b = torch.exp(ff + m - new), torch.exp(fi - new)
                S = a[:, None, None] * S + (b[:, None] * kk[t])[:, :, None] * vv[t][:, None, :]
                nn = a[:, None] * nn + b[:, None] * kk[t]
                m = new
                den = torch.maximum((nn * qq[t]).sum(-1).abs(), torch.exp(-m)) + 1e-6
                o[t] = torch.einsum("hij,hi->hj", S, qq[t]) / den[:, None]
            states.append(torch.cat((torch.cat((S, nn[:, :, None]), 2).flatten(1), m[:, None]), 1).flatten())
        else:
            qq, kk, vv = q[span], k[span], v[span]
            if rule == "retention":
                pos = torch.arange(n, device=x.device)
                qq, kk = _rotate(qq, pos, D), _rotate(kk, pos, D) * D ** -0.5
            else:
                qq = qq * D ** -0.5
            for t in range(n):
                S = (keep if rule == "retention" else keep[at + t]) * S + kk[t][:, :, None] * vv[t][:, None, :]
                o[t] = torch.einsum("hij,hi->hj", S, qq[t])
            states.append(S.flatten())
        outs.append(o)
        at += n
    y = _head_rms(torch.cat(outs))
    if rule == "mlstm":
        y = y * w["norm"] * torch.sigmoid(g)
    elif rule == "retention":
        y = y * F.silu(g)
    else:
        y = y * w["norm"].repeat(H) * F.silu(g)
    return y @ w["o"].T, torch.stack(states)


def _exact_experts(case, w, x):
    z = x @ w["router"].double().T + w["router.b"].double()
    top, chosen = z.topk(case["top"], -1)
    c = torch.softmax(top, -1)
    out = torch.sigmoid(x @ w["shared.sg"].double().T) * _exact_mlp(w, x, ("shared.gate", "shared.up", "shared.down"))
    for e in range(case["experts"]):
        rows, place = torch.where(chosen == e)
        if len(rows):
            out[rows] += c[rows, place][:, None] * _exact_mlp(w, x[rows], (f"e{e}.gate", f"e{e}.up", f"e{e}.down"))
    return out


def _exact_latent(case, w, x, held):
    H, D, R, C = (case[k] for k in ("heads", "dim", "rot", "kv_rank"))
    w = {n: t.double() for n, t in w.items()}
    _, had = _requests(case)
    q = (_rms(x @ w["dq"].T) * w["dq.norm"] @ w["uq"].T).view(-1, H, D + R)
    down = x @ w["dkv"].T
    c = _rms(down[:, :C]) * w["dkv.norm"]
    gate = torch.sigmoid(x @ w["g"].T)
    uk, uv = w["uk"].view(H, D, C), w["uv"].view(H, D, C)
    outs = []
    for i, (h, (rows, _)) in enumerate(zip(had, held)):
        pos = torch.tensor([h], device=x.device)
        old = rows.double()[:, 0]
        cc, rr = torch.cat((old[:, :C], c[i:i + 1])), torch.cat((old[:, C:], _rotate(down[i:i + 1, None, C:], pos, R, True)[:, 0]))
        ql = torch.einsum("hd,hdc->hc", q[i, :, :D], uk)
        qr = _rotate(q[i:i + 1, :, D:], pos, R, True)[0]
        s = (ql @ cc.T + qr @ rr.T) * (D + R) ** -0.5
        top = torch.maximum(s.amax(-1), w["sink"])[:, None]
        e = torch.exp(s - top)
        p = e / (e.sum(-1, keepdim=True) + torch.exp(w["sink"][:, None] - top))
        outs.append((torch.einsum("hc,hdc->hd", p @ cc, uv) * gate[i][:, None]).flatten())
    return torch.stack(outs) @ w["o"].T


def _exact_step(case, given):
    w, held = given["weights"], given["held"]
    x = w["model.embed_tokens.weight"][given["tokens"]].double()
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        x = x + _exact_attention(case, w, p + "self_attn.", _rms(x) * w[p + "input_layernorm.weight"].double(), held[i])
        h = _rms(x) * w[p + "post_attention_layernorm.weight"].double()
        x = x + _exact_mlp(w, h, (p + "mlp.gate_proj.weight", p + "mlp.up_proj.weight", p + "mlp.down_proj.weight"))
    lens, _ = _requests(case)
    last = torch.tensor(lens, device=x.device).cumsum(0) - 1
    y = _rms(x[last]) * w["model.norm.weight"].double()
    return torch.cat([y @ part.double().T for part in w["lm_head.weight"].split(16384)], 1)


@torch.inference_mode()
def exact(case: dict, seed: int):
    given, kind = _inputs(case, seed), case["kind"]
    if kind == "step":
        return _exact_step(case, given)
    x, w = given["rows"].double(), given["weights"]
    if kind == "attention":
        return _exact_attention(case, w, "", x, given["held"][0])
    if kind == "mlp":
        return _exact_mlp(w, x, ("gate_proj.weight", "up_proj.weight", "down_proj.weight"))
    if kind == "recurrent":
        return _exact_recurrent(case, w, x)
    if kind == "experts":
        return _exact_experts(case, w, x)
    return _exact_latent(case, w, x, given["held"][0])
