"""The work that programs have this engine do, as cases that can be timed and compared.

A case is a dictionary of plain values.  Its ``kind`` says which public entry point a pass goes through:

generate   ``Engine.generate``: prompts in, greedy tokens out (the engine's scheduler, cache, step and sampler)
replay     ``ModelRunner.step`` driven with given token ids: requests are admitted, their prompts go in as far as the
           step's token budget allows, ``new`` further tokens follow one a step, the requests are released; ``new`` 0
           is a prefill.  Output: the logits of every wanted place (each prompt's last token, every further token)
decode     one ``ModelRunner.step`` in which every request, its prompt cached, brings one token; the caches grow by it
mixed      one ``ModelRunner.step`` of continuous batching: live requests bring a token each, new prompts go in beside
           them (and are released after the step)
sample     ``Sampler.sample`` on a step's logits with the command line's options

Models have random weights N(0, 0.02), norm weights 1 + U(-0.1, 0.1) and uniform token ids.  The Qwen3 sizes are
those of the benchmark (0.6B, 8B, 32B), with fewer layers where all of them would only repeat the same work; the two
designs stand for the architectures with scans and with attention over latents, at the benchmark's first size.
"""
from __future__ import annotations

import math
import random
from typing import Dict, List, Sequence, Tuple

import torch

from inferrs_b200 import Engine, SamplingParams
from inferrs_b200.engine.batch import StepEntry
from inferrs_b200.engine.loading import spec_from_config
from inferrs_b200.engine.runner import ModelRunner
from inferrs_b200.runtime import Runtime, parse_dtype
from inferrs_b200.sampling.sampler import Sampler

PAGE = 16
BUDGET = 2048             # the engine's default token budget of a step
L2_BYTES = 126e6          # weights that fit here need not come from memory again for the next step of a pass
EXACT_FLOPS = 4e14        # about ten seconds of 64-bit products

# hidden, heads, key/value heads, head size, feed-forward, layers, vocabulary, rotation base, eps, tied head
QWEN3 = {
    "tiny-a": (64, 4, 2, 16, 128, 2, 256, 1e4, 1e-6, True),
    "tiny-b": (96, 8, 2, 32, 256, 3, 512, 1e6, 1e-5, False),
    "0.6b": (1024, 16, 8, 128, 3072, 28, 151936, 1e6, 1e-6, True),
    "8b": (4096, 32, 8, 128, 12288, 36, 151936, 1e6, 1e-6, False),
    "32b": (5120, 64, 8, 128, 25600, 64, 151936, 1e6, 1e-6, False),
}
# width, heads, feed-forward, query rank, latent, vocabulary, window
DESIGNS = {"vebonex": (2048, 16, 8192, 768, 512, 32000, 0), "dasusun": (2048, 16, 8192, 768, 512, 32000, 1024)}


def listed() -> List[dict]:
    return [
        # the smallest calls: a toy model through the whole engine in true 32-bit; nothing but launches and host work
        dict(name="generate tiny f32", kind="generate", model="tiny-a", layers=2, dtype="f32", requests=3, shortest=5,
             longest=33, new=16),
        # the 32-bit path in earnest use: checking a small checkpoint's logits, prompts and a few decoded tokens
        dict(name="replay 0.6b f32", kind="replay", model="0.6b", layers=28, dtype="f32", requests=4, shortest=33,
             longest=200, new=8, budget=BUDGET),
        # one chat on a small model: a decoded token's latency
        dict(name="decode 0.6b b1", kind="decode", model="0.6b", layers=28, dtype="bf16", requests=1, shortest=1500,
             longest=1500),
        # the benchmark's headline: a decode step of eight requests with 2,048 tokens each
        dict(name="decode 8b b8", kind="decode", model="8b", layers=8, dtype="bf16", requests=8, shortest=2048,
             longest=2048),
        # a busy server's decode step: 64 requests of every age
        dict(name="decode 8b b64", kind="decode", model="8b", layers=8, dtype="bf16", requests=64, shortest=128,
             longest=2048),
        # time to first token of a short question on a small model
        dict(name="prompt 0.6b 137", kind="replay", model="0.6b", layers=28, dtype="bf16", requests=1, shortest=137,
             longest=137, new=0, budget=BUDGET),
        # the benchmark's prefill: one 2,048-token prompt in one step
        dict(name="prompt 8b 2048", kind="replay", model="8b", layers=8, dtype="bf16", requests=1, shortest=2048,
             longest=2048, new=0, budget=BUDGET),
        # a long document on a large model, in portions of 2,048 tokens
        dict(name="prompt 32b 8192", kind="replay", model="32b", layers=6, dtype="bf16", requests=1, shortest=8192,
             longest=8192, new=0, budget=BUDGET),
        # continuous batching: 96 requests decode while new prompts of any length fill the step
        dict(name="mixed 0.6b", kind="mixed", model="0.6b", layers=28, dtype="bf16", requests=96, shortest=64,
             longest=1024, prompts=5, prompt_shortest=101, prompt_longest=700),
        # the command line's default sampling for a batch of 64 over the whole vocabulary
        dict(name="sample b64", kind="sample", vocab=151936, rows=64, temperature=0.7, top_k=50, top_p=0.9,
             repetition_penalty=1.1),
        # prompts and decoded tokens of the design with scans of a matrix state and attention over latents
        dict(name="replay vebonex", kind="replay", model="vebonex", layers=4, dtype="bf16", requests=4, shortest=100,
             longest=900, new=16, budget=BUDGET),
        # ... and of the design with latent attention with a rotated part and windows
        dict(name="replay dasusun", kind="replay", model="dasusun", layers=4, dtype="bf16", requests=4, shortest=200,
             longest=1300, new=16, budget=BUDGET),
    ]


def draw(rng: random.Random) -> dict:
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def spread(lo, hi):
        a, b = log(lo, hi), log(lo, hi)
        return dict(shortest=min(a, b), longest=max(a, b))

    kind = rng.choice(["generate", "f32", "decode", "decode", "decode", "prompt", "prompt", "mixed", "sample", "design"])
    if kind == "generate":
        model = rng.choice(["tiny-a", "tiny-b"])
        return dict(kind=kind, model=model, layers=QWEN3[model][5], dtype="f32", requests=log(1, 8),
                    **spread(2, 90), new=rng.randint(4, 24))
    if kind == "f32":
        return dict(kind="replay", model="0.6b", layers=rng.randint(4, 28), dtype="f32", requests=log(1, 6),
                    **spread(8, 250), new=rng.randint(0, 10), budget=rng.choice([64, 256, BUDGET]))
    if kind == "decode":
        model = rng.choice(["0.6b", "8b", "32b"])
        layers = {"0.6b": 28, "8b": rng.randint(3, 8), "32b": rng.randint(2, 6)}[model]
        return dict(kind=kind, model=model, layers=layers, dtype="bf16", requests=log(1, 64), **spread(32, 2048))
    if kind == "prompt":
        model = rng.choice(["0.6b", "8b", "32b"])
        layers = {"0.6b": 28, "8b": rng.randint(3, 8), "32b": rng.randint(2, 6)}[model]
        return dict(kind="replay", model=model, layers=layers, dtype="bf16", requests=rng.choice([1, 1, 2, 5]),
                    **spread(20, 1600), new=0, budget=rng.choice([512, BUDGET]))
    if kind == "mixed":
        a, b = log(30, 300), log(30, 300)
        return dict(kind=kind, model="0.6b", layers=28, dtype="bf16", requests=log(4, 128), **spread(32, 1024),
                    prompts=rng.randint(1, 6), prompt_shortest=min(a, b), prompt_longest=max(a, b))
    if kind == "sample":
        return dict(kind=kind, vocab=rng.choice([32000, 151936]), rows=log(1, 128), temperature=rng.uniform(0.3, 1.5),
                    top_k=rng.choice([0, log(2, 400)]), top_p=rng.choice([1.0, rng.uniform(0.5, 0.99)]),
                    repetition_penalty=rng.choice([1.0, 1.1]))
    return dict(kind="replay", model=rng.choice(sorted(DESIGNS)), layers=4, dtype="bf16", requests=log(1, 6),
                **spread(50, 1500), new=rng.randint(1, 24), budget=rng.choice([512, BUDGET]))


# ---- a model's configuration and tensors ------------------------------------------------------------------------
def config_of(case: dict, positions: int) -> dict:
    n = case["layers"]
    if case["model"] in QWEN3:
        H, nh, nkv, d, ff, _, vocab, theta, eps, tied = QWEN3[case["model"]]
        return {"architectures": ["Qwen3ForCausalLM"], "model_type": "qwen3", "num_hidden_layers": n, "hidden_size": H,
                "num_attention_heads": nh, "num_key_value_heads": nkv, "head_dim": d, "intermediate_size": ff,
                "vocab_size": vocab, "rope_theta": theta, "rms_norm_eps": eps, "max_position_embeddings": positions,
                "tie_word_embeddings": tied, "hidden_act": "silu"}
    W, heads, ff, q_rank, rank, vocab, window = DESIGNS[case["model"]]
    mlp = {"kind": "dense", "ff": ff}
    layers = []
    for i in range(n):
        if case["model"] == "dasusun":
            m = {"heads": heads, "dim": 128, "rot_dim": 64, "vdim": 128, "q_rank": q_rank, "kv_rank": rank,
                 "scale": 192 ** -0.5, "rot": {"base": 1e6, "dims": 64}}
            if i % 4 != 3:
                m["mask"] = {"size": window}
            layers.append({"type": "latent_attention", "mixer": m, "mlp": mlp})
        elif i % 4 == 0:
            layers.append({"type": "mlstm", "mixer": {"heads": heads, "dim": 128, "vdim": 128, "gate_cap": 15.0}, "mlp": mlp})
        elif i % 4 == 1:
            layers.append({"type": "gla", "mlp": mlp,
                           "mixer": {"heads": heads, "dim": 128, "vdim": 128, "tau": 16.0, "a_rank": 16}})
        else:
            m = {"heads": heads, "dim": 128, "vdim": 128, "q_rank": q_rank, "kv_rank": rank, "scale": 128 ** -0.5}
            layers.append({"type": "latent_attention", "mlp": mlp, "mixer": dict(m, kv_from=i - 1) if i % 4 == 3 else m})
    out = {"vocab": vocab, "width": W, "max_positions": positions, "norm": {"eps": 1e-5}, "layers": layers}
    if case["model"] == "dasusun":
        return dict(out, architecture="Dasusun", canon={"taps": 3})
    return dict(out, architecture="Vebonex", streams=2, norm={"eps": 1e-5, "groups": 4})


#: (name, shape, (kind, centre, spread))
Tensors = List[Tuple[str, Tuple[int, ...], Tuple[str, float, float]]]
NORMAL, NORM, ZERO = ("normal", 0.0, 0.02), ("uniform", 1.0, 0.1), ("uniform", 0.0, 0.1)


def tensors_of(cfg: dict) -> Tensors:
    if "hidden_size" in cfg:
        H, I, V = cfg["hidden_size"], cfg["intermediate_size"], cfg["vocab_size"]
        nh, nkv, d = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"]
        out = [("model.embed_tokens.weight", (V, H), NORMAL), ("model.norm.weight", (H,), NORM)]
        if not cfg["tie_word_embeddings"]:
            out.append(("lm_head.weight", (V, H), NORMAL))
        for i in range(cfg["num_hidden_layers"]):
            a, m = f"model.layers.{i}.self_attn", f"model.layers.{i}.mlp"
            out += [(f"model.layers.{i}.input_layernorm.weight", (H,), NORM),
                    (f"model.layers.{i}.post_attention_layernorm.weight", (H,), NORM),
                    (f"{a}.q_proj.weight", (nh * d, H), NORMAL), (f"{a}.k_proj.weight", (nkv * d, H), NORMAL),
                    (f"{a}.v_proj.weight", (nkv * d, H), NORMAL), (f"{a}.o_proj.weight", (H, nh * d), NORMAL),
                    (f"{a}.q_norm.weight", (d,), NORM), (f"{a}.k_norm.weight", (d,), NORM),
                    (f"{m}.gate_proj.weight", (I, H), NORMAL), (f"{m}.up_proj.weight", (I, H), NORMAL),
                    (f"{m}.down_proj.weight", (H, I), NORMAL)]
        return out
    W, V = cfg["width"], cfg["vocab"]
    dasusun = cfg["architecture"] == "Dasusun"
    norm = ZERO if dasusun else NORM
    out = [("embed", (V, W), NORMAL), ("final.norm", (W,), norm)]
    if not dasusun:
        out += [("pos", (cfg["max_positions"], W), NORMAL), ("head", (V, W), NORMAL)]
    for i, layer in enumerate(cfg["layers"]):
        m, p, ff = layer["mixer"], f"l{i}.mix", layer["mlp"]["ff"]
        h, D, E = m["heads"], m["dim"], m["vdim"]
        out += [(f"l{i}.norm1", (W,), norm), (f"l{i}.norm2", (W,), norm), (f"l{i}.mlp.up", (ff, W), NORMAL),
                (f"l{i}.mlp.down", (W, ff), NORMAL), (f"{p}.o", (W, h * E), NORMAL)]
        if layer["type"] == "latent_attention":
            rot = m.get("rot_dim", 0)
            out += [(f"{p}.dq", (m["q_rank"], W), NORMAL), (f"{p}.dq.norm", (m["q_rank"],), NORM),
                    (f"{p}.uq", (h * (D + rot), m["q_rank"]), NORMAL), (f"{p}.uk", (h * D, m["kv_rank"]), NORMAL),
                    (f"{p}.uv", (h * E, m["kv_rank"]), NORMAL)]
            if "kv_from" not in m:
                out += [(f"{p}.dkv", (m["kv_rank"] + rot, W), NORMAL), (f"{p}.dkv.norm", (m["kv_rank"],), NORM)]
        else:
            out += [(f"{p}.q", (h * D, W), NORMAL), (f"{p}.k", (h * D, W), NORMAL), (f"{p}.v", (h * E, W), NORMAL)]
            if layer["type"] == "mlstm":
                out += [(f"{p}.norm", (h * E,), NORM), (f"{p}.i", (h, W), NORMAL), (f"{p}.f", (h, W), NORMAL),
                        (f"{p}.i.b", (h,), ("uniform", 0.0, 1.0)), (f"{p}.f.b", (h,), ("uniform", 3.0, 2.0))]
            else:
                out += [(f"{p}.norm", (E,), NORM), (f"{p}.a1", (m["a_rank"], W), NORMAL),
                        (f"{p}.a2", (h * D, m["a_rank"]), NORMAL), (f"{p}.a2.b", (h * D,), ("uniform", 3.0, 2.0))]
        if dasusun:
            out += [(f"l{i}.norm1b", (W,), ZERO), (f"l{i}.norm2b", (W,), ZERO), (f"l{i}.ls1", (W,), ("uniform", 1.0, 0.3)),
                    (f"l{i}.ls2", (W,), ("uniform", 1.0, 0.3)), (f"l{i}.canon1", (W, 3), ("uniform", 0.0, 0.3)),
                    (f"l{i}.dwa", (i + 2,), ("uniform", 1.0 / (i + 2), 0.5 / (i + 2)))]
        else:
            out += [(f"{p}.g", (h * E, W), NORMAL), (f"l{i}.mlp.act", (4,), ("uniform", 0.4, 0.3))]
            for hc in (f"l{i}.hc1", f"l{i}.hc2"):
                out += [(f"{hc}.in", (2,), ("uniform", 0.5, 0.1)), (f"{hc}.out", (2,), ("uniform", 1.0, 0.2)),
                        (f"{hc}.mix", (2, 2), ("identity", 0.0, 0.1))]
    return out


def weights_of(cfg: dict, dtype: torch.dtype, seed: int) -> Dict[str, torch.Tensor]:
    g = torch.Generator(device="cuda").manual_seed(seed)
    out = {}
    for name, shape, (kind, centre, spread) in tensors_of(cfg):
        t = torch.empty(shape, dtype=dtype, device="cuda")
        if kind == "normal":
            t.normal_(centre, spread, generator=g)
        else:
            t.uniform_(centre - spread, centre + spread, generator=g)
            if kind == "identity":
                t += torch.eye(shape[0], dtype=dtype, device="cuda")
        out[name] = t
    return out


# ---- requests ---------------------------------------------------------------------------------------------------
def lengths(n: int, shortest: int, longest: int) -> List[int]:
    """``n`` lengths spread evenly over the logarithm, the longest first."""
    if n == 1:
        return [longest]
    return [int(round(longest * (shortest / longest) ** (i / (n - 1)))) for i in range(n)]


def tokens_of(case: dict, seed: int) -> Tuple[List[List[int]], List[List[int]]]:
    """(token ids of every request that the case names, of its new prompts): for ``replay`` prompt and further tokens,
    for ``decode`` and ``mixed`` prompt and the token that a pass brings."""
    vocab = (QWEN3[case["model"]][6] if case["model"] in QWEN3 else DESIGNS[case["model"]][5])
    rng = random.Random(seed)
    more = case["new"] if case["kind"] in ("replay", "generate") else 1
    own = [rng.choices(range(vocab), k=n + more) for n in lengths(case["requests"], case["shortest"], case["longest"])]
    if case["kind"] != "mixed":
        return own, []
    return own, [rng.choices(range(vocab), k=n)
                 for n in lengths(case["prompts"], case["prompt_shortest"], case["prompt_longest"])]


def trace_of(rids: Sequence, tokens: List[List[int]], new: int, budget: int) -> List[List[StepEntry]]:
    """The steps that take every request from nothing to its last token: requests past their prompts bring one token,
    the others as much of their prompts as the step's budget still holds."""
    at, steps = [0] * len(tokens), []
    while any(a < len(t) for a, t in zip(at, tokens)):
        left, entries = budget, []
        order = sorted(range(len(tokens)), key=lambda i: at[i] < len(tokens[i]) - new)     # decoding requests first
        for i in order:
            prompt = len(tokens[i]) - new
            n = min(prompt - at[i], left) if at[i] < prompt else min(1, len(tokens[i]) - at[i])
            if n > 0:
                at[i] += n
                left -= n
                entries.append(StepEntry(rids[i], tokens[i][at[i] - n:at[i]], [n - 1] if at[i] >= prompt else []))
        steps.append(entries)
    return steps


# ---- the passes -------------------------------------------------------------------------------------------------
class _State:
    pass


def prepare(case: dict, seed: int):
    s = _State()
    s.case = case
    if case["kind"] == "sample":
        g = torch.Generator(device="cuda").manual_seed(seed)
        rng = random.Random(seed)
        s.logits = torch.randn((case["rows"], case["vocab"]), generator=g, device="cuda").mul_(1.5)
        s.params = [SamplingParams(temperature=case["temperature"], top_k=case["top_k"], top_p=case["top_p"],
                                   repetition_penalty=case["repetition_penalty"])] * case["rows"]
        s.seeds = [rng.getrandbits(63) for _ in range(case["rows"])]
        s.histories = [rng.choices(range(case["vocab"]), k=rng.randint(30, 400)) for _ in range(case["rows"])]
        s.sampler = Sampler(s.logits.device, torch.bfloat16)
        return s
    own, prompts = tokens_of(case, seed)
    if case["kind"] == "generate":
        s.prompts = [t[:len(t) - case["new"]] for t in own]
        s.engine = Engine(config=config_of(case, 128), random_weights=seed, dtype=case["dtype"], block_size=PAGE,
                          num_blocks=8 * case["requests"], max_batch_size=case["requests"])
        s.engine.warm_up()
        s.sampling = SamplingParams.greedy(max_tokens=case["new"], ignore_eos=True)
        return s
    live = case["requests"] + case.get("prompts", 0)
    room = max(len(t) for t in own + prompts)
    # a decoding request may grow by 2,048 tokens before its state starts again from its prompt
    s.limit = (room + (2048 if case["kind"] != "replay" else 0) + PAGE) // PAGE * PAGE
    cfg = config_of(case, s.limit)
    rt = Runtime.cuda(parse_dtype(case["dtype"]))
    spec, _ = spec_from_config(cfg)
    n_pages = live * (s.limit // PAGE)
    s.runner = ModelRunner(spec, weights_of(cfg, rt.dtype, seed), rt, page_size=PAGE, n_pages=n_pages,
                           max_requests=live, max_context=s.limit, consume_weights=True)
    if case["kind"] == "replay":
        s.rids = list(range(case["requests"]))
        s.steps = trace_of(s.rids, own, case["new"], case["budget"])
        for entries in s.steps:                 # a serving program's graphs are captured before its first request
            for e in entries:
                if not s.runner.has(e.rid):
                    s.runner.admit(e.rid)
            s.runner.step([StepEntry(e.rid, [0] * len(e.tokens), e.want) for e in entries], own_output=False)
        for rid in s.rids:
            s.runner.release(rid)
        return s
    s.rids = list(range(case["requests"]))
    s.fill = trace_of(s.rids, [t[:-1] for t in own], 0, BUDGET)
    s.entries = [StepEntry(rid, t[-1:], [0]) for rid, t in zip(s.rids, own)]
    s.new_rids = [("new", i) for i in range(len(prompts))]
    s.entries += [StepEntry(rid, t, [len(t) - 1]) for rid, t in zip(s.new_rids, prompts)]
    if case["kind"] == "decode":
        s.runner.warm_up([case["requests"]])
    else:
        for e in s.entries:
            s.runner.admit(e.rid)
        s.runner.step(s.entries, own_output=False)
        for e in s.entries:
            s.runner.release(e.rid)
    fill(s)
    return s


def fill(s) -> None:
    """Bring the decoding requests' prompts into the cache."""
    for rid in s.rids:
        if s.runner.has(rid):
            s.runner.release(rid)
        s.runner.admit(rid)
    for entries in s.fill:
        s.runner.step([StepEntry(e.rid, e.tokens) for e in entries], own_output=False)


def run(s):
    kind = s.case["kind"]
    if kind == "generate":
        return [torch.tensor(t) for t in s.engine.generate(s.prompts, s.sampling)]
    if kind == "sample":
        logits = s.logits.clone()               # the penalties work in place, as on a step's own logits
        tokens = s.sampler.sample(logits, s.params, s.seeds, s.histories)
        return {"logits": logits, "tokens": tokens}
    if kind == "replay":
        for rid in s.rids:
            s.runner.admit(rid)
        out = [s.runner.step(entries) for entries in s.steps]
        for rid in s.rids:
            s.runner.release(rid)
        return out
    if s.runner.n_tokens(s.rids[0]) >= s.limit:
        fill(s)
    for rid in s.new_rids:
        s.runner.admit(rid)
    logits = s.runner.step(s.entries, own_output=False)
    for rid in s.new_rids:
        s.runner.release(rid)
    return logits


# ---- what a pass cannot do without ------------------------------------------------------------------------------
def steps_of(case: dict) -> List[List[Tuple[int, int, int]]]:
    """Every step of a pass as (tokens cached before, new tokens, wanted places) of its requests."""
    if case["kind"] in ("replay", "generate"):
        n = lengths(case["requests"], case["shortest"], case["longest"])
        at = [0] * len(n)
        # the last token that ``generate`` returns is not fed back
        new = case["new"] - (case["kind"] == "generate")
        steps = trace_of(range(len(n)), [[0] * (x + new) for x in n], new, case.get("budget", BUDGET))
        out = []
        for entries in steps:
            out.append([(at[e.rid], len(e.tokens), len(e.want)) for e in entries])
            for e in entries:
                at[e.rid] += len(e.tokens)
        return out
    step = [(n, 1, 1) for n in lengths(case["requests"], case["shortest"], case["longest"])]
    if case["kind"] == "mixed":
        step += [(0, n, 1) for n in lengths(case["prompts"], case["prompt_shortest"], case["prompt_longest"])]
    return [step]


def pairs(before: int, new: int, window: int = 0) -> int:
    """(query, key) pairs of ``new`` tokens behind ``before`` cached ones."""
    if not window:
        return new * before + new * (new + 1) // 2
    return sum(min(before + i + 1, window) for i in range(new))


def work(case: dict) -> dict:
    if case["kind"] == "sample":
        return {"bytes": 4 * case["rows"] * case["vocab"] * 2 + 4 * case["rows"], "flops": 4 * case["rows"] * case["vocab"]}
    cfg = config_of(case, 4096)
    size = 4 if case["dtype"] == "f32" else 2
    shapes = {name: shape for name, shape, _ in tensors_of(cfg)}
    tables = ("model.embed_tokens.weight", "lm_head.weight", "embed", "head", "pos")
    head = next(shapes[n] for n in ("lm_head.weight", "head", "model.embed_tokens.weight", "embed") if n in shapes)
    matrices = sum(math.prod(s) for n, s in shapes.items() if n not in tables)
    products = sum(math.prod(s) for n, s in shapes.items() if n not in tables and len(s) == 2 and min(s) > 4)
    # per layer: numbers cached per token, flops per (query, key) pair, window, flops per token of a scan
    layers = []
    if "hidden_size" in cfg:
        nh, nkv, d = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"]
        layers = [(2 * nkv * d, 4 * nh * d, 0, 0)] * cfg["num_hidden_layers"]
    for layer in cfg.get("layers", ()):
        m = layer["mixer"]
        if layer["type"] == "latent_attention":
            rot = m.get("rot_dim", 0)
            layers.append((m["kv_rank"] + rot if "kv_from" not in m else 0, 2 * m["heads"] * (m["dim"] + rot + m["vdim"]),
                           m.get("mask", {}).get("size", 0), 0))
        else:
            layers.append((0, 0, 0, 6 * m["heads"] * m["dim"] * m["vdim"]))
    bytes_, flops = 0.0, 0.0
    for i, step in enumerate(steps_of(case)):
        rows, wanted = sum(n for _, n, _ in step), sum(w for _, _, w in step)
        weights = size * (matrices + (math.prod(head) if wanted else 0))
        if i == 0 or weights > L2_BYTES:
            bytes_ += weights
        bytes_ += size * rows * head[1] + 4 * wanted * head[0]
        flops += 2.0 * rows * products + 2.0 * wanted * math.prod(head)
        for cached, per_pair, window, scan in layers:
            seen = sum(min(b, window) if window else b for b, _, _ in step)
            bytes_ += size * cached * (seen + rows)
            flops += per_pair * sum(pairs(b, n, window) for b, n, _ in step) + scan * rows
    return {"bytes": bytes_, "flops": flops}


def tolerance(case: dict):
    """Tokens are compared as they are.  32-bit logits: four times what a pass is off from 64 bits (2e-6).  bfloat16: every
    sub-layer's inputs and outputs are rounded to eight bits, and in another order of sums they are rounded to other
    neighbours; a prompt in portions of 96 tokens against the same prompt at once differs by 0.005 (0.6b, 28 layers),
    0.004 (the designs, 4 layers), 0.017 (8b, 8 layers) and 0.016 (32b, 6 layers), single logits by up to 0.09 of their
    root mean square."""
    if case["kind"] in ("generate", "sample"):
        return "exact"
    if case["dtype"] == "f32":
        return {"rel": 1e-5, "max": 1e-4}
    return {"rel": 0.03, "max": 0.35} if case["model"] in ("8b", "32b") else {"rel": 0.02, "max": 0.1}


# ---- the same in 64 bits, in plain torch ------------------------------------------------------------------------
def exact(case: dict, seed: int):
    if case["kind"] == "generate":
        return None
    if case["kind"] == "sample":
        s = prepare(case, seed)
        logits = s.logits.double()
        if case["repetition_penalty"] != 1.0:
            p = torch.tensor(case["repetition_penalty"], dtype=torch.float32).double().item()
            for row, history in zip(logits, s.histories):
                seen = torch.tensor(sorted(set(history[-s.params[0].repeat_last_n:])), device=row.device)
                v = row[seen]
                row[seen] = torch.where(v >= 0, v / p, v * p)
        return {"logits": logits, "tokens": None}
    own, prompts = tokens_of(case, seed)
    seqs = own + prompts
    rids = list(range(len(seqs)))
    if case["kind"] == "replay":
        steps = trace_of(rids, own, case["new"], case["budget"])
    else:
        steps = [[StepEntry(i, t[-1:] if i < len(own) else t, [0 if i < len(own) else len(t) - 1])
                  for i, t in enumerate(seqs)]]
    limit = (max(len(t) for t in seqs) + (2048 if case["kind"] != "replay" else 0) + PAGE) // PAGE * PAGE
    cfg = config_of(case, limit)
    n_weights = sum(math.prod(s) for n, s, _ in tensors_of(cfg) if len(s) == 2)
    if 2.0 * n_weights * sum(len(t) for t in seqs) > EXACT_FLOPS:
        return None
    w = weights_of(cfg, parse_dtype(case["dtype"]), seed)
    at = [len(t) - 1 if case["kind"] != "replay" and i < len(own) else 0 for i, t in enumerate(seqs)]
    places = []                                     # (step, request, position) in the order of the outputs
    for k, entries in enumerate(steps):
        for e in entries:
            places += [(k, e.rid, at[e.rid] + p) for p in e.want]
            at[e.rid] += len(e.tokens)
    stack = _qwen3 if "hidden_size" in cfg else (_dasusun if cfg["architecture"] == "Dasusun" else _vebonex)
    with torch.no_grad():
        ids = [torch.tensor(t, device="cuda") for t in seqs]
        hidden, head = stack(cfg, w, ids)
        rows = [hidden[r][p] for _, r, p in places]
        logits = torch.stack(rows) @ head.double().T if rows else None
    out, taken = [], 0
    for k in range(len(steps)):
        n = sum(1 for step, _, _ in places if step == k)
        out.append(logits[taken:taken + n] if n else torch.zeros((0, head.shape[0]), dtype=torch.float64, device="cuda"))
        taken += n
    return out if case["kind"] == "replay" else out[0]


def _rms(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _rotate(x, base, dims):
    """x [tokens, heads, size]: number i of a head turns with number i + dims / 2."""
    f = base ** (-torch.arange(dims // 2, dtype=torch.float64, device=x.device) * 2.0 / dims)
    a = torch.arange(x.shape[0], dtype=torch.float64, device=x.device)[:, None, None] * f
    u, v = x[..., :dims // 2], x[..., dims // 2:dims]
    return torch.cat([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin(), x[..., dims:]], -1)


def _attend(q, k, v, scale, window=0):
    """q, k [tokens, heads, size], v [tokens, heads, value size]; a head at a time."""
    T = q.shape[0]
    i = torch.arange(T, device=q.device)
    hide = i[None, :] > i[:, None]
    if window:
        hide |= i[None, :] <= i[:, None] - window
    out = [torch.softmax((q[:, h] @ k[:, h].T * scale).masked_fill(hide, -math.inf), -1) @ v[:, h] for h in range(q.shape[1])]
    return torch.stack(out, 1).reshape(T, -1)


def _qwen3(cfg, w, ids):
    nh, nkv, d, eps = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"], cfg["rms_norm_eps"]
    xs = [w["model.embed_tokens.weight"][t].double() for t in ids]
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        m = {k[len(p):-len(".weight")]: t.double() for k, t in w.items() if k.startswith(p)}
        for r, x in enumerate(xs):
            T = x.shape[0]
            h = _rms(x, eps) * m["input_layernorm"]
            q = _rms((h @ m["self_attn.q_proj"].T).view(T, nh, d), eps) * m["self_attn.q_norm"]
            k = _rms((h @ m["self_attn.k_proj"].T).view(T, nkv, d), eps) * m["self_attn.k_norm"]
            v = (h @ m["self_attn.v_proj"].T).view(T, nkv, d).repeat_interleave(nh // nkv, 1)
            q = _rotate(q, cfg["rope_theta"], d)
            k = _rotate(k, cfg["rope_theta"], d).repeat_interleave(nh // nkv, 1)
            x = x + _attend(q, k, v, d ** -0.5) @ m["self_attn.o_proj"].T
            h = _rms(x, eps) * m["post_attention_layernorm"]
            g = h @ m["mlp.gate_proj"].T
            xs[r] = x + (torch.nn.functional.silu(g) * (h @ m["mlp.up_proj"].T)) @ m["mlp.down_proj"].T
    head = w.get("lm_head.weight", w["model.embed_tokens.weight"])
    return [_rms(x, eps) * w["model.norm.weight"].double() for x in xs], head


def _dasusun(cfg, w, ids):
    eps = cfg["norm"]["eps"]
    w = {k: t.double() if k != "embed" else t for k, t in w.items()}
    out = []
    for t in ids:
        x = w["embed"][t].double()
        T, results = x.shape[0], [x]
        for i, layer in enumerate(cfg["layers"]):
            m, p = layer["mixer"], f"l{i}.mix."
            h = _rms(x, eps) * (1 + w[f"l{i}.norm1"])
            taps = w[f"l{i}.canon1"]
            n = taps.shape[1]
            back = torch.nn.functional.pad(h, (0, 0, n - 1, 0))
            h = h + sum(back[j:j + T] * taps[:, j] for j in range(n))
            H, D, P, R = m["heads"], m["dim"], m["rot_dim"], m["kv_rank"]
            q = ((_rms(h @ w[p + "dq"].T, eps) * w[p + "dq.norm"]) @ w[p + "uq"].T).view(T, H, D + P)
            down = h @ w[p + "dkv"].T
            c = _rms(down[:, :R], eps) * w[p + "dkv.norm"]
            turned = _rotate(down[:, None, R:], m["rot"]["base"], P).expand(T, H, P)
            q = torch.cat([q[..., :D], _rotate(q[..., D:], m["rot"]["base"], P)], -1)
            k = torch.cat([(c @ w[p + "uk"].T).view(T, H, D), turned], -1)
            v = (c @ w[p + "uv"].T).view(T, H, m["vdim"])
            y = _attend(q, k, v, m["scale"], m.get("mask", {}).get("size", 0)) @ w[p + "o"].T
            x = x + _rms(y, eps) * (1 + w[f"l{i}.norm1b"]) * w[f"l{i}.ls1"]
            h = _rms(x, eps) * (1 + w[f"l{i}.norm2"])
            y = torch.nn.functional.gelu(h @ w[f"l{i}.mlp.up"].T, approximate="tanh") @ w[f"l{i}.mlp.down"].T
            x = x + _rms(y, eps) * (1 + w[f"l{i}.norm2b"]) * w[f"l{i}.ls2"]
            results.append(x)
            x = sum(a * r for a, r in zip(w[f"l{i}.dwa"], results))
        out.append(_rms(x, eps) * (1 + w["final.norm"]))
    return out, w["embed"]


def _scan(q, k, v, keep, take):
    """S_t = keep_t S_(t-1) + take_t k_t v_t^T and S_t^T q_t for every t; keep [tokens, heads, key size]."""
    S = torch.zeros((q.shape[1], q.shape[2], v.shape[2]), dtype=q.dtype, device=q.device)
    out = []
    for t in range(q.shape[0]):
        S = torch.baddbmm(keep[t][:, :, None] * S, (take[t][:, None] * k[t])[:, :, None], v[t][:, None, :])
        out.append(torch.bmm(q[t][:, None], S)[:, 0])
    return torch.stack(out)


def _vebonex(cfg, w, ids):
    eps, groups = cfg["norm"]["eps"], cfg["norm"]["groups"]
    w = {k: t.double() if k not in ("embed", "head") else t for k, t in w.items()}

    def norm(x, weight):
        return _rms(x.view(x.shape[0], groups, -1), eps).view(x.shape) * weight

    def mixer(h, i, latents):
        layer, p = cfg["layers"][i], f"l{i}.mix."
        m, T = layer["mixer"], h.shape[0]
        H, D, E = m["heads"], m["dim"], m["vdim"]
        gate = h @ w[p + "g"].T
        if layer["type"] == "latent_attention":
            if "kv_from" not in m:
                latents[i] = _rms(h @ w[p + "dkv"].T, eps) * w[p + "dkv.norm"]
            c = latents[m.get("kv_from", i)]
            q = (_rms(h @ w[p + "dq"].T, eps) * w[p + "dq.norm"]) @ w[p + "uq"].T
            y = _attend(q.view(T, H, D), (c @ w[p + "uk"].T).view(T, H, D), (c @ w[p + "uv"].T).view(T, H, E), m["scale"])
            return (y * torch.sigmoid(gate)) @ w[p + "o"].T
        q = (h @ w[p + "q"].T).view(T, H, D) * D ** -0.5
        k, v = (h @ w[p + "k"].T).view(T, H, D), (h @ w[p + "v"].T).view(T, H, E)
        if layer["type"] == "gla":
            z = (h @ w[p + "a1"].T) @ w[p + "a2"].T + w[p + "a2.b"]
            y = _scan(q, k, v, torch.sigmoid(z).pow(1.0 / m["tau"]).view(T, H, D), torch.ones_like(q[..., 0]))
            y = (_rms(y, eps) * w[p + "norm"]).reshape(T, -1) * torch.nn.functional.silu(gate)
            return y @ w[p + "o"].T
        cap = m["gate_cap"]
        log_i = cap * torch.tanh((h @ w[p + "i"].T + w[p + "i.b"]) / cap)
        log_f = torch.nn.functional.logsigmoid(cap * torch.tanh((h @ w[p + "f"].T + w[p + "f.b"]) / cap))
        peak, top = torch.zeros_like(log_i[0]), []
        for t in range(T):
            peak = torch.maximum(log_f[t] + peak, log_i[t])
            top.append(peak)
        top = torch.stack(top)
        keep = torch.exp(log_f + torch.cat([torch.zeros_like(top[:1]), top[:-1]]) - top)
        take = torch.exp(log_i - top)
        # the sum of the keys beside the matrix: one more value, always one
        y = _scan(q, k, torch.cat([v, torch.ones_like(v[..., :1])], -1), keep[..., None].expand_as(q), take)
        y = y[..., :E] / (torch.maximum(y[..., E:].abs(), torch.exp(-top)[..., None]) + 1e-6)
        return ((_rms(y, eps).reshape(T, -1) * w[p + "norm"]) * torch.sigmoid(gate)) @ w[p + "o"].T

    def feed_forward(h, i):
        z, a = h @ w[f"l{i}.mlp.up"].T, w[f"l{i}.mlp.act"]
        return (a[0] * _rms(z, eps) + a[1] * _rms(z * z, eps) + a[2] * _rms(z * z * z, eps) + a[3]) @ w[f"l{i}.mlp.down"].T

    out = []
    for t in ids:
        x = w["embed"][t].double() + w["pos"][:t.shape[0]]
        streams, latents = [x, x], {}
        for i in range(len(cfg["layers"])):
            for sub in (1, 2):
                into, back, mix = (w[f"l{i}.hc{sub}.{n}"] for n in ("in", "out", "mix"))
                h = norm(into[0] * streams[0] + into[1] * streams[1], w[f"l{i}.norm{sub}"])
                y = mixer(h, i, latents) if sub == 1 else feed_forward(h, i)
                streams = [mix[0, j] * streams[0] + mix[1, j] * streams[1] + back[j] * y for j in (0, 1)]
        out.append(norm(streams[0] + streams[1], w["final.norm"]))
    return out, w["head"]
