"""The work this engine is measured by, as a program that serves models calls it.

Three ways of use:

* ``score``: prompts go through `Engine.step` in portions, the logits at a few wanted places come back (ranking, perplexity,
  the first token of an answer);
* ``decode``: the loop under `LLM`: one step over the prompts, captured decode steps chained on the device, the ids read, and one
  step of single tokens launched kernel by kernel whose logits come back (what a program reads that wants the distribution
  behind an answer), from the pages and states which the captured steps wrote;
* ``generate``: `LLM.generate`, scheduler and sampler included.

Seven architectures: the sizes of Qwen2.5-0.5B and 7B as ``bench.py`` has them, and the six other designs at the two widths of its
side-by-side workloads.  Weights are drawn, and drawn so that a pass says something: the embedding stays visible in the stream
and the head answers token t with token t + 4099 (a tied head with token t itself) by a wide margin, as a trained model is sure
of most of its tokens; a token's embedding leans towards two experts, as trained routers have margins.  So ids and choices of
experts do not hang on the last bit of a sum, while the logits carry every layer's terms.
"""

from __future__ import annotations

import math
import random
import zlib

import numpy as np
import torch

EXPERTS = 8
NEXT = 4099                       # an untied head answers token t with token t + NEXT
PAGE = 16

QWEN = {
    "qwen2-0.5b": {"num_hidden_layers": 24, "hidden_size": 896, "num_attention_heads": 14, "num_key_value_heads": 2, "head_dim": 64,
                   "intermediate_size": 4864, "vocab_size": 151936, "tie_word_embeddings": True},
    "qwen2-7b": {"num_hidden_layers": 28, "hidden_size": 3584, "num_attention_heads": 28, "num_key_value_heads": 4, "head_dim": 128,
                 "intermediate_size": 18944, "vocab_size": 152064, "tie_word_embeddings": False},
}
DESIGNS = ("rososun", "nutopel", "kidolorn", "gerupel", "sezopel", "muzulorn")
WIDTHS = {2048: dict(layers=8, heads=16, ff=5632), 4096: dict(layers=4, heads=32, ff=11008)}
VOCAB, DIM, RANK = 32000, 128, 128


# ---- the cases ----------------------------------------------------------------------------------------------------------

def _case(name, model, kind, batch, prompt, new, width=0, dtype="bfloat16", sampled=False, portion=4096):
    return {"name": name, "model": model, "width": width, "dtype": dtype, "kind": kind, "batch": batch, "prompt": prompt, "new": new,
            "sampled": sampled, "portion": portion}


def listed():
    return [
        # one person's short question to a small model: latency and launches
        _case("qwen2-0.5b chat", "qwen2-0.5b", "generate", 1, 23, 16),
        # a small model under load: requests of mixed length, portions beside decoded tokens, Qwen2.5's own sampling defaults
        _case("qwen2-0.5b serving", "qwen2-0.5b", "generate", 32, 1024, 48, sampled=True, portion=512),
        # the 32-bit path: a few requests that are compared with another implementation
        _case("qwen2-0.5b float32", "qwen2-0.5b", "decode", 3, 181, 12, dtype="float32"),
        # a prompt of a common size on the main model: the time to the first token
        _case("qwen2-7b prompt", "qwen2-7b", "score", 1, 2048, 0),
        # the main model's decode batch
        _case("qwen2-7b batch", "qwen2-7b", "decode", 8, 512, 32),
        # a long document and an answer about it
        _case("qwen2-7b document", "qwen2-7b", "decode", 1, 12001, 48),
        # the other designs, prompts of one and of several requests, single answers and batches
        _case("rososun batch", "rososun", "decode", 8, 200, 40, width=2048),
        _case("nutopel prompt", "nutopel", "score", 1, 2048, 0, width=2048),
        _case("kidolorn ragged prompts", "kidolorn", "score", 3, 1001, 0, width=4096),
        _case("gerupel batch", "gerupel", "decode", 16, 300, 24, width=2048),
        _case("sezopel answer", "sezopel", "decode", 1, 700, 32, width=4096),
        _case("muzulorn ragged prompts", "muzulorn", "score", 5, 700, 0, width=2048),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    most = max(_cost(c) for c in listed())
    while True:
        model = rng.choice(("qwen2-0.5b", "qwen2-0.5b", "qwen2-7b", "qwen2-7b") + DESIGNS)
        kind = rng.choice(("score", "decode", "generate"))
        dtype = "float32" if model == "qwen2-0.5b" and rng.random() < 0.3 else "bfloat16"
        batch, prompt = _log(rng, 1, 48), _log(rng, 5, 8192)
        case = _case("", model, kind, batch, prompt, 0 if kind == "score" else _log(rng, 4, 64),
                     width=rng.choice((2048, 4096)) if model in DESIGNS else 0, dtype=dtype,
                     sampled=kind == "generate" and rng.random() < 0.5, portion=rng.choice((512, 1024, 4096)))
        del case["name"]
        tokens = sum(_lens(case))
        if tokens > (2048 if dtype == "float32" else 16384) or (model in DESIGNS and tokens > 4096) or _cost(case) > most:
            continue
        return case


def _lens(case):
    """Prompt lengths of the case's requests: the first as long as said, the others anything down to half of it."""
    p = case["prompt"]
    return [p - (i * 7919) % (p // 2 + 1) for i in range(case["batch"])]


# ---- configurations -----------------------------------------------------------------------------------------------------

def config_of(case):
    """config.json's keys of the case's model."""
    m = case["model"]
    if m in QWEN:
        return dict({"architectures": ["Qwen2ForCausalLM"], "model_type": "qwen2", "rope_theta": 1000000.0, "rms_norm_eps": 1e-6,
                     "max_position_embeddings": 32768, "hidden_act": "silu"}, **QWEN[m])
    W, D = case["width"], DIM
    n, H, ff = (WIDTHS[W][k] for k in ("layers", "heads", "ff"))
    G, rot = max(1, H // 8), D // 4
    heads, eff, shared = W // 64, ff // 4 // 64 * 64, ff // 2 // 64 * 64
    decay = [1.0 - 2.0 ** (-5.0 - 5.0 * h / (heads - 1)) for h in range(heads)]
    c = {"architecture": m.capitalize(), "vocab": VOCAB, "width": W, "norm": {"eps": 1e-5}}
    plain = {"heads": H, "kv_heads": G, "dim": D, "vdim": D, "scale": D ** -0.5}
    latent = {"heads": H, "dim": D - rot, "rot_dim": rot, "vdim": D, "kv_rank": RANK - rot, "scale": D ** -0.5, "rot": {"base": 10000.0, "dims": rot}}
    if m == "rososun":
        mlp = {"kind": "dense", "ff": ff}
        kinds = [{"type": "general_delta", "mixer": {"heads": heads, "dim": 64, "decay_rank": 64}, "mlp": mlp},
                 {"type": "latent_attention", "mixer": {"heads": H, "dim": D, "vdim": D, "kv_rank": RANK, "scale": D ** -0.5}, "mlp": mlp}]
        return dict(c, embedding={"scale": 1.0}, norm={"eps": 1e-5, "groups": 4}, layers=[kinds[i % 2] for i in range(n)])
    if m == "nutopel":
        mlp = {"kind": "moe", "expert": {"ff": eff}, "shared": {"ff": shared},
               "router": {"experts": EXPERTS, "top": 2, "scale": 2.0, "groups": {"count": 4, "keep": 2}}}
        left = dict(plain, mask={"size": 1024}, rot={"base": 10000.0, "dims": D // 2, "scaling": {"factor": 4.0, "original": 2048, "fast": 32.0, "slow": 1.0}})
        right = {"heads": W // 128, "kv_heads": W // 256, "dim": 128, "vdim": 128, "conv": 4}
        kinds = [{"type": "gla", "mixer": {"heads": heads, "dim": 64, "vdim": 64, "tau": 8.0, "decay_rank": 64}, "mlp": mlp},
                 {"type": "parallel", "mixer": {"left": left, "right": right}, "mlp": mlp}]
        return dict(c, logit_scale=1.0, layers=[kinds[i % 2] for i in range(n)])
    if m == "kidolorn":
        moe = {"kind": "moe", "expert": {"ff": eff, "limit": 7.0}, "router": {"experts": EXPERTS, "top": 2}}
        dense = {"kind": "dense", "ff": ff, "limit": 7.0}
        layers = []
        for i in range(n):
            layers.append([{"type": "lightning", "mixer": {"heads": heads, "dim": 64, "vdim": 64, "decay": decay}, "mlp": moe},
                           {"type": "latent_attention", "mixer": latent, "mlp": dense},
                           {"type": "mingru", "mixer": {"width": W}, "mlp": moe},
                           {"type": "latent_attention", "mixer": dict(latent, kv_from=i - 2), "mlp": dense}][i % 4])
        return dict(c, canon={"taps": 4}, layers=layers)
    if m == "gerupel":
        mlp = {"kind": "moe", "expert": {"ff": eff}, "router": {"experts": EXPERTS, "top": 2, "scale": 2.0}}
        left = dict(plain, mask={"size": 1024, "pool": 64}, rot={"base": 10000.0, "dims": D // 2, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 2048}})
        layer = {"type": "parallel", "mlp": mlp, "mixer": {"left": left, "right": {"heads": W // 128, "dim": 128, "vdim": 128}, "left_scale": 1.0, "right_scale": 1.0}}
        k = n - 2
        return dict(c, residual_mult=0.5, loop={"start": k // 2 - 1, "stop": k // 2 + 1, "times": 2}, layers=[layer] * k)
    if m == "sezopel":
        mlp = {"kind": "dense", "ff": ff * 3 // 2 // 64 * 64}
        a = dict(plain, softcap=30.0, rot={"base": 10000.0, "dims": D // 2})
        r = {"type": "retention", "mlp": mlp, "mixer": {"heads": heads, "dim": 64, "vdim": 64, "decay": decay, "rot": {"base": 10000.0, "dims": 64}}}
        layers = [r if i % 2 else {"type": "attention", "mixer": dict(a, kv_from=i - 2) if i % 4 == 2 else a, "mlp": mlp} for i in range(n)]
        return dict(c, embedding={"scale": 1.0}, token_side={"dim": 256}, logit_softcap=60.0, layers=layers)
    dense = {"kind": "dense", "ff": ff * 3 // 2 // 64 * 64}
    moe = {"kind": "moe", "expert": {"ff": eff}, "shared": {"ff": shared}, "router": {"experts": EXPERTS, "top": 2}}
    a = dict(plain, softcap=30.0, bias_max=128, q_temp={"coef": 0.1, "every": 1024})
    layers = []
    for i in range(n):
        layers.append([{"type": "attention", "mixer": a, "mlp": dense},
                       {"type": "mamba2", "mixer": {"heads": 2 * W // 64, "vdim": 64, "state": 128, "groups": 1, "conv": 4, "norm_groups": 1}, "mlp": moe},
                       {"type": "latent_attention", "mixer": dict(latent, q_rank=W // 2, mask={"size": 1024}), "mlp": moe},
                       {"type": "attention", "mixer": dict(a, kv_from=i - 3), "mlp": dense}][i % 4])
    return dict(c, streams=4, residual_mult=0.5, embedding={"bigram": {"buckets": 65536, "mul_prev": 37, "mul_cur": 19}}, layers=layers)


# ---- weights ------------------------------------------------------------------------------------------------------------

class Weights:
    """Every tensor by its name, drawn from the seed and the name alone, rounded to the compute type."""

    def __init__(self, case, seed):
        self.case, self.seed = case, seed
        self.dtype = getattr(torch, case["dtype"])
        cfg = config_of(case)
        self.qwen = case["model"] in QWEN
        self.W = cfg["hidden_size"] if self.qwen else cfg["width"]
        layers = cfg["num_hidden_layers"] if self.qwen else len(cfg["layers"])
        self.branch = 1.0 / math.sqrt(2 * layers)            # what a sublayer adds to a stream that starts at one
        self.table = self.bare = None                        # the embedding, with and without its leanings

    def _normal(self, name, shape, mean=0.0, std=1.0):
        g = torch.Generator(device="cuda")
        g.manual_seed((self.seed * 1000003 + zlib.crc32(name.encode())) % (1 << 62))
        return torch.empty(shape, dtype=self.dtype, device="cuda").normal_(mean, std, generator=g)

    def _uniform(self, name, shape, lo, hi):
        g = torch.Generator(device="cuda")
        g.manual_seed((self.seed * 1000003 + zlib.crc32(name.encode())) % (1 << 62))
        return torch.empty(shape, dtype=torch.float32, device="cuda").uniform_(lo, hi, generator=g)

    def _leanings(self):
        return self._normal("leanings", (EXPERTS, self.W))

    def __call__(self, name, *shape):
        return self._value(name, shape).to(self.dtype)

    def _value(self, name, shape):
        parts = name.split(".")
        last = parts[-1] if not self.qwen else parts[-2]
        if self.qwen and parts[-1] == "bias":
            return self._normal(name, shape, 0.0, 0.2)
        if last in ("embed", "embed_tokens"):
            if parts[0] == "side":
                return self._normal(name, shape)
            if self.table is None:                            # (the head asks again)
                self.table = self.bare = self._normal(name, shape)
                if not self.qwen:
                    t = torch.arange(shape[0], device="cuda")
                    first = t % EXPERTS
                    second = (first + 1 + t // EXPERTS % (EXPERTS - 1)) % EXPERTS
                    d = self._leanings()
                    self.bare, self.table = self.table, self.table + 0.3 * d[first] + 0.2 * d[second]
            return self.table
        if last in ("head", "lm_head"):
            self(*(("model.embed_tokens.weight",) if self.qwen else ("embed",)), *shape)
            return torch.roll(self.bare, NEXT, 0)
        if last == "router":
            # the embedding's leanings, each layer with its experts in another order
            return (torch.roll(self._leanings(), int(parts[0][1:]), 0).float() * (12.0 / self.W))
        if last in ("norm", "norm1", "norm2", "norm1b", "norm2b", "out", "input_layernorm", "post_attention_layernorm"):
            mean, about_one = 1.0, self.case["model"] in ("nutopel", "muzulorn") and last in ("norm1", "norm2")
            if parts[-2] == "final" or (self.qwen and parts[-2:] == ["norm", "weight"]):
                mean, about_one = 40.0 / self.W, self.case["model"] in ("nutopel", "muzulorn")
            elif last in ("norm1b", "norm2b") or (self.case["model"] == "sezopel" and (last in ("norm1", "norm2") or parts[-2] == "side")):
                mean = self.branch
            elif last == "out" and parts[-2] in ("left", "right"):
                mean = self.branch
            return self._normal(name, shape, mean - (1.0 if about_one else 0.0), 0.1 * mean)
        special = {"w0": (-2.0, 1.5), "dt_bias": (-3.0, 1.0), "D": (1.0, 0.1), "temp": (1.0, 0.1), "sink": (0.0, 0.5), "rel": (0.0, 0.5),
                   "correction": (0.0, 0.01), "step": (0.0, 0.1), "bigram": (0.0, 0.3), "conv": (0.0, 0.5), "canon1": (0.0, 0.2), "canon2": (0.0, 0.2)}
        if last in special:
            return self._normal(name, shape, *special[last])
        if last == "A_log":
            return self._uniform(name, shape, 1.0, 16.0).log()
        if last in ("shift", "lower"):
            return self._uniform(name, shape, 0.05, 0.95)
        if last == "b":
            if parts[-2] in ("a2", "f"):
                return self._normal(name, shape, 2.0, 1.0)
            if len(shape) == 1:
                return self._normal(name, shape, 0.0, 0.01 if parts[-2] == "router" else 0.1)
        if len(parts) > 2 and parts[1].startswith("hc"):
            if last == "mix":
                return torch.eye(*shape, device="cuda") + self._normal(name, shape, 0.0, 0.05)
            return self._normal(name, shape, 0.25 if last == "in" else 1.0, 0.02)
        gain = 1.0
        if last in ("o", "down", "proj", "o_proj", "down_proj"):
            gain = (4.0 if last == "o" else 2.0) * self.branch
        elif last in ("q", "q_proj", "uq"):
            gain = 1.5
        return self._normal(name, shape, 0.0, gain / math.sqrt(shape[-1]))


# ---- what a program has in hand -------------------------------------------------------------------------------------------

def _prompts(case, seed):
    rng = np.random.default_rng((seed, 1))
    return [rng.integers(0, config_of(case)["vocab_size" if case["model"] in QWEN else "vocab"], size=n).tolist() for n in _lens(case)]


def _wanted(n):
    """Places of a scored prompt whose logits are asked for."""
    return sorted({n - 1 - k * n // 4 for k in range(4)})


def _model(case, seed):
    from sllm_b200.config.registry import architecture_of
    from sllm_b200.engine import loading                     # noqa: F401  (registers the architectures)
    from sllm_b200.models.causal_lm import CausalLM
    config = config_of(case)
    arch = architecture_of(config)
    model = CausalLM(arch.plan(arch.config_cls.from_dict(config)), dtype=getattr(torch, case["dtype"]), device="cuda:0")
    weights, specs = Weights(case, seed), {s.name: s for s in model.tensor_specs()}
    model.bind(lambda name: weights(name, *specs[name].concrete_shape()))
    return model


def prepare(case, seed):
    from sllm_b200.engine.engine import Engine
    from sllm_b200.engine.llm import LLM
    model = _model(case, seed)
    prompts, B = _prompts(case, seed), case["batch"]
    longest = max(len(p) for p in prompts) + case["new"] + 8
    pages = sum(-(-(len(p) + case["new"] + 8) // PAGE) + 1 for p in prompts)
    state = {"case": case, "prompts": prompts}
    if case["kind"] == "generate":
        state["llm"] = LLM(model=model, block_size=PAGE, num_pages=pages, max_num_seqs=B, max_model_len=longest, chunk_size=case["portion"],
                           max_batch_tokens=max(2048, B * min(case["portion"], 512)))
        state["llm"].warmup([n for n in range(1, B + 1)] if B <= 4 else [B], penalised=case["sampled"])
    else:
        state["engine"] = Engine(model, page_size=PAGE, num_pages=pages, max_requests=B, max_model_len=longest)
        if case["kind"] == "decode":
            n = max(len(p) for p in prompts)
            state["engine"].graphs.warmup([B], [n + 1, n + case["new"]])
    return state


# ---- one pass -------------------------------------------------------------------------------------------------------------

def _feed(engine, prompts, portion, want):
    """The prompts' tokens in portions, every request's next one in each step; the logits of the wanted places, in the requests' order."""
    from sllm_b200.engine.engine import StepEntry
    rows = [[] for _ in prompts]
    for at in range(0, max(len(p) for p in prompts), portion):
        entries, whose = [], []
        for i, p in enumerate(prompts):
            if at < len(p):
                part = p[at:at + portion]
                places = [w - at for w in want(len(p)) if at <= w < at + len(part)]
                entries.append(StepEntry(i, part, places))
                whose += [i] * len(places)
        logits = engine.step(entries)
        for r, i in enumerate(whose):
            rows[i].append(logits[r])
    return torch.stack([r for part in rows for r in part])


def run(state):
    case, prompts = state["case"], state["prompts"]
    if case["kind"] == "generate":
        from sllm_b200.sampling import SamplingParams
        if case["sampled"]:
            params = [SamplingParams(max_new=case["new"], temperature=0.7, top_k=20, top_p=0.8, repetition_penalty=1.05, seed=i) for i in range(len(prompts))]
        else:
            params = SamplingParams(max_new=case["new"])
        return {"ids": torch.tensor([r.ids for r in state["llm"].generate(prompts, params)])}
    engine = state["engine"]
    if case["kind"] == "score":
        logits = _feed(engine, prompts, case["portion"], _wanted)
        for i in range(len(prompts)):
            engine.finish(i)
        return {"logits": logits}
    from sllm_b200 import ops
    from sllm_b200.engine.engine import StepEntry
    first = _feed(engine, prompts, case["portion"], lambda n: [n - 1])
    step_ids = [ops.sample_rows(first).tolist()]
    B = len(prompts)
    temps, uniforms = np.zeros(B, np.float32), np.zeros(B, np.float64)
    flying = None
    for n in range(case["new"] - 1):                         # each step is queued behind the one whose ids are read
        entries = [StepEntry(i, [step_ids[0][i]], [0]) for i in range(B)]
        queued = engine.graphs.launch(entries, temps, uniforms, after=flying)
        if flying is not None:
            step_ids.append(engine.graphs.read(flying))
        flying = queued
    step_ids.append(engine.graphs.read(flying))
    last = engine.step([StepEntry(i, [step_ids[-1][i]], [0]) for i in range(B)])
    for i in range(B):
        engine.finish(i)
    return {"first": first, "ids": torch.tensor(step_ids).T.contiguous(), "last": last}


# ---- what a pass cannot do without ------------------------------------------------------------------------------------------

def _sizes(case):
    """(bytes of the weights that a step over so many tokens reads, multiplications of one token, bytes of the head, multiplications of
    one row of it, cached bytes of so many tokens, channels of queries and values over all attention layers)."""
    cfg, item = config_of(case), 2 if case["dtype"] == "bfloat16" else 4
    if case["model"] in QWEN:
        L, W, F, V = (cfg[k] for k in ("num_hidden_layers", "hidden_size", "intermediate_size", "vocab_size"))
        q, kv = cfg["num_attention_heads"] * cfg["head_dim"], cfg["num_key_value_heads"] * cfg["head_dim"]
        body = L * (2 * W * q + 2 * W * kv + 3 * W * F)
        return lambda tokens: body * item, body, V * W * item, V * W, lambda n: L * 2 * kv * item * n, L * 2 * q
    W, V = cfg["width"], cfg["vocab"]
    dense = moe = cached = channels = 0
    order = list(cfg["layers"])
    if cfg.get("loop"):
        lo, hi, times = (cfg["loop"][k] for k in ("start", "stop", "times"))
        order = order[:lo] + order[lo:hi] * times + order[hi:]
    for layer in order:
        m, mlp = layer["mixer"], layer["mlp"]
        for s in (m["left"], m["right"]) if "left" in m else (m,):
            if "mask" in s or layer["type"] in ("attention", "latent_attention"):
                H, D, V2 = s["heads"], s["dim"] + s.get("rot_dim", 0), s["vdim"]
                channels += H * (D + V2)
                own = s.get("kv_from") is None
                if "kv_rank" in s:
                    row = s["kv_rank"] + s.get("rot_dim", 0)
                    dense += W * H * D if "q_rank" not in s else s["q_rank"] * (W + H * D)
                    dense += own * W * row + s["kv_rank"] * H * (s["dim"] + V2) + W * H * V2 * (2 if "rot_dim" in s else 1)
                else:
                    row = s["kv_heads"] * (D + V2)
                    dense += 2 * W * H * D + own * W * row
                cached += row * item
            elif layer["type"] == "mamba2":
                inner = s["heads"] * s["vdim"]
                dense += W * (3 * inner + 2 * s["groups"] * s["state"]) + s["heads"] * s["state"] * s["vdim"] * 2
            elif layer["type"] == "mingru":
                dense += 4 * W * W
            else:
                kd, vd = s.get("kv_heads", s["heads"]) * s["dim"], s["heads"] * s.get("vdim", s["dim"])
                dense += W * (2 * kd + 3 * vd) + s["heads"] * s["dim"] * s.get("vdim", s["dim"]) * 2
        if mlp["kind"] == "dense":
            dense += W * mlp["ff"] * (3 if case["model"] in ("rososun", "kidolorn") else 2)
        else:
            three = 2 if case["model"] == "nutopel" else 3
            moe += W * mlp["expert"]["ff"] * three
            dense += W * mlp["shared"]["ff"] * three if mlp.get("shared") else 0
    used = lambda tokens: EXPERTS * (1 - (1 - 2 / EXPERTS) ** tokens)  # noqa: E731  (experts that some token of the step uses)
    return lambda tokens: (dense + moe * used(tokens)) * item, dense + 2 * moe, V * W * item, V * W, lambda n: cached * n, channels


def work(case):
    weights, per_token, head, head_mults, cached, channels = _sizes(case)
    lens = _lens(case)
    B, item = case["batch"], 2 if case["dtype"] == "bfloat16" else 4
    rows = sum(len(_wanted(n)) for n in lens) if case["kind"] == "score" else B
    V = config_of(case)["vocab_size" if case["model"] in QWEN else "vocab"]
    bytes_ = weights(sum(lens)) + head + cached(sum(lens)) + rows * V * 4
    flops = 2 * (sum(lens) * per_token + rows * head_mults) + sum(n * n * channels for n in lens)
    steps = max(0, case["new"] - 1) + (case["kind"] == "decode")
    for s in range(steps):                                   # a decoded token reads the weights and its context
        bytes_ += weights(B) + head + cached(sum(lens) + B * s)
        flops += 2 * B * (per_token + head_mults) + 2 * sum(n + s for n in lens) * channels
    if case["kind"] == "decode":
        bytes_ += B * V * 4
    return {"bytes": float(bytes_), "flops": float(flops)}


def _cost(case):
    """Seconds, roughly: what decides whether a drawn case is no dearer than the listed ones."""
    w = work(case)
    steps = case["new"] + sum(_lens(case)) / 2048
    return w["bytes"] / 5e12 + w["flops"] / (1e15 if case["dtype"] == "bfloat16" else 3e13) + steps * 1e-3


def tolerance(case):
    """bfloat16 activations over the depth of the model; 32-bit sums in another order.  Ids are whole numbers; the head's margin keeps them."""
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 1e-4, "differ": 0.0}      # 1.5e-6 off the 64-bit statement
    return {"rel": 0.025, "max": 0.25, "differ": 0.002}       # 0.0016 to 0.0094 off, by design and size


# ---- the same in 64 bits, in plain torch -------------------------------------------------------------------------------------

def _unit(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(x):
    return x * torch.sigmoid(x)


def _rotate(x, freqs, mag=1.0, pairs=False):
    """x [B, T, heads, d]: the first 2 len(freqs) channels turn with the position, channel i with i + half (or 2i with 2i + 1)."""
    n = len(freqs)
    ang = torch.arange(x.shape[1], device=x.device, dtype=x.dtype)[:, None] * freqs[None, :]
    c, s = (torch.cos(ang) * mag)[None, :, None], (torch.sin(ang) * mag)[None, :, None]
    out = x.clone()
    if pairs:
        u, v = x[..., 0:2 * n:2], x[..., 1:2 * n:2]
        out[..., 0:2 * n:2], out[..., 1:2 * n:2] = u * c - v * s, v * c + u * s
    else:
        u, v = x[..., :n], x[..., n:2 * n]
        out[..., :n], out[..., n:2 * n] = u * c - v * s, v * c + u * s
    return out


def _freqs(rot):
    """(frequencies, factor of cos and sin), with the two kinds of scaling the designs have."""
    dims, base = rot["dims"], float(rot["base"])
    i = torch.arange(dims // 2, device="cuda", dtype=torch.float64)
    f = base ** (-2.0 * i / dims)
    sc = rot.get("scaling")
    if sc is None:
        return f, 1.0
    if "fast" in sc:
        at = lambda turns: dims * math.log(sc["original"] / (2 * math.pi * turns)) / (2 * math.log(base))  # noqa: E731
        lo, hi = max(math.floor(at(sc["fast"])), 0), min(math.ceil(at(sc["slow"])), dims - 1)
        ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0, 1)
        return f / sc["factor"] * ramp + f * (1 - ramp), 0.1 * math.log(sc["factor"]) + 1.0
    wave = 2 * math.pi / f
    s = ((sc["original"] / wave - sc["low"]) / (sc["high"] - sc["low"])).clamp(0, 1)
    return (1 - s) * f / sc["factor"] + s * f, 1.0


def _attend(q, k, v, scale, seen=None, cap=None, bias=None, sink=None, extra=None):
    """q [B, T, H, d], k [B, T, G, d], v [B, T, G, dv], causal.  ``seen(i, j)``: which of the earlier keys count; ``bias`` [H, T] by distance;
    ``sink`` [H]: one more term in the denominator; ``extra`` = (keys, values, seen) more of them in front.  Queries in blocks."""
    B, T, H, _ = q.shape
    G = k.shape[2]
    j = torch.arange(T, device=q.device)
    if extra is not None:
        k, v = torch.cat([extra[0], k], 1), torch.cat([extra[1], v], 1)
    k, v = k.permute(0, 2, 3, 1), v.transpose(1, 2)
    out = []
    for lo in range(0, T, 512):
        i = torch.arange(lo, min(T, lo + 512), device=q.device)
        qb = q[:, lo:lo + 512].transpose(1, 2)                                       # [B, H, t, d]
        s = (qb.reshape(B, G, -1, qb.shape[-1]) @ k).reshape(B, H, len(i), -1) * scale
        if cap is not None:
            s = cap * torch.tanh(s / cap)
        ok = j[None, :] <= i[:, None]
        if bias is not None:
            s = s + bias[:, (i[:, None] - j[None, :]).clamp(min=0)]
        if seen is not None:
            ok = ok & seen(i[:, None], j[None, :])
        if extra is not None:
            ok = torch.cat([extra[2](i), ok], 1)
        s = s.masked_fill(~ok, -math.inf)
        top = s.amax(-1, keepdim=True)
        if sink is not None:
            top = torch.maximum(top, sink[:, None, None])
        e = torch.exp(s - top)
        den = e.sum(-1, keepdim=True) + (torch.exp(sink[:, None, None] - top) if sink is not None else 0.0)
        o = ((e / den).reshape(B, G, -1, e.shape[-1]) @ v).reshape(B, H, len(i), -1)
        out.append(o.transpose(1, 2))
    return torch.cat(out, 1)


def _conv(x, taps):
    """x [B, T, C], taps [C, n]: per channel over the last n tokens, zeros before the start."""
    n = taps.shape[1]
    padded = torch.cat([torch.zeros_like(x[:, :1]).expand(-1, n - 1, -1), x], 1)
    return sum(padded[:, m:m + x.shape[1]] * taps[:, m] for m in range(n))


def _walk(q, k, v, keep):
    """S <- keep S + k v^T, o = S^T q, token by token; ``keep`` [B, T, H, d or 1]."""
    S = torch.zeros(q.shape[0], q.shape[2], q.shape[3], v.shape[3], device=q.device, dtype=q.dtype)
    out = torch.empty_like(v)
    for t in range(q.shape[1]):
        S = S * keep[:, t, :, :, None] + k[:, t, :, :, None] * v[:, t, :, None, :]
        out[:, t] = (q[:, t, :, None, :] @ S)[:, :, 0]
    return out


class _Plain:
    def __init__(self, case, seed):
        self.cfg, self.draw = config_of(case), Weights(case, seed)
        self.model, self.W = case["model"], self.draw.W
        self.kept = {}

    def w(self, name, *shape):
        return self.draw(name, *shape).double()

    def lin(self, x, name, n, bias=False):
        y = x @ self.w(name, n, x.shape[-1]).T
        return y + self.w(name + ".b", n) if bias else y

    def gain(self, x, name, eps, offset=0.0):
        return _unit(x, eps) * (offset + self.w(name, *((x.shape[-1],) if self.model != "kidolorn" or name.count(".") == 3 or name.endswith("mix.norm") else ())))

    # -- mixers
    def latent(self, h, p, m, eps, i):
        B, T, W = h.shape
        H, d, r, dv, rank = m["heads"], m["dim"], m.get("rot_dim", 0), m["vdim"], m["kv_rank"]
        pairs = self.model == "muzulorn"
        if "q_rank" in m:
            q = self.lin(_unit(self.lin(h, p + "dq", m["q_rank"]), eps) * self.w(p + "dq.norm", m["q_rank"]), p + "uq", H * (d + r))
        else:
            q = self.lin(h, p + "q", H * (d + r))
        q = q.reshape(B, T, H, d + r)
        if m.get("kv_from") is None:
            down = self.lin(h, p + "dkv", rank + r)
            c = _unit(down[..., :rank], eps) * self.w(p + "dkv.norm", rank)
            self.kept[i] = (c, _rotate(down[:, :, None, rank:], *_freqs(m["rot"]), pairs=pairs)[:, :, 0] if r else None)
        c, kr = self.kept[i if m.get("kv_from") is None else m["kv_from"]]
        k = self.lin(c, p + "uk", H * d).reshape(B, T, H, d)
        v = self.lin(c, p + "uv", H * dv).reshape(B, T, H, dv)
        if r:
            q = torch.cat([q[..., :d], _rotate(q[..., d:], *_freqs(m["rot"]), pairs=pairs)], -1)
            k = torch.cat([k, kr[:, :, None].expand(-1, -1, H, -1)], -1)
        size = (m.get("mask") or {}).get("size")
        o = _attend(q, k, v, m["scale"], seen=(lambda a, b: a - b < size) if size else None, sink=self.w(p + "sink", H) if r else None)
        if r:
            return self.lin(o.reshape(B, T, H * dv) * torch.sigmoid(self.lin(h, p + "g", H * dv)), p + "o", W)
        return self.lin((o * torch.sigmoid(self.lin(h, p + "g", H))[..., None]).reshape(B, T, H * dv), p + "o", W)

    def general_delta(self, h, p, m, eps):
        B, T, W = h.shape
        H, d = m["heads"], m["dim"]
        r, k, v = (self.lin(h, p + n, H * d).reshape(B, T, H, d) for n in "rkv")
        keep = torch.exp(-math.exp(-0.5) * torch.sigmoid(self.lin(torch.tanh(self.lin(h, p + "w1", m["decay_rank"])), p + "w2", H * d) + self.w(p + "w0", H * d)))
        a = torch.sigmoid(self.lin(h, p + "a", H * d, bias=True)).reshape(B, T, H, d)
        keep = keep.reshape(B, T, H, d)
        u = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
        S, o = torch.zeros(B, H, d, d, device=h.device, dtype=h.dtype), torch.empty_like(v)
        for t in range(T):
            S = keep[:, t, :, :, None] * S - (a[:, t] * u[:, t])[..., None] * (u[:, t, :, None] @ S) + k[:, t, :, :, None] * v[:, t, :, None]
            o[:, t] = (r[:, t, :, None] @ S)[:, :, 0]
        o = _unit(o, eps).reshape(B, T, H * d) * self.w(p + "norm", H * d) * torch.sigmoid(self.lin(h, p + "g", H * d))
        return self.lin(o, p + "o", W)

    def gated_delta(self, h, p, m, eps):
        B, T, W = h.shape
        H, G, d, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        q, k, v = (_silu(_conv(self.lin(h, p + n, c), self.w(p + n + ".conv", c, m["conv"]))) for n, c in (("q", G * d), ("k", G * d), ("v", H * dv)))
        q, k, v = q.reshape(B, T, G, d), k.reshape(B, T, G, d), v.reshape(B, T, H, dv)
        q, k = (x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6) for x in (q, k))
        q, k = (x.repeat_interleave(H // G, 2) for x in (q * d ** -0.5, k))
        beta = torch.sigmoid(self.lin(h, p + "b", H))
        keep = torch.exp(-torch.exp(self.w(p + "A_log", H)) * torch.nn.functional.softplus(self.lin(h, p + "a", H) + self.w(p + "dt_bias", H)))
        S, o = torch.zeros(B, H, d, dv, device=h.device, dtype=h.dtype), torch.empty_like(v)
        for t in range(T):
            S = keep[:, t, :, None, None] * S
            S = S + k[:, t, :, :, None] * (beta[:, t, :, None] * (v[:, t] - (k[:, t, :, None] @ S)[:, :, 0]))[:, :, None]
            o[:, t] = (q[:, t, :, None] @ S)[:, :, 0]
        o = _unit(o, eps) * self.w(p + "norm", dv) * _silu(self.lin(h, p + "g", H * dv)).reshape(B, T, H, dv)
        return self.lin(o.reshape(B, T, H * dv), p + "o", W)

    def grouped(self, h, p, m, eps, i):
        """Attention with keys and values per group of heads, in the forms the designs have."""
        B, T, W = h.shape
        H, G, d, dv, name = m["heads"], m["kv_heads"], m["dim"], m["vdim"], self.model
        q = self.lin(h, p + "q", H * d, bias=name == "muzulorn")
        if m.get("kv_from") is None:
            k, v = (self.lin(h, p + n, G * c, bias=name == "muzulorn") for n, c in (("k", d), ("v", dv)))
            if name == "muzulorn":
                k = _unit(k, eps) * self.w(p + "k.norm", G * d)
            k, v = k.reshape(B, T, G, d), v.reshape(B, T, G, dv)
            if name == "nutopel":
                k = _unit(k, eps) * self.w(p + "k.norm", d)
            if m.get("rot"):
                k = _rotate(k, *_freqs(m["rot"]))
            if name == "sezopel":
                k = _unit(k, eps)
            self.kept[i] = (k, v)
        k, v = self.kept[i if m.get("kv_from") is None else m["kv_from"]]
        if name == "muzulorn":
            q = _unit(q, eps) * self.w(p + "q.norm", H * d)
            t = torch.arange(T, device=h.device, dtype=h.dtype)
            q = q * (1 + m["q_temp"]["coef"] * torch.log(torch.floor((t + 1) / m["q_temp"]["every"]) + 1))[None, :, None]
        q = q.reshape(B, T, H, d)
        if name == "nutopel":
            q = _unit(q, eps) * self.w(p + "q.norm", d)
        if m.get("rot"):
            q = _rotate(q, *_freqs(m["rot"]))
        if name == "sezopel":
            o = _attend(_unit(q, eps), k, v, m["scale"], cap=m["softcap"]) * torch.sigmoid(self.lin(h, p + "g", H))[..., None]
        elif name == "nutopel":
            size = m["mask"]["size"]
            o = _attend(q, k, v, m["scale"], seen=lambda a, b: a // size == b // size)
        elif name == "gerupel":
            size, pool = m["mask"]["size"], m["mask"]["pool"]
            nb = T // pool
            pk, pv = (x[:, :nb * pool].reshape(B, nb, pool, G, -1).mean(2) for x in (k, v))
            ends = torch.arange(nb, device=h.device) * pool + pool - 1
            o = _attend(q * self.w(p + "temp", H)[:, None], k, v, m["scale"], seen=lambda a, b: a - b < size,
                        sink=torch.zeros(H, device=h.device, dtype=h.dtype), extra=(pk, pv, lambda a: ends[None, :] <= a[:, None] - size))
        else:
            rel = self.w(p + "rel", 16, H)
            n, half = torch.arange(T), rel.shape[0] // 2
            bucket = torch.tensor([x if x < half else min(rel.shape[0] - 1, half + math.floor(math.log(x / half) / math.log(m["bias_max"] / half) * (rel.shape[0] - half)))
                                   for x in n.tolist()], device=h.device)
            o = _attend(q, k, v, m["scale"], cap=m["softcap"], bias=rel[bucket].T)
        return self.lin(o.reshape(B, T, H * dv), p + "o", W, bias=name == "muzulorn")

    def linear_kind(self, h, p, m, eps, kind):
        B, T, W = h.shape
        H, d, dv = m["heads"], m["dim"], m["vdim"]
        q = self.lin(h, p + "q", H * d).reshape(B, T, H, d)
        v = self.lin(h, p + "v", H * dv).reshape(B, T, H, dv)
        if kind == "hgrn2":
            low = self.w(p + "lower", H * d)
            keep = (low + (1 - low) * torch.sigmoid(self.lin(h, p + "f", H * d, bias=True))).reshape(B, T, H, d)
            o = _unit(_walk(_silu(q), 1 - keep, v, keep), eps) * self.w(p + "norm", dv)
            return self.lin(o.reshape(B, T, H * dv), p + "o", W)
        k = self.lin(h, p + "k", H * d).reshape(B, T, H, d)
        if kind == "gla":
            z = self.lin(self.lin(h, p + "a1", m["decay_rank"]), p + "a2", H * d, bias=True)
            o = _walk(q * d ** -0.5, k, v, (torch.sigmoid(z) ** (1.0 / m["tau"])).reshape(B, T, H, d))
            o = (_unit(o, eps) * self.w(p + "norm", dv)).reshape(B, T, H * dv) * _silu(self.lin(h, p + "g", H * dv))
            return self.lin(o, p + "o", W)
        keep = torch.tensor(m["decay"], device=h.device, dtype=h.dtype)[None, None, :, None].expand(B, T, H, 1)
        if kind == "lightning":
            o = _walk(_silu(q), _silu(k), _silu(v), keep).reshape(B, T, H * dv)
            o = _unit(o, eps) * self.w(p + "norm", H * dv) * torch.sigmoid(self.lin(h, p + "g", H * dv))
            return self.lin(o, p + "o", W)
        f = _freqs(m["rot"])
        o = _walk(_rotate(q, *f), _rotate(k, *f) * d ** -0.5, v, keep)
        return self.lin(_unit(o, eps).reshape(B, T, H * dv) * _silu(self.lin(h, p + "g", H * dv)), p + "o", W)

    def mingru(self, h, p, W):
        z, u = torch.sigmoid(self.lin(h, p + "z", W, bias=True)), self.lin(h, p + "x", W, bias=True)
        cand, S, y = torch.where(u >= 0, u + 0.5, torch.sigmoid(u)), torch.zeros_like(h[:, 0]), torch.empty_like(h)
        for t in range(h.shape[1]):
            S = (1 - z[:, t]) * S + z[:, t] * cand[:, t]
            y[:, t] = S
        return self.lin(y * _silu(self.lin(h, p + "g", W)), p + "o", W)

    def mamba2(self, h, p, m, eps):
        B, T, W = h.shape
        H, dv, N = m["heads"], m["vdim"], m["state"]
        inner = H * dv
        z, xbc, dt = self.lin(h, p + "in", 2 * inner + 2 * N + H).split([inner, inner + 2 * N, H], -1)
        xbc = _silu(_conv(xbc, self.w(p + "conv", inner + 2 * N, m["conv"])) + self.w(p + "conv.b", inner + 2 * N))
        x, b, c = xbc.split([inner, N, N], -1)
        x = x.reshape(B, T, H, dv)
        dt = torch.nn.functional.softplus(dt + self.w(p + "dt_bias", H))
        keep = torch.exp(-torch.exp(self.w(p + "A_log", H)) * dt)[..., None]
        y = _walk(c[:, :, None].expand(-1, -1, H, -1), dt[..., None] * b[:, :, None], x, keep) + self.w(p + "D", H)[:, None] * x
        y = _unit(y.reshape(B, T, inner) * _silu(z), eps) * self.w(p + "norm", inner)
        return self.lin(y, p + "o", W)

    # -- feed-forwards
    def experts(self, h, p, mlp):
        B, T, W = h.shape
        x, r, ff, name = h.reshape(-1, W), mlp["router"], mlp["expert"]["ff"], self.model
        z = self.lin(x, p + "router", EXPERTS, bias=name == "muzulorn")
        if name == "nutopel":
            s = torch.sigmoid(z)
            choice = s + self.w(p + "correction", EXPERTS)
            n, keep = r["groups"]["count"], r["groups"]["keep"]
            score = choice.reshape(-1, n, EXPERTS // n).topk(2, -1).values.sum(-1)
            kept = torch.zeros_like(score, dtype=torch.bool).scatter_(1, score.topk(keep, -1).indices, True)
            idx = choice.masked_fill(~kept.repeat_interleave(EXPERTS // n, 1), -math.inf).topk(2, -1).indices
            wt = s.gather(1, idx) * r["scale"]
        elif name == "gerupel":
            top = torch.softmax(z, -1).topk(2, -1)
            idx, wt = top.indices, top.values / (top.values.sum(-1, keepdim=True) + 1e-20) * r["scale"]
        else:
            top = z.topk(2, -1)
            idx, wt = top.indices, torch.softmax(top.values, -1)
        out = torch.zeros_like(x)
        for e in range(EXPERTS):
            rows, place = (idx == e).nonzero(as_tuple=True)
            if len(rows):
                out[rows] += wt[rows, place][:, None] * self.unit(x[rows], f"{p}e{e}.", ff, mlp["expert"].get("limit"))
        if mlp.get("shared"):
            y = self.unit(x, p + "shared.", mlp["shared"]["ff"])
            out = out + (y * torch.sigmoid(self.lin(x, p + "shared.sg", 1)) if name == "muzulorn" else y)
        return out.reshape(B, T, W)

    def unit(self, x, p, ff, limit=None, bias=False):
        up = self.lin(x, p + "up", ff, bias=bias)
        if self.model == "sezopel":
            y = up.clamp(min=0) ** 2
        elif self.model == "nutopel" or (self.model == "muzulorn" and "mlp.e" not in p and "shared" not in p):
            y = torch.nn.functional.gelu(up)
        else:
            g = self.lin(x, p + "gate", ff, bias=bias)
            if limit is not None:
                g = g.clamp(max=limit)
                y = g * torch.sigmoid(1.702 * g) * (up.clamp(-limit, limit) + 1)
            elif self.model == "rososun":
                y = torch.nn.functional.gelu(g, approximate="tanh") * up
            else:
                y = _silu(g) * up
        return self.lin(y, p + "down", self.W, bias=bias)

    def ff(self, h, p, mlp):
        if mlp["kind"] == "moe":
            return self.experts(h, p, mlp)
        return self.unit(h, p, mlp["ff"], mlp.get("limit"), bias=self.model in ("rososun", "kidolorn"))

    def mixer(self, h, p, layer, eps, i):
        m, kind = layer["mixer"], layer["type"]
        if kind == "parallel":
            left = self.grouped(h, p + "left.", m["left"], eps, i)
            if self.model == "gerupel":
                return left + self.linear_kind(h, p + "right.", m["right"], eps, "hgrn2")
            right = self.gated_delta(h, p + "right.", m["right"], eps)
            return 0.5 * (_unit(left, eps) * self.w(p + "left.out", self.W) + _unit(right, eps) * self.w(p + "right.out", self.W))
        if kind == "general_delta":
            return self.general_delta(h, p, m, eps)
        if kind == "latent_attention":
            return self.latent(h, p, m, eps, i)
        if kind == "attention":
            return self.grouped(h, p, m, eps, i)
        if kind == "mamba2":
            return self.mamba2(h, p, m, eps)
        return self.mingru(h, p, self.W) if kind == "mingru" else self.linear_kind(h, p, m, eps, kind)

    # -- the models
    def stream(self, ids):
        """ids [B, T] -> the last stream [B, T, W], normed, ready for the head."""
        if self.model in QWEN:
            return self.qwen(ids)
        cfg, W = self.cfg, self.W
        eps = cfg["norm"]["eps"]
        table = self.w("embed", cfg["vocab"], W)
        x = table[ids]
        if self.model == "rososun":
            return self.rososun(x, eps)
        if self.model == "muzulorn":
            return self.muzulorn(x, ids, eps)
        if self.model == "gerupel":
            return self.gerupel(x, eps)
        side = self.w("side.embed", cfg["vocab"], 256 * len(cfg["layers"]))[ids] if self.model == "sezopel" else None
        for i, layer in enumerate(cfg["layers"]):
            p = f"l{i}."
            if self.model == "nutopel":
                x = x + self.mixer(self.gain(x, p + "norm1", eps, 1.0), p + "mix.", layer, eps, i)
                x = x + self.ff(self.gain(x, p + "norm2", eps, 1.0), p + "mlp.", layer["mlp"])
            elif self.model == "kidolorn":
                for n, sub in (("1", lambda h: self.mixer(h, p + "mix.", layer, eps, i)), ("2", lambda h: self.ff(h, p + "mlp.", layer["mlp"]))):
                    h = _unit(x, eps) * self.w(p + "norm" + n)
                    h = h + _conv(h, self.w(p + "canon" + n, W, 4))
                    x = x + _unit(sub(h), eps) * self.w(p + f"norm{n}b")
            else:
                x = x + self.gain(self.mixer(x, p + "mix.", layer, eps, i), p + "norm1", eps)
                x = x + self.gain(self.ff(x, p + "mlp.", layer["mlp"]), p + "norm2", eps)
                g = torch.nn.functional.gelu(self.lin(x, p + "side.gate", 256), approximate="tanh")
                x = x + self.gain(self.lin(g * side[..., 256 * i:256 * (i + 1)], p + "side.proj", W), p + "side.norm", eps)
        if self.model == "kidolorn":
            return _unit(x, eps) * self.w("final.norm")
        return self.gain(x, "final.norm", eps, 1.0 if self.model == "nutopel" else 0.0)

    def rososun(self, x, eps):
        W, groups = self.W, self.cfg["norm"]["groups"]
        norm = lambda y, name: _unit(y.reshape(*y.shape[:2], groups, -1), eps).reshape(y.shape) * self.w(name, W)  # noqa: E731
        ang = torch.arange(x.shape[1], device=x.device, dtype=x.dtype)[:, None] * 10000.0 ** (-2.0 * torch.arange(W // 2, device=x.device, dtype=x.dtype) / W)
        x = x + torch.stack([torch.sin(ang), torch.cos(ang)], -1).reshape(1, -1, W)
        for i, layer in enumerate(self.cfg["layers"]):
            h = norm(x, f"l{i}.norm1")
            before = torch.cat([torch.zeros_like(h[:, :1]), h[:, :-1]], 1)
            x = x + self.mixer(h + (before - h) * self.w(f"l{i}.shift", W), f"l{i}.mix.", layer, eps, i) + self.ff(h, f"l{i}.mlp.", layer["mlp"])
        return norm(x, "final.norm")

    def gerupel(self, x, eps):
        cfg, W = self.cfg, self.W
        emb = x = self.gain(x, "embed.norm", eps)
        loop = cfg["loop"]
        order = [(i, None) for i in range(loop["start"])] + [(i, t) for t in range(loop["times"]) for i in range(loop["start"], loop["stop"])]
        order += [(i, None) for i in range(loop["stop"], len(cfg["layers"]))]
        for i, t in order:
            if t is not None and i == loop["start"]:
                x = x + (emb if t > 0 else 0) + self.w("loop.step", loop["times"], W)[t]
            layer, p = cfg["layers"][i], f"l{i}."
            term = self.mixer(self.gain(x, p + "norm1", eps), p + "mix.", layer, eps, i) + self.ff(self.gain(x, p + "norm2", eps), p + "mlp.", layer["mlp"])
            x = x + cfg["residual_mult"] * term
        return self.gain(x, "final.norm", eps)

    def muzulorn(self, x, ids, eps):
        cfg, W = self.cfg, self.W
        bg, n = cfg["embedding"]["bigram"], cfg["streams"]
        rows = torch.full_like(ids, bg["buckets"])
        rows[:, 1:] = (ids[:, :-1] * bg["mul_prev"] + ids[:, 1:] * bg["mul_cur"]) % bg["buckets"]
        xs = (x + self.w("bigram", bg["buckets"] + 1, W)[rows])[None].expand(n, -1, -1, -1)

        def connect(xs, p, sub):
            y = sub(torch.einsum("s,sbtw->btw", self.w(p + "in", n), xs))
            return torch.einsum("sbtw,sr->rbtw", xs, self.w(p + "mix", n, n)) + cfg["residual_mult"] * self.w(p + "out", n)[:, None, None, None] * y
        for i, layer in enumerate(cfg["layers"]):
            p = f"l{i}."
            xs = connect(xs, p + "hc1.", lambda u: self.mixer(self.gain(u, p + "norm1", eps, 1.0), p + "mix.", layer, eps, i))
            xs = connect(xs, p + "hc2.", lambda u: self.ff(self.gain(u, p + "norm2", eps, 1.0), p + "mlp.", layer["mlp"]))
        return self.gain(xs.sum(0), "final.norm", eps, 1.0)

    def qwen(self, ids):
        c, W = self.cfg, self.W
        eps, H, G, d = (c[k] for k in ("rms_norm_eps", "num_attention_heads", "num_key_value_heads", "head_dim"))
        B, T = ids.shape
        x = self.draw("model.embed_tokens.weight", c["vocab_size"], W)[ids].double()
        f = _freqs({"dims": d, "base": c["rope_theta"]})
        for i in range(c["num_hidden_layers"]):
            p = f"model.layers.{i}."
            h = _unit(x, eps) * self.w(p + "input_layernorm.weight", W)
            q, k, v = ((h @ self.w(f"{p}self_attn.{n}_proj.weight", m * d, W).T + self.w(f"{p}self_attn.{n}_proj.bias", m * d)).reshape(B, T, m, d)
                       for n, m in (("q", H), ("k", G), ("v", G)))
            o = _attend(_rotate(q, *f), _rotate(k, *f), v, d ** -0.5)
            x = x + o.reshape(B, T, H * d) @ self.w(p + "self_attn.o_proj.weight", W, H * d).T
            h = _unit(x, eps) * self.w(p + "post_attention_layernorm.weight", W)
            F = c["intermediate_size"]
            y = _silu(h @ self.w(p + "mlp.gate_proj.weight", F, W).T) * (h @ self.w(p + "mlp.up_proj.weight", F, W).T)
            x = x + y @ self.w(p + "mlp.down_proj.weight", W, F).T
        return _unit(x, eps) * self.w("model.norm.weight", W)

    def logits(self, rows):
        c = self.cfg
        if self.model in QWEN:
            tied, V = c["tie_word_embeddings"], c["vocab_size"]
            head = self.draw("model.embed_tokens.weight" if tied else "lm_head.weight", V, self.W)
        else:
            tied, V = self.model == "gerupel", c["vocab"]
            head = self.draw("embed" if tied else "head", V, self.W)
        z = torch.cat([rows @ head[lo:lo + 16384].double().T for lo in range(0, V, 16384)], -1)
        cap = c.get("logit_softcap")
        return cap * torch.tanh(z / cap) if cap is not None else z


def exact(case, seed):
    if case["kind"] == "generate":
        return None                                          # whole numbers alone
    prompts = _prompts(case, seed)
    plain = _Plain(case, seed)
    V = plain.cfg["vocab_size" if case["model"] in QWEN else "vocab"]
    tied = plain.cfg.get("tie_word_embeddings", False) or case["model"] == "gerupel"
    step = 0 if tied else NEXT
    full = [p + [(p[-1] + step * (n + 1)) % V for n in range(case["new"])] for p in prompts]
    ids = torch.zeros(len(full), max(len(s) for s in full), dtype=torch.int64, device="cuda")
    for i, s in enumerate(full):
        ids[i, :len(s)] = torch.tensor(s, device="cuda")
    x = plain.stream(ids)
    if case["kind"] == "score":
        return {"logits": plain.logits(torch.stack([x[i, w] for i, p in enumerate(prompts) for w in _wanted(len(p))]))}
    out = torch.stack([plain.logits(x[i, len(p) - 1:len(p) + case["new"] - 1]).argmax(-1) for i, p in enumerate(prompts)])
    if any(out[i].tolist() != s[len(p):] for i, (p, s) in enumerate(zip(prompts, full))):
        return None                                          # the answers are not the ones assumed above
    return {"first": plain.logits(torch.stack([x[i, len(p) - 1] for i, p in enumerate(prompts)])), "ids": out.cpu(),
            "last": plain.logits(torch.stack([x[i, len(s) - 1] for i, s in enumerate(full)]))}
