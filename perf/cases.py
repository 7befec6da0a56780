"""The work that a user of this engine has it do, as cases that can be timed and checked.

A case is one pass of serving through the step function: requests are opened, their prompts run in
steps of at most `portion` tokens (prompt portions beside decoded tokens, as the scheduler packs
them), `new` further tokens are decoded one per step and request, and the requests are closed.  The
pass returns the float32 logits of every request's last prompt token and of every decoded token, and
the tokens the sampler chose from them.  The tokens fed in are given (as in a trace replay), so that
the work of a pass does not depend on rounding.

Weights are N(0, 0.02) matrices and gains near one, rounded to bfloat16, at the layer sizes of
bench.py and of the tests; everything is drawn from the seed on the device.  `exact` is the same pass
in 64-bit torch over whole sequences, written from the designs' formulas.
"""

from __future__ import annotations

import math

import torch
import torch.nn.functional as F

DEVICE = "cuda:0"
PAGE = 16
F64 = torch.float64

# --------------------------------------------------------------------------------- configurations
# (layers, width, heads, kv heads, head size, feed-forward, vocabulary, rope base, eps, tied head, window,
# first windowed layer)
QWEN2 = {
    "7B": (28, 3584, 28, 4, 128, 18944, 152064, 1e6, 1e-6, False, 0, 0),
    "1.5B": (28, 1536, 12, 2, 128, 8960, 151936, 1e6, 1e-6, True, 0, 0),
    "14B": (48, 5120, 40, 8, 128, 13824, 152064, 1e6, 1e-6, False, 0, 0),
    "w2048": (8, 2048, 16, 4, 128, 8192, 32000, 1e4, 1e-6, False, 1024, 0),      # every layer windowed
    "F": (2, 192, 6, 2, 128, 256, 300, 1e5, 1e-6, False, 0, 0),
}
WINDOW, VOCAB = 1024, 32000


def qwen2_config(size, layers):
    full, width, heads, kv, dim, ff, vocab, base, eps, tied, window, first = QWEN2[size]
    return dict(architectures=["Qwen2ForCausalLM"], model_type="qwen2", num_hidden_layers=layers or full,
                hidden_size=width, num_attention_heads=heads, num_key_value_heads=kv, head_dim=dim,
                intermediate_size=ff, vocab_size=vocab, rope_theta=base, rms_norm_eps=eps,
                tie_word_embeddings=tied, max_position_embeddings=32768, use_sliding_window=window > 0,
                sliding_window=window, max_window_layers=first)


def hybrid_config(design, width, layers):
    """The designs beside Qwen2, at the sizes of bench.py's workloads (width 2,048 or 4,096)."""
    wide = width // 2048                    # 1 or 2: heads and feed-forward grow with the width
    heads, kv, dim = 16 * wide, 4 * wide, 128
    ff = 8192 if wide == 1 else 14336
    gqa = {"heads": heads, "kv_heads": kv, "dim": dim, "vdim": dim, "scale": dim ** -0.5}
    config = {"vocab": VOCAB, "width": width, "norm": {"eps": 1e-6}, "architecture": design.capitalize()}
    if design == "metulix":                 # three layers of linear attention, then one of windowed attention
        mlp = {"kind": "dense", "ff": ff}
        linear = {"type": "lightning", "mlp": mlp, "mixer": {
            "heads": heads, "dim": dim, "vdim": dim, "decay": [1.0 - 2.0 ** -(3 + 5 * h / heads) for h in range(heads)]}}
        windowed = {"type": "attention", "mlp": mlp, "mixer": dict(
            gqa, conv=4, rot={"base": 10000.0, "dims": dim}, mask={"size": WINDOW, "keep_first": 4})}
        return dict(config, layers=[windowed if i % 4 == 3 else linear for i in range(layers)])
    if design == "zadepel":                 # latent attention, attention, recurrence, attention
        mlp = {"kind": "dense", "ff": ff}
        latent = {"type": "latent_attention", "mlp": mlp, "mixer": {
            "heads": heads, "dim": dim, "rot_dim": dim // 2, "vdim": dim, "kv_rank": 4 * dim,
            "scale": (dim + dim // 2) ** -0.5, "rot": {"base": 10000.0, "dims": dim // 2}, "mask": {"size": WINDOW}}}
        full = {"type": "attention", "mlp": mlp, "mixer": dict(
            gqa, rot={"base": 250000.0, "dims": dim // 2}, v_mix=True)}
        mingru = {"type": "mingru", "mlp": mlp, "mixer": {"width": 2 * width}}
        return dict(config, layers=[(latent, full, mingru, full)[i % 4] for i in range(layers)])
    if design == "tapalix":                 # latent attention in two forms, routed experts beside a shared one, a loop
        experts, top, groups, keep, eff, shared = (64, 6, 8, 4, 1408, 2816) if wide == 1 else (32, 4, 4, 2, 2048, 4096)
        mlp = {"kind": "moe", "expert": {"ff": eff}, "shared": {"ff": shared}, "router": {
            "experts": experts, "top": top, "scale": 2.5, "groups": {"count": groups, "keep": keep}}}
        rotated = {"type": "latent_attention", "mlp": mlp, "mixer": {
            "heads": heads, "dim": dim, "rot_dim": 64, "vdim": dim, "kv_rank": 512, "scale": (dim + 64) ** -0.5,
            "rot": {"base": 10000.0, "dims": 64,
                    "scaling": {"factor": 4.0, "original": 4096, "fast": 32.0, "slow": 1.0}}}}
        gated = {"type": "latent_attention_2", "mlp": mlp, "mixer": {
            "heads": heads, "dim": dim, "vdim": dim, "kv_rank": 512, "scale": dim ** -0.5}}
        return dict(config, embedding={"scale": 1.0}, logit_scale=1.0, logit_softcap=30.0,
                    loop={"start": 1, "stop": max(layers - 1, 2), "times": 2},
                    layers=[(rotated, gated)[i % 2] for i in range(layers)])
    if design == "kufulix":                 # windowed attention beside a state-space mixer, chunked attention, experts
        experts, identity, top, groups, keep, eff = (32, 4, 4, 6, 4, 1024) if wide == 1 else (16, 2, 2, 3, 2, 2048)
        mlp = {"kind": "moe", "expert": {"ff": eff}, "router": {
            "experts": experts, "identity": identity, "top": top, "groups": {"count": groups, "keep": keep}}}
        mixer = dict(gqa, rot={"base": 10000.0, "dims": dim // 2,
                               "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 2048}})
        parallel = {"type": "parallel", "mlp": mlp, "mixer": {
            "left": dict(mixer, mask={"size": WINDOW}), "left_scale": 0.7, "right_scale": 1.2,
            "right": {"heads": 32 * wide, "vdim": 64, "state": 128, "groups": 1, "conv": 4, "norm_groups": 1}}}
        chunked = {"type": "attention", "mlp": mlp, "mixer": dict(mixer, mask={"size": 2 * WINDOW})}
        order = (parallel, chunked, dict(parallel, weights_of=0), dict(chunked, weights_of=1))
        return dict(config, logit_softcap=30.0, layers=[order[i] if i < 2 else order[2 + i % 2] for i in range(layers)])
    if design == "deginex":                 # four residual streams, capped chunked attention, dense and routed in turn
        dense, experts, top, eff = (6144, 32, 4, 1024) if wide == 1 else (12288, 16, 2, 2048)
        mlps = ({"kind": "dense", "ff": dense},
                {"kind": "moe", "expert": {"ff": eff}, "router": {"experts": experts, "top": top}})
        mixer = dict(gqa, softcap=30.0, mask={"size": 2 * WINDOW})
        return dict(config, streams=4, loop={"start": 1, "stop": max(layers - 1, 2), "times": 2},
                    layers=[{"type": "attention", "mixer": mixer, "mlp": mlps[i % 2]} for i in range(layers)])
    if design == "lanilorn":                # differential, windowed and gated linear attention, squared relu
        rot = {"base": 500000.0, "dims": dim // 2,
               "scaling": {"factor": 8.0, "original": 4096, "fast": 32.0, "slow": 1.0}}
        mixers = {"attention": dict(gqa, mask={"size": WINDOW}, rot=rot),
                  "attention_2": dict(gqa, dim=dim // 2, diff=0.5, q_temp={"coef": 0.1, "every": 4096}),
                  "gla": {"heads": heads, "dim": dim // 2, "vdim": dim, "tau": 16.0}}
        kinds = [("attention_2", "attention", "gla", "attention")[i % 4] for i in range(layers)]
        return dict(config, streams=4, embedding={"scale": 2.0}, logit_scale=0.5, layers=[
            {"type": kind, "mixer": mixers[kind],
             "mlp": None if kind == "gla" else {"kind": "dense", "ff": 9216 * wide}} for kind in kinds])
    raise ValueError(design)


def config_of(case):
    if case["model"] == "qwen2":
        return qwen2_config(case["size"], case["layers"])
    return hybrid_config(case["model"], case["width"], case["layers"])


def vocab_of(case):
    return QWEN2[case["size"]][6] if case["model"] == "qwen2" else VOCAB


def run_order(config):
    """The layers in the order they run; a loop's layers run several times."""
    layers = len(config["layers"])
    loop = config.get("loop")
    if not loop:
        return list(range(layers))
    return (list(range(loop["start"])) + list(range(loop["start"], loop["stop"])) * loop["times"]
            + list(range(loop["stop"], layers)))


# ---------------------------------------------------------------------------------------- tensors
def tensors_of(case):
    """Every tensor of the case's model: (name, shape, how it is drawn, the layer it belongs to or None)."""
    config, out, layer = config_of(case), [], None

    def add(name, *shape, draw="normal"):
        out.append((name, shape, draw, layer))

    if case["model"] == "qwen2":
        c = config
        width, ff, dim = c["hidden_size"], c["intermediate_size"], c["head_dim"]
        add("model.embed_tokens.weight", c["vocab_size"], width)
        add("model.norm.weight", width, draw="gain")
        if not c["tie_word_embeddings"]:
            add("lm_head.weight", c["vocab_size"], width)
        for layer in range(c["num_hidden_layers"]):
            p = f"model.layers.{layer}."
            for name, heads in (("q", c["num_attention_heads"]), ("k", c["num_key_value_heads"]),
                                ("v", c["num_key_value_heads"])):
                add(f"{p}self_attn.{name}_proj.weight", heads * dim, width)
                add(f"{p}self_attn.{name}_proj.bias", heads * dim)
            add(p + "self_attn.o_proj.weight", width, c["num_attention_heads"] * dim)
            add(p + "mlp.gate_proj.weight", ff, width)
            add(p + "mlp.up_proj.weight", ff, width)
            add(p + "mlp.down_proj.weight", width, ff)
            add(p + "input_layernorm.weight", width, draw="gain")
            add(p + "post_attention_layernorm.weight", width, draw="gain")
        return out

    design, width = case["model"], config["width"]
    kufulix = design == "kufulix"
    norm = "normal" if kufulix else "gain"          # Kufulix stores its gains around zero
    with_bias = design in ("tapalix", "deginex")    # layer norms with a bias
    add("embed", VOCAB, width)
    if design in ("metulix", "tapalix", "kufulix"):
        add("head", VOCAB, width)
    if kufulix:
        add("embed.norm", width)
    add("final.norm", width, draw=norm)
    if with_bias:
        add("final.norm.b", width)
    if config.get("loop") and design == "tapalix":
        add("loop.in", width, 2 * width)

    def norms(name):
        add(name, width, draw=norm)
        if with_bias:
            add(name + ".b", width)

    def streams(p, q):
        s = config["streams"]
        add(f"{p}hc{q}.in", s, draw="gain")
        add(f"{p}hc{q}.out", s, draw="gain")
        add(f"{p}hc{q}.mix", s, s, draw="eye")
        if design == "lanilorn":
            add(f"{p}ls{q}", width, draw="gain")

    def gqa(p, m, bias):
        for name, size in (("q", m["heads"] * m["dim"]), ("k", m["kv_heads"] * m["dim"]),
                           ("v", m["kv_heads"] * m["vdim"])):
            add(p + name, size, width)
            if bias:
                add(f"{p}{name}.b", size)
        add(p + "o", width, m["heads"] * m["vdim"])

    for layer, entry in enumerate(config["layers"]):
        if "weights_of" in entry:
            continue
        p, kind, m, mlp = f"l{layer}.", entry["type"], entry["mixer"], entry["mlp"]
        x = p + "mix."
        norms(p + "norm1")
        if design == "zadepel":
            add(p + "norm1b", width, draw="gain")
            add(p + "norm2b", width, draw="gain")
        if config.get("streams"):
            streams(p, 1)
        if kind == "lightning":
            for name, per in (("q", m["dim"]), ("k", m["dim"]), ("v", m["vdim"]), ("g", m["vdim"])):
                add(x + name, m["heads"] * per, width)
            add(x + "o", width, m["heads"] * m["vdim"])
            add(x + "norm", m["heads"] * m["vdim"], draw="gain")
        elif kind in ("latent_attention", "latent_attention_2"):
            turned = m.get("rot_dim", 0)
            add(x + "q", m["heads"] * (m["dim"] + turned), width)
            add(x + "dkv", m["kv_rank"] + turned, width)
            add(x + "dkv.norm", m["kv_rank"], draw="gain")
            add(x + "uk", m["heads"] * m["dim"], m["kv_rank"])
            add(x + "uv", m["heads"] * m["vdim"], m["kv_rank"])
            add(x + "o", width, m["heads"] * m["vdim"])
            if kind == "latent_attention_2":
                add(x + "g", m["heads"] * m["vdim"], width)
        elif kind == "mingru":
            for name in ("z", "x", "g"):
                add(x + name, m["width"], width)
            add(x + "z.b", m["width"])
            add(x + "x.b", m["width"])
            add(x + "o", width, m["width"])
        elif kind == "parallel":
            left, right = m["left"], m["right"]
            inner, shared = right["heads"] * right["vdim"], right["groups"] * right["state"]
            gqa(x + "left.", left, True)
            add(x + "left.q.norm", left["dim"], draw="gain")
            add(x + "left.k.norm", left["dim"], draw="gain")
            add(x + "right.in", 2 * inner + 2 * shared + right["heads"], width)
            add(x + "right.conv", inner + 2 * shared, right["conv"], draw="taps")
            add(x + "right.conv.b", inner + 2 * shared)
            add(x + "right.dt_bias", right["heads"], draw="steps")
            add(x + "right.A_log", right["heads"], draw="rates")
            add(x + "right.D", right["heads"], draw="gain")
            add(x + "right.norm", inner, draw="gain")
            add(x + "right.o", width, inner)
        elif kind == "gla":
            add(x + "q", m["heads"] * m["dim"], width)
            add(x + "k", m["heads"] * m["dim"], width)
            add(x + "v", m["heads"] * m["vdim"], width)
            add(x + "a1", 16, width)
            add(x + "a2", m["heads"] * m["dim"], 16)
            add(x + "a2.b", m["heads"] * m["dim"])
            add(x + "norm", m["vdim"], draw="gain")
            add(x + "g", m["heads"] * m["vdim"], width)
            add(x + "o", width, m["heads"] * m["vdim"])
        elif kind == "attention_2":
            add(x + "q", m["heads"] * 2 * m["dim"], width)
            add(x + "k", m["kv_heads"] * 2 * m["dim"], width)
            add(x + "v", m["kv_heads"] * m["vdim"], width)
            add(x + "g", m["heads"], width)
            add(x + "o", width, m["heads"] * m["vdim"])
            for name in ("lq1", "lk1", "lq2", "lk2"):
                add(x + name, m["dim"])
        elif design == "lanilorn":
            add(x + "q", m["heads"] * m["dim"], width)
            add(x + "k", m["kv_heads"] * m["dim"], width)
            add(x + "q.norm", m["heads"] * m["dim"], draw="gain")
            add(x + "k.norm", m["kv_heads"] * m["dim"], draw="gain")
            add(x + "sink", m["heads"])
            add(x + "g", m["heads"], width)
            add(x + "o", width, m["heads"] * m["dim"])
        else:
            gqa(x, m, design in ("zadepel", "kufulix"))
            if design == "metulix":
                for name, size in (("q", m["heads"] * m["dim"]), ("k", m["kv_heads"] * m["dim"]),
                                   ("v", m["kv_heads"] * m["vdim"])):
                    add(f"{x}{name}.conv", size, m["conv"], draw="taps")
                add(x + "q.norm", m["heads"] * m["dim"], draw="gain")
                add(x + "k.norm", m["kv_heads"] * m["dim"], draw="gain")
                add(x + "talk", m["heads"], m["heads"], draw="eye")
            elif design == "zadepel":
                add(x + "vmix", draw="half")
                add(x + "temp", m["heads"], draw="gain")
            elif design == "kufulix":
                add(x + "g", m["heads"], width)
            elif design == "deginex":
                add(x + "g", m["heads"] * m["vdim"], width)
        if mlp is None:
            continue
        if design != "tapalix":
            norms(p + "norm2")
        if config.get("streams"):
            streams(p, 2)
        x = p + "mlp."
        gated = ("up",) if design in ("kufulix", "lanilorn") else ("gate", "up")
        parts = [(x, mlp["ff"])] if mlp["kind"] == "dense" else \
            [(f"{x}e{e}.", mlp["expert"]["ff"]) for e in range(mlp["router"]["experts"])]
        if mlp.get("shared"):
            parts.append((x + "shared.", mlp["shared"]["ff"]))
        for prefix, inner in parts:
            for name in gated:
                add(prefix + name, inner, width)
                if design == "metulix":
                    add(f"{prefix}{name}.b", inner)
            add(prefix + "down", width, inner)
            if design == "metulix":
                add(prefix + "down.b", width)
        if mlp["kind"] == "moe":
            routed = mlp["router"]["experts"] + mlp["router"].get("identity", 0)
            add(x + "router", routed, width)
            add(*((x + "router.b", routed) if design == "deginex" else (x + "correction", routed)))
    return out


def weights_of(case, seed):
    """The tensors, drawn on the device in bfloat16: the engine gets them as a loaded checkpoint."""
    generator = torch.Generator(device=DEVICE).manual_seed(seed)
    # Models with routed experts get a residual stream that the embedding dominates, as trained ones have: where
    # the first layers' outputs make up most of it, bfloat16 rounding turns every tenth choice of an expert.
    routed, quiet, out = routing(case)[0] > 0, 0.02 / math.sqrt(2 * sum(layer_runs(case).values())), {}
    for name, shape, draw, _ in tensors_of(case):
        t = torch.empty(shape, dtype=torch.bfloat16, device=DEVICE)
        if draw == "taps":
            t.normal_(0.0, 0.5, generator=generator)
        elif draw in ("gain", "half"):
            t.normal_(1.0 if draw == "gain" else 0.5, 0.02, generator=generator)
        elif draw == "rates":        # state-space heads that remember hundreds of tokens beside fast ones
            t.copy_(torch.linspace(-4.0, 0.5, shape[0], device=DEVICE))
        elif draw == "steps":
            t.uniform_(-2.0, 1.0, generator=generator)
        else:
            std = 0.02
            if routed and name == "embed":
                std = 1.0 if case["model"] == "tapalix" else 0.2
            elif routed and name.split(".")[-1] in ("o", "down"):
                std = quiet
            t.normal_(0.0, std, generator=generator)
            if draw == "eye":
                t += torch.eye(shape[0], dtype=torch.bfloat16, device=DEVICE)
        out[name] = t
    return out


# -------------------------------------------------------------------------------- the pass itself
def prompt_lengths(case):
    """Tokens each request brings beyond its cached ones: all alike, or spread from one to `prompt`."""
    n, longest = case["requests"], case["prompt"]
    if not case["ragged"]:
        return [longest] * n
    return [1 + (longest - 1) * (2 * i + 1) // (2 * n) for i in range(n - 1)] + [longest]


def plan_of(case):
    """The steps of a pass, [(request, first token, count, whether its last token's logits are wanted)]:
    requests past their prompt take one token each, the rest of the budget goes to the prompts in order."""
    lengths = prompt_lengths(case)
    total = [n + max(case["new"] - 1, 0) for n in lengths]
    at, steps = [0] * len(lengths), []
    while any(a < t for a, t in zip(at, total)):
        budget, step = case["portion"], []
        for decoding in (True, False):
            for r, n in enumerate(lengths):
                if (at[r] >= n) != decoding or at[r] >= total[r] or budget <= 0:
                    continue
                count = 1 if decoding else min(n - at[r], budget)
                step.append((r, at[r], count, at[r] + count >= n))
                budget -= count
        for r, _, count, _ in step:
            at[r] += count
        steps.append(step)
    return steps


def tokens_of(case, seed):
    """Per request the cached tokens and the ones the pass brings."""
    generator = torch.Generator().manual_seed(seed + 77)
    return [torch.randint(0, vocab_of(case), (case["cached"] + n + max(case["new"] - 1, 0),),
                          generator=generator).tolist() for n in prompt_lengths(case)]


def prepare(case, seed):
    """A loaded model, a runner with its cache and a sampler; where the case says so, contexts that
    earlier requests left in the prefix cache."""
    from from_scratch_inference_engine_b200 import LoadedModel, ModelRunner, SamplingParams, StepEntry
    from from_scratch_inference_engine_b200.config import config_from_dict
    from from_scratch_inference_engine_b200.sampling.sampler import Sampler

    ids, cached, count = tokens_of(case, seed), case["cached"], case["requests"]
    longest = max(map(len, ids))
    model = LoadedModel.from_tensors(config_from_dict(config_of(case)), weights_of(case, seed), case["dtype"],
                                     DEVICE, max_positions=longest + PAGE)
    runner = ModelRunner(model.model, model.runtime, page_size=PAGE, num_pages=count * (longest // PAGE + 2),
                         max_requests=count, enable_prefix_cache=cached > 0,
                         max_step_tokens=max(case["portion"], count, 2048 if cached else 0))
    if cached:
        for r in range(count):
            handle = runner.cache.open(r)
            for start in range(0, cached, 2048):
                runner.step([StepEntry(handle, ids[r][start:min(start + 2048, cached)])])
            runner.cache.register_prefix(handle, ids[r][:cached])
            runner.cache.close(handle)
    steps = [[(r, ids[r][cached + start:cached + start + n], [n - 1] if wanted else [])
              for r, start, n, wanted in step] for step in plan_of(case)]
    rows = sum(bool(want) for step in steps for _, _, want in step)
    # temperature <= 0 is greedy; else top-k and nucleus sampling with a seed per request
    params = [SamplingParams(0.0) if case["sampling"] == "greedy" else SamplingParams(0.8, 40, 0.95, seed=r)
              for r in range(count)]
    return {"runner": runner, "model": model, "sampler": Sampler(DEVICE), "params": params, "steps": steps,
            "entry": StepEntry, "contexts": [row[:cached] for row in ids],
            "logits": torch.empty((rows, vocab_of(case)), dtype=torch.float32, device=DEVICE),
            "tokens": torch.empty(rows, dtype=torch.int32, device=DEVICE)}


def run(state):
    """One pass: open, prompts and decoded tokens step by step with sampling, close."""
    runner, params, row = state["runner"], state["params"], 0
    cache, entry = runner.cache, state["entry"]
    handles = [cache.open(r) for r in range(len(params))]
    for handle, context in zip(handles, state["contexts"]):
        if context:
            cache.acquire_prefix(handle, context)
    drawn = [0] * len(params)
    for step in state["steps"]:
        logits = runner.step([entry(handles[r], tokens, want) for r, tokens, want in step])
        wanted = [r for r, _, want in step if want]
        if not wanted:
            continue
        picked = state["sampler"].sample_async(logits, [params[r] for r in wanted], wanted,
                                               [drawn[r] for r in wanted])
        state["logits"][row:row + len(wanted)].copy_(logits)       # a step's logits live until the next step
        state["tokens"][row:row + len(wanted)].copy_(picked.device)
        row += len(wanted)
        for r in wanted:
            drawn[r] += 1
    for handle in handles:
        cache.close(handle)
    return {"logits": state["logits"], "tokens": state["tokens"]}


# ---------------------------------------------------------------------------------------- 64 bits
def rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def layer_norm(x, w, b, eps):
    x = x - x.mean(-1, keepdim=True)
    x = rms(x, eps) * w
    return x if b is None else x + b


def turn_angles(rot, positions):
    """(cos, sin) [tokens, dims / 2] of a rotation entry; with `scaling` by wavelength or YaRN."""
    dims, base, scaling = int(rot["dims"]), float(rot["base"]), rot.get("scaling")
    freq, magnitude = [base ** (-2.0 * i / dims) for i in range(dims // 2)], 1.0
    if scaling and "low" in scaling:
        for i, f in enumerate(freq):
            turns = scaling["original"] * f / (2 * math.pi)
            t = min(max((turns - scaling["low"]) / (scaling["high"] - scaling["low"]), 0.0), 1.0)
            freq[i] = (1 - t) * f / scaling["factor"] + t * f
    elif scaling:
        def place(turns):
            return dims * math.log(scaling["original"] / (2 * math.pi * turns)) / (2 * math.log(base))
        lo, hi = max(math.floor(place(scaling["fast"])), 0), min(math.ceil(place(scaling["slow"])), dims - 1)
        for i, f in enumerate(freq):
            ramp = min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0)
            freq[i] = f / scaling["factor"] * ramp + f * (1 - ramp)
        magnitude = 0.1 * math.log(scaling["factor"]) + 1.0
    angle = positions.to(F64)[:, None] * torch.tensor(freq, dtype=F64, device=positions.device)
    return torch.cos(angle) * magnitude, torch.sin(angle) * magnitude


def turn(x, rot, interleaved=False):
    """x [batch, tokens, heads, dim]: the first rot.dims columns of a head turned by the token's place."""
    if not rot or not rot["dims"]:
        return x
    dims = int(rot["dims"])
    c, s = (t[None, :, None, :] for t in turn_angles(rot, torch.arange(x.shape[1], device=x.device)))
    out = x.clone()
    pair = (slice(0, dims, 2), slice(1, dims, 2)) if interleaved else (slice(0, dims // 2), slice(dims // 2, dims))
    u, v = x[..., pair[0]], x[..., pair[1]]
    out[..., pair[0]], out[..., pair[1]] = u * c - v * s, v * c + u * s
    return out


def visible(n, mask, chunked=False):
    i = torch.arange(n, device=DEVICE)
    see = i[None, :] <= i[:, None]
    size = (mask or {}).get("size", 0)
    if size and chunked:
        see &= i[:, None] // size == i[None, :] // size
    elif size:
        see &= (i[:, None] - i[None, :] < size) | (i[None, :] < mask.get("keep_first", 0))
    return see


def attend(q, k, v, scale, see, cap=0.0, sink=None, talk=None):
    """q [batch, tokens, heads, dim], k and v [batch, tokens, kv heads, *]; `scale` a number or one per
    head; `sink` a score per head without a value; `talk` mixes the heads' weights."""
    heads, group = q.shape[2], q.shape[2] // k.shape[2]
    out = q.new_empty(q.shape[0], q.shape[1], heads, v.shape[3])
    scale = torch.as_tensor(scale, dtype=F64, device=q.device).expand(heads)
    for b in range(q.shape[0]):
        def weights(h):
            s = (q[b, :, h] @ k[b, :, h // group].T) * scale[h]
            if cap:
                s = cap * torch.tanh(s / cap)
            s = s.masked_fill(~see, -math.inf)
            if sink is not None:
                s = torch.cat([s, sink[h].expand(s.shape[0], 1)], dim=1)
            return torch.softmax(s, dim=1)[:, :see.shape[1]]
        mixed = None if talk is None else torch.einsum("hg,gij->hij", talk, torch.stack([weights(h) for h in range(heads)]))
        for h in range(heads):
            out[b, :, h] = (weights(h) if mixed is None else mixed[h]) @ v[b, :, h // group]
    return out.flatten(2)


def recurrence(q, k, v, decay):
    """S <- decay S + k v^T, o = S^T q, token by token; decay [batch, tokens, heads, dim or 1]."""
    batch, tokens, heads, dim = q.shape
    state, out = q.new_zeros(batch, heads, dim, v.shape[3]), torch.empty_like(v)
    for t in range(tokens):
        state = decay[:, t, :, :, None] * state + k[:, t, :, :, None] * v[:, t, :, None, :]
        out[:, t] = torch.einsum("bhdv,bhd->bhv", state, q[:, t])
    return out


def causal_conv(x, taps):
    """x [batch, tokens, channels], taps [channels, n]; the last tap meets the current token."""
    n = taps.shape[1]
    padded = F.pad(x, (0, 0, n - 1, 0))
    return sum(padded[:, j:j + x.shape[1]] * taps[:, j] for j in range(n))


def choose(z, correction, router, design):
    """The chosen experts of every row and their weights (router outputs z)."""
    if design == "deginex":
        top, ids = torch.topk(z, router["top"], dim=-1)
        return ids, torch.softmax(top, dim=-1)
    s = torch.sigmoid(z) if design == "tapalix" else torch.softmax(z, dim=-1)
    c, groups = s + correction, router["groups"]
    parts = c.view(c.shape[0], groups["count"], -1)
    score = parts.topk(2, dim=-1).values.sum(-1) if design == "tapalix" else parts.max(-1).values
    kept = torch.zeros_like(score, dtype=torch.bool).scatter_(1, score.topk(groups["keep"], dim=-1).indices, True)
    ids = parts.masked_fill(~kept[:, :, None], -math.inf).flatten(1).topk(router["top"], dim=-1).indices
    chosen = s.gather(1, ids)
    return ids, chosen / (chosen.sum(-1, keepdim=True) + 1e-20) * router.get("scale", 1.0)


class Oracle:
    """The designs' formulas over whole sequences in 64 bits; x is [batch, tokens, width]."""

    def __init__(self, case, weights):
        self.case, self.config, self.raw = case, config_of(case), weights
        self.design = case["model"]
        self.eps = self.config["rms_norm_eps"] if self.design == "qwen2" else self.config["norm"]["eps"]
        self.values = None                    # Zadepel: the values of the first layer that shares them

    def w(self, name):
        return self.raw[name].to(F64)

    def lin(self, x, name, bias=False):
        y = x @ self.w(name).T
        return y + self.w(name + ".b") if bias else y

    def heads(self, x, name, count, bias=False):
        return self.lin(x, name, bias).unflatten(-1, (count, -1))

    # ------------------------------------------------------------------------------------- mixers
    def lightning(self, h, p, m):
        q, k, v = (F.silu(self.heads(h, p + name, m["heads"])) for name in "qkv")
        decay = torch.tensor(m["decay"], dtype=F64, device=DEVICE)[None, None, :, None].expand(*q.shape[:3], 1)
        o = rms(recurrence(q, k, v, decay).flatten(2), self.eps) * self.w(p + "norm")
        return self.lin(o * torch.sigmoid(self.lin(h, p + "g")), p + "o")

    def metulix_attention(self, h, p, m):
        def made(name, count):
            y = causal_conv(self.lin(h, p + name), self.w(f"{p}{name}.conv"))
            if name == "v":
                return rms(y.unflatten(-1, (count, -1)), self.eps)
            return turn((rms(y, self.eps) * self.w(f"{p}{name}.norm")).unflatten(-1, (count, -1)), m["rot"], True)
        o = attend(made("q", m["heads"]), made("k", m["kv_heads"]), made("v", m["kv_heads"]), m["scale"],
                   visible(h.shape[1], m["mask"]), talk=self.w(p + "talk"))
        return self.lin(o, p + "o")

    def latent(self, h, p, m):
        heads, dim, rank, turned = m["heads"], m["dim"], m["kv_rank"], m.get("rot_dim", 0)
        q, d = self.heads(h, p + "q", heads), self.lin(h, p + "dkv")
        c = rms(d[..., :rank], self.eps) * self.w(p + "dkv.norm")
        k, v = self.heads(c, p + "uk", heads), self.heads(c, p + "uv", heads)
        if turned:
            inter = self.design == "zadepel"
            q = torch.cat([q[..., :dim], turn(q[..., dim:], m["rot"], inter)], dim=-1)
            kr = turn(d[..., None, rank:], m["rot"], inter).expand(-1, -1, heads, -1)
            k = torch.cat([k, kr], dim=-1)
        o = attend(q, k, v, m["scale"], visible(h.shape[1], m.get("mask")))
        if self.design == "tapalix" and not turned:
            o = o * torch.sigmoid(self.lin(h, p + "g"))
        return self.lin(o, p + "o")

    def zadepel_attention(self, h, p, m):
        q, k = self.heads(h, p + "q", m["heads"], True), self.heads(h, p + "k", m["kv_heads"], True)
        v = self.heads(h, p + "v", m["kv_heads"], True)
        if self.values is None:
            self.values = v
        else:
            mix = self.w(p + "vmix")
            v = (1.0 - mix) * v + mix * self.values
        o = attend(turn(q, m["rot"]), turn(k, m["rot"]), v, m["scale"] * self.w(p + "temp"), visible(h.shape[1], None))
        return self.lin(o, p + "o")

    def mingru(self, h, p, m):
        z, u = torch.sigmoid(self.lin(h, p + "z", True)), self.lin(h, p + "x", True)
        cand = torch.where(u >= 0, u + 0.5, torch.sigmoid(u))
        state, states = torch.zeros_like(z[:, 0]), torch.empty_like(z)
        for t in range(z.shape[1]):
            state = (1.0 - z[:, t]) * state + z[:, t] * cand[:, t]
            states[:, t] = state
        return self.lin(states * F.silu(self.lin(h, p + "g")), p + "o")

    def kufulix_attention(self, h, p, m, normed):
        q, k = self.heads(h, p + "q", m["heads"], True), self.heads(h, p + "k", m["kv_heads"], True)
        v = self.heads(h, p + "v", m["kv_heads"], True)
        if normed:
            q, k = rms(q, self.eps) * self.w(p + "q.norm"), rms(k, self.eps) * self.w(p + "k.norm")
        o = attend(turn(q, m["rot"]), turn(k, m["rot"]), v, m["scale"], visible(h.shape[1], m["mask"], not normed))
        if not normed:
            o = (o.unflatten(-1, (m["heads"], -1)) * torch.sigmoid(self.lin(h, p + "g"))[..., None]).flatten(2)
        return self.lin(o, p + "o")

    def state_space(self, h, p, m):
        heads, n = m["heads"], m["state"]
        inner = heads * m["vdim"]
        z, xbc, dt = self.lin(h, p + "in").split([inner, inner + 2 * n, heads], dim=-1)
        xbc = F.silu(causal_conv(xbc, self.w(p + "conv")) + self.w(p + "conv.b"))
        x, b, c = xbc.split([inner, n, n], dim=-1)
        x = x.unflatten(-1, (heads, -1))
        dt = F.softplus(dt + self.w(p + "dt_bias"))[..., None]
        b, c = (t[:, :, None, :].expand(-1, -1, heads, -1) for t in (b, c))
        y = recurrence(c, b, dt * x, torch.exp(-torch.exp(self.w(p + "A_log"))[None, None, :, None] * dt))
        y = (y + self.w(p + "D")[:, None] * x).flatten(2) * F.silu(z)
        return self.lin(rms(y, self.eps) * self.w(p + "norm"), p + "o")

    def parallel(self, h, p, m):
        return (m["left_scale"] * self.kufulix_attention(h, p + "left.", m["left"], True)
                + m["right_scale"] * self.state_space(h, p + "right.", m["right"]))

    def deginex_attention(self, h, p, m):
        q, k = (rms(self.heads(h, p + name, m[count]), self.eps) for name, count in (("q", "heads"), ("k", "kv_heads")))
        o = attend(q, k, self.heads(h, p + "v", m["kv_heads"]), m["scale"], visible(h.shape[1], m["mask"], True),
                   cap=m["softcap"])
        return self.lin(o * torch.sigmoid(self.lin(h, p + "g")), p + "o")

    def gate_heads(self, o, h, p, m):
        o = o.unflatten(-1, (m["heads"], -1)) * torch.sigmoid(self.lin(h, p + "g"))[..., None]
        return self.lin(o.flatten(2), p + "o")

    def lanilorn_attention(self, h, p, m):
        q, k = self.lin(h, p + "q"), self.lin(h, p + "k")
        v = k.unflatten(-1, (m["kv_heads"], -1))
        q = (rms(q, self.eps) * self.w(p + "q.norm")).unflatten(-1, (m["heads"], -1))
        k = (rms(k, self.eps) * self.w(p + "k.norm")).unflatten(-1, (m["kv_heads"], -1))
        o = attend(turn(q, m["rot"]), turn(k, m["rot"]), v, m["scale"], visible(h.shape[1], m["mask"]),
                   sink=self.w(p + "sink"))
        return self.gate_heads(o, h, p, m)

    def difference(self, h, p, m):
        at = torch.arange(h.shape[1], device=DEVICE, dtype=F64)
        temperature = 1 + m["q_temp"]["coef"] * torch.log(torch.floor((at + 1) / m["q_temp"]["every"]) + 1)
        q = self.heads(h, p + "q", m["heads"]) * temperature[None, :, None, None]
        k, v = self.heads(h, p + "k", m["kv_heads"]), self.heads(h, p + "v", m["kv_heads"])
        see, dim = visible(h.shape[1], None), m["dim"]
        o1, o2 = (attend(q[..., s], k[..., s], v, m["scale"], see) for s in (slice(0, dim), slice(dim, 2 * dim)))
        lam = (torch.exp(self.w(p + "lq1") @ self.w(p + "lk1")) - torch.exp(self.w(p + "lq2") @ self.w(p + "lk2"))
               + m["diff"])
        o = rms((o1 - lam * o2).unflatten(-1, (m["heads"], -1)), self.eps) * (1 - m["diff"])
        return self.gate_heads(o.flatten(2), h, p, m)

    def gated_linear(self, h, p, m):
        q = self.heads(h, p + "q", m["heads"]) * m["dim"] ** -0.5
        k, v = self.heads(h, p + "k", m["heads"]), self.heads(h, p + "v", m["heads"])
        z = self.lin(h, p + "a1") @ self.w(p + "a2").T + self.w(p + "a2.b")
        decay = torch.exp(F.logsigmoid(z) / m["tau"]).unflatten(-1, (m["heads"], -1))
        o = (rms(recurrence(q, k, v, decay), self.eps) * self.w(p + "norm")).flatten(2)
        return self.lin(o * F.silu(self.lin(h, p + "g")), p + "o")

    def mixer(self, h, p, layer):
        kind, m = layer["type"], layer["mixer"]
        if kind == "attention":
            of = {"metulix": self.metulix_attention, "zadepel": self.zadepel_attention,
                  "deginex": self.deginex_attention, "lanilorn": self.lanilorn_attention}.get(self.design)
            return self.kufulix_attention(h, p, m, False) if of is None else of(h, p, m)
        return {"lightning": self.lightning, "latent_attention": self.latent, "latent_attention_2": self.latent,
                "mingru": self.mingru, "parallel": self.parallel, "attention_2": self.difference,
                "gla": self.gated_linear}[kind](h, p, m)

    # ------------------------------------------------------------------------------- feed-forward
    def dense(self, h, p):
        bias = self.design == "metulix"
        up = self.lin(h, p + "up", bias)
        if self.design in ("kufulix", "lanilorn"):
            return self.lin(torch.relu(up) ** 2, p + "down")
        gate = self.lin(h, p + "gate", bias)
        gate = F.gelu(gate, approximate="tanh") if self.design == "zadepel" else F.silu(gate)
        return self.lin(gate * up, p + "down", bias)

    def feed_forward(self, h, p, mlp):
        if mlp["kind"] == "dense":
            return self.dense(h, p)
        shape, router = h.shape, mlp["router"]
        rows = h.flatten(0, 1)
        z = self.lin(rows, p + "router")
        if self.design == "deginex":
            z = z + self.w(p + "router.b")
        ids, share = choose(z, self.w(p + "correction") if self.design != "deginex" else None, router, self.design)
        out = self.dense(rows, p + "shared.") if mlp.get("shared") else torch.zeros_like(rows)
        for e in range(z.shape[1]):
            at, place = (ids == e).nonzero(as_tuple=True)
            if len(at):
                y = self.dense(rows[at], f"{p}e{e}.") if e < router["experts"] else rows[at]
                out.index_add_(0, at, y * share[at, place][:, None])
        return out.view(shape)

    # -------------------------------------------------------------------------------------- model
    def qwen2_layer(self, x, index):
        c, p = self.config, f"model.layers.{index}."

        def project(name, heads):
            y = self.lin(h, f"{p}self_attn.{name}_proj.weight") + self.w(f"{p}self_attn.{name}_proj.bias")
            return y.unflatten(-1, (heads, -1))
        h = rms(x, self.eps) * self.w(p + "input_layernorm.weight")
        rot = {"base": c["rope_theta"], "dims": c["head_dim"]}
        kv = c["num_key_value_heads"]
        window = c["sliding_window"] if c["use_sliding_window"] and index >= c["max_window_layers"] else 0
        o = attend(turn(project("q", c["num_attention_heads"]), rot), turn(project("k", kv), rot), project("v", kv),
                   c["head_dim"] ** -0.5, visible(x.shape[1], {"size": window}))
        x = x + self.lin(o, p + "self_attn.o_proj.weight")
        h = rms(x, self.eps) * self.w(p + "post_attention_layernorm.weight")
        gate, up = p + "mlp.gate_proj.weight", p + "mlp.up_proj.weight"
        rows = [self.lin(F.silu(self.lin(part, gate)) * self.lin(part, up), p + "mlp.down_proj.weight")
                for part in h.split(1)]
        return x + torch.cat(rows)

    def qwen2(self, ids, want):
        x = self.w("model.embed_tokens.weight")[ids]
        for index in range(self.config["num_hidden_layers"]):
            x = self.qwen2_layer(x, index)
        head = "model.embed_tokens.weight" if self.config["tie_word_embeddings"] else "lm_head.weight"
        return self.lin(rms(x[want], self.eps) * self.w("model.norm.weight"), head)

    def sublayer(self, x, p, q, f):
        """Streams [streams, batch, tokens, width]: a sublayer reads a weighted sum, every stream changes."""
        u = torch.einsum("s,sbtc->btc", self.w(f"{p}hc{q}.in"), x)
        if self.design == "lanilorn":
            y = f(rms(u, self.eps) * self.w(f"{p}norm{q}")) * self.w(f"{p}ls{q}")
        else:
            y = f(layer_norm(u, self.w(f"{p}norm{q}"), self.w(f"{p}norm{q}.b"), self.eps))
        return torch.einsum("rs,rbtc->sbtc", self.w(f"{p}hc{q}.mix"), x) + self.w(f"{p}hc{q}.out").view(-1, 1, 1, 1) * y

    def layer(self, x, p, layer):
        design, eps, mlp = self.design, self.eps, layer["mlp"]
        if design == "metulix":
            x = x + layer_norm(self.mixer(x, p + "mix.", layer), self.w(p + "norm1"), None, eps)
            return x + layer_norm(self.feed_forward(x, p + "mlp.", mlp), self.w(p + "norm2"), None, eps)
        if design == "zadepel":
            y = self.mixer(rms(x, eps) * self.w(p + "norm1"), p + "mix.", layer)
            x = x + rms(y, eps) * self.w(p + "norm1b")
            y = self.feed_forward(rms(x, eps) * self.w(p + "norm2"), p + "mlp.", mlp)
            return x + rms(y, eps) * self.w(p + "norm2b")
        if design == "tapalix":
            h = layer_norm(x, self.w(p + "norm1"), self.w(p + "norm1.b"), eps)
            return x + self.mixer(h, p + "mix.", layer) + self.feed_forward(h, p + "mlp.", mlp)
        if design == "kufulix":
            x = x + self.mixer(rms(x, eps) * (1 + self.w(p + "norm1")), p + "mix.", layer)
            return x + self.feed_forward(rms(x, eps) * (1 + self.w(p + "norm2")), p + "mlp.", mlp)
        x = self.sublayer(x, p, 1, lambda h: self.mixer(h, p + "mix.", layer))
        return x if mlp is None else self.sublayer(x, p, 2, lambda h: self.feed_forward(h, p + "mlp.", mlp))

    def logits(self, ids, want):
        """ids [batch, tokens]; want [batch, tokens] bool: logits of those places, request by request."""
        if self.design == "qwen2":
            return self.qwen2(ids, want)
        config = self.config
        x = self.w("embed")[ids] * (config.get("embedding") or {}).get("scale", 1.0)
        if self.design == "kufulix":
            x = rms(x, self.eps) * (1 + self.w("embed.norm"))
        start, x0 = (config.get("loop") or {}).get("start", -1), x
        if config.get("streams"):
            x = x.expand(config["streams"], *x.shape)
        for index in run_order(config):
            if self.design == "tapalix" and index == start:
                x = self.lin(torch.cat([x, x0], dim=-1), "loop.in")
            layer = config["layers"][index]
            x = self.layer(x, f"l{layer.get('weights_of', index)}.", layer)
        x = x.sum(0) if config.get("streams") else x
        x = x[want]
        if self.design in ("metulix", "tapalix", "deginex"):
            bias = None if self.design == "metulix" else self.w("final.norm.b")
            x = layer_norm(x, self.w("final.norm"), bias, self.eps)
        else:
            x = rms(x, self.eps) * (self.w("final.norm") + (1 if self.design == "kufulix" else 0))
        y = self.lin(x, "head" if "head" in self.raw else "embed") * config.get("logit_scale", 1.0)
        cap = config.get("logit_softcap", 0.0)
        return cap * torch.tanh(y / cap) if cap else y


def exact(case, seed):
    """The pass's logits in 64 bits and the tokens greedy sampling takes from them (a nucleus draw has
    no such value); None where this would take over about 20 seconds (64-bit products run at about
    30 TFLOP/s)."""
    lengths = prompt_lengths(case)
    ids = tokens_of(case, seed)
    longest = max(map(len, ids))
    if 2.0 * len(ids) * longest * active_numbers(case) > 6e14:
        return None
    padded = torch.zeros((len(ids), longest), dtype=torch.long)
    want = torch.zeros((len(ids), longest), dtype=torch.bool)
    for r, row in enumerate(ids):
        padded[r, :len(row)] = torch.tensor(row)
        want[r, case["cached"] + lengths[r] - 1:len(row)] = True
    rows = Oracle(case, weights_of(case, seed)).logits(padded.to(DEVICE), want.to(DEVICE))
    # rows come request by request; the pass returns them step by step
    first = [0]
    for r, row in enumerate(ids):
        first.append(first[-1] + len(row) - (case["cached"] + lengths[r] - 1))
    given, order = [0] * len(ids), []
    for step in plan_of(case):
        for r, _, _, wanted in step:
            if wanted:
                order.append(first[r] + given[r])
                given[r] += 1
    logits = rows[torch.tensor(order, device=DEVICE)]
    return {"logits": logits, "tokens": logits.argmax(-1) if case["sampling"] == "greedy" else None}


# ------------------------------------------------------------------------------- work, tolerances
def layer_runs(case):
    """How often each layer's tensors run in one step."""
    config = config_of(case)
    if case["model"] == "qwen2":
        return {i: 1 for i in range(config["num_hidden_layers"])}
    runs = {}
    for i in run_order(config):
        source = config["layers"][i].get("weights_of", i)
        runs[source] = runs.get(source, 0) + 1
    return runs


def routing(case):
    """(experts, chosen per token) of the routed feed-forwards, else (0, 0)."""
    if case["model"] == "qwen2":
        return 0, 0
    for layer in config_of(case)["layers"]:
        if layer["mlp"] and layer["mlp"]["kind"] == "moe":
            router = layer["mlp"]["router"]
            return router["experts"], router["top"] * router["experts"] / (router["experts"] + router.get("identity", 0))
    return 0, 0


def matrix_numbers(case):
    """(numbers of the head, numbers of all other matrices, of the experts' matrices) and the same of the
    last two weighted with how often their layer runs."""
    runs, head, plain, routed, plain_run, routed_run = layer_runs(case), 0, 0, 0, 0, 0
    for name, shape, _, layer in tensors_of(case):
        if len(shape) < 2:
            continue
        numbers = math.prod(shape)
        if layer is None:
            if "embed" not in name and name != "loop.in":
                head = numbers
            elif name == "loop.in":
                plain, plain_run = plain + numbers, plain_run + 2 * numbers
            continue
        if ".mlp.e" in name:
            routed, routed_run = routed + numbers, routed_run + numbers * runs[layer]
        else:
            plain, plain_run = plain + numbers, plain_run + numbers * runs[layer]
    if not head:
        head = math.prod(tensors_of(case)[0][1])
    return head, plain, routed, plain_run, routed_run


def active_numbers(case):
    """Matrix numbers that a token's path multiplies, without the head."""
    _, _, _, plain, routed = matrix_numbers(case)
    experts, top = routing(case)
    return plain + (routed * top / experts if experts else 0)


def mixers(case):
    """Per mixer run: (numbers of a token's cache row, multiply-adds per query and key, keys a query sees at
    most, numbers of state)."""
    config, out = config_of(case), []
    if case["model"] == "qwen2":
        c = config
        for i in range(c["num_hidden_layers"]):
            window = c["sliding_window"] if c["use_sliding_window"] and i >= c["max_window_layers"] else 1 << 30
            out.append((2 * c["num_key_value_heads"] * c["head_dim"], 2 * c["num_attention_heads"] * c["head_dim"], window, 0))
        return out
    for i in run_order(config):
        layer = config["layers"][i]
        kinds = [("attention", layer["mixer"]["left"]), ("state", layer["mixer"]["right"])] \
            if layer["type"] == "parallel" else [(layer["type"], layer["mixer"])]
        for kind, m in kinds:
            size = (m.get("mask") or {}).get("size", 1 << 30)
            if kind in ("lightning", "gla"):
                out.append((0, 0, 0, m["heads"] * m["dim"] * m["vdim"]))
            elif kind == "state":
                out.append((0, 0, 0, m["heads"] * m["state"] * m["vdim"]))
            elif kind == "mingru":
                out.append((0, 0, 0, m["width"]))
            elif kind.startswith("latent"):
                turned = m.get("rot_dim", 0)
                out.append((m["kv_rank"] + turned, m["heads"] * (m["dim"] + turned + m["vdim"]), size, 0))
            elif kind == "attention_2":
                out.append((m["kv_heads"] * (2 * m["dim"] + m["vdim"]), m["heads"] * 2 * (m["dim"] + m["vdim"]), size, 0))
            else:
                out.append((m["kv_heads"] * (m["dim"] + m["vdim"]), m["heads"] * (m["dim"] + m["vdim"]), size, 0))
    return out


def work(case):
    """A step reads the matrices its tokens meet once and the live requests' keys, values and state, and writes
    what it adds to them and its logits; a step's matrices do not stay on the chip until the next."""
    number = 2 if case["dtype"] == "bfloat16" else 4
    head, plain, routed, plain_run, routed_run = matrix_numbers(case)
    experts, top = routing(case)
    vocab, parts = vocab_of(case), mixers(case)
    at, nbytes, flops = [case["cached"]] * case["requests"], 0.0, 0.0
    for step in plan_of(case):
        tokens = sum(n for _, _, n, _ in step)
        rows = sum(wanted for *_, wanted in step)
        met = 1.0 - (1.0 - top / experts) ** tokens if experts else 0.0
        nbytes += number * (plain + routed * met + (head if rows else 0)) + 4.0 * rows * vocab
        flops += 2.0 * tokens * active_numbers(case) + 2.0 * rows * head
        for r, _, n, _ in step:
            end = at[r] + n
            for row, per_key, sees, state in parts:
                seen = sum(min(p + 1, sees) for p in range(at[r], end)) if sees else 0
                nbytes += number * row * (min(end, sees + n) if sees else 0) + 8.0 * state
                flops += 2.0 * per_key * seen + 4.0 * state * n
            at[r] = end
    return {"bytes": nbytes, "flops": flops}


# About four times what this code shows against 64 bits: (logits' 2-norm, largest difference over the logits'
# root mean square or None, share of tokens that a rounding may turn).  In bfloat16 a choice of experts that
# is close turns with the rounding and changes its row of logits: there only the 2-norm is bounded.
TOLERANCE = {
    ("qwen2", "bfloat16"): (0.16, 0.95, 0.4), ("metulix", "bfloat16"): (4e-2, 0.2, 0.3),
    ("zadepel", "bfloat16"): (4.5e-2, 0.25, 0.3), ("lanilorn", "bfloat16"): (4e-2, 0.2, 0.3),
    ("tapalix", "bfloat16"): (0.2, None, 0.4), ("kufulix", "bfloat16"): (0.3, None, 0.4),
    ("deginex", "bfloat16"): (0.15, None, 0.4), ("qwen2", "float32"): (2e-5, 2e-4, 0.05),
}


def tolerance(case):
    rel, largest, differ = TOLERANCE.get((case["model"], case["dtype"]), (1.5e-5, 1e-4, 0.05))
    return {"rel": rel, "differ": differ, **({} if largest is None else {"max": largest})}


# ------------------------------------------------------------------------------------------ cases
def case_of(name, model, size, layers, dtype="bfloat16", requests=1, cached=0, prompt=1, ragged=False, new=0,
            portion=2048, sampling="greedy"):
    """`size`: a Qwen2 size, or the width of another design; `layers` 0: the size's own depth."""
    case = {"model": model, "layers": layers, "dtype": dtype, "requests": requests, "cached": cached,
            "prompt": prompt, "ragged": ragged, "new": new, "portion": portion, "sampling": sampling}
    case["size" if model == "qwen2" else "width"] = size
    return dict({"name": name}, **case) if name else case


def listed():
    return [
        # one user's short question to a small model: latency and launches
        case_of("chat-1.5b", "qwen2", "1.5B", 0, prompt=45, new=8, sampling="nucleus"),
        # the benchmark's headline: eight long conversations at the 7B shape, every one continued
        case_of("decode-7b-b8", "qwen2", "7B", 0, requests=8, cached=4096, prompt=1, new=16),
        # a loaded server: 64 conversations
        case_of("decode-7b-b64", "qwen2", "7B", 0, requests=64, cached=1024, prompt=1, new=8),
        # a long prompt's time to its first token
        case_of("prefill-7b", "qwen2", "7B", 0, prompt=2048),
        # continuous batching: prompts of all lengths in portions beside decoded tokens, nucleus sampling
        case_of("serving-1.5b", "qwen2", "1.5B", 0, requests=24, prompt=700, ragged=True, new=12, portion=512,
                sampling="nucleus"),
        # the true 32-bit path, prompts and decoded tokens
        case_of("fp32-1.5b", "qwen2", "1.5B", 0, dtype="float32", requests=3, prompt=1000, ragged=True, new=8),
        # the other designs: prompts, then decoded tokens
        case_of("metulix", "metulix", 2048, 8, requests=4, prompt=901, ragged=True, new=16),
        case_of("zadepel", "zadepel", 2048, 8, requests=1, prompt=2048, new=8),
        case_of("tapalix", "tapalix", 2048, 4, requests=8, prompt=400, ragged=True, new=16),
        case_of("kufulix", "kufulix", 4096, 4, requests=1, prompt=2048, new=8),
        case_of("deginex", "deginex", 2048, 4, requests=6, prompt=517, ragged=True, new=16, portion=512),
        case_of("lanilorn", "lanilorn", 2048, 4, requests=2, prompt=1500, ragged=True, new=16),
    ]


def cost(case):
    """Seconds of a pass, roughly: what orders cases by size."""
    w = work(case)
    return w["bytes"] / 6e12 + w["flops"] / (1.2e15 if case["dtype"] == "bfloat16" else 35e12)


def draw(rng):
    def spread(low, high):
        return min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high + 1))))))
    dtype = "float32" if rng.random() < 0.25 else "bfloat16"
    model = "qwen2" if rng.random() < 0.5 else rng.choice(["metulix", "zadepel", "tapalix", "kufulix", "deginex", "lanilorn"])
    if model == "qwen2":
        size = rng.choice(["7B", "7B", "1.5B", "1.5B", "14B", "w2048", "F"])
        layers = spread(2, min(QWEN2[size][0], 28))
    else:
        size, layers = rng.choice([2048, 2048, 4096]), rng.randint(3, 8)
    requests = spread(1, 64)
    prompt = spread(1, max(1, min(4096 // requests, 2048)))
    cached = PAGE * spread(1, max(1, 16384 // requests // PAGE)) if model == "qwen2" and rng.random() < 0.4 else 0
    if cached and QWEN2[size][10]:          # windowed layers share no prefixes
        cached = 0
    case = case_of(None, model, size, layers, dtype, requests, cached, prompt, rng.random() < 0.5, spread(1, 16),
                   rng.choice([2048, 512, spread(100, 2000)]), rng.choice(["greedy", "nucleus"]))
    largest = max(cost(c) for c in listed())
    while cost(case) > largest:
        case["prompt"], case["new"] = (case["prompt"] + 1) // 2, (case["new"] + 1) // 2
        case["requests"] = max(1, case["requests"] * 3 // 4)
    return case
