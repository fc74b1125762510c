"""What users of the engine have it do, as cases that can be timed and checked.

There are two things a program does with this engine. It *scores* prompts: one ``LLM.step``
takes them whole and gives logits at the places of their last tokens (an answer's tokens behind
a question; the last of them is where a generation would begin). And it *generates*:
``LLM.generate`` takes a batch of prompts to the end, prompt portions beside decode steps as the
scheduler plans them, and the program then scores a sample of what came out, as one does that
keeps the likelihood of its samples. Both are here for GPT-2 at its small, large and XL sizes and
for the other designs with six layer runs at widths 1,024 and 2,048, the sizes of the
repository's own benchmark; bfloat16 is what is served, float32 what is verified with.

Weights are random. Their sizes are those of trained models in one respect that matters: the
token's own embedding stays a good part of the residual stream, so that a router's choices do not
hang on the last bit, and greedy tokens win by a wide margin (``_successor`` says which token
follows which), so that two correct implementations generate the same ones.

``exact`` restates the models in float64 with torch alone.
"""

from __future__ import annotations

import json
import math
import random
import tempfile
from collections.abc import Callable, Iterator
from pathlib import Path

import torch

from ayaka_b200.config.engine import EngineConfig
from ayaka_b200.engine.llm import LLM
from ayaka_b200.engine.runner import StepEntry
from ayaka_b200.sampling.params import SamplingParams

GPT2 = {"small": (768, 12, 12), "large": (1280, 36, 20), "xl": (1600, 48, 25)}
DESIGNS = ("mapuvik", "gagotar", "semadra", "rizitar", "senurax", "kakilorn")
SCORED = 16  # places at the end of a sequence whose logits are asked for
EPS = 1e-5
#: size of the entries of a token's embedding in the residual stream
STREAM = {"mapuvik": 6.0, "gagotar": 6.0, "semadra": 8.0, "rizitar": 10.0, "senurax": 6.0,
          "kakilorn": 3.0}


# ---- the cases -------------------------------------------------------------------------------

def _case(model: str, size: str, use: str, prompts: list[int], new: int = 0,
          dtype: str = "bfloat16", name: str | None = None) -> dict:
    case = {"model": model, "size": size, "use": use, "new": new, "dtype": dtype,
            "prompts": ",".join(str(n) for n in prompts)}
    return case if name is None else {"name": name, **case}


def listed() -> list[dict]:
    ragged = random.Random(7)
    chat = [ragged.randint(16, 896) for _ in range(64)]
    return [
        # the smallest call: one short question, where launches and latency are the time
        _case("gpt2", "small", "score", [21], name="gpt2 small, one question"),
        # the verification path, true 32-bit arithmetic, over a few hundred tokens
        _case("gpt2", "small", "score", [333, 180], dtype="float32", name="gpt2 small, float32"),
        # a batch of chats with prompts of any length: prompt portions beside decode steps
        _case("gpt2", "small", "generate", chat, 64, name="gpt2 small, 64 chats"),
        # eight users of the largest GPT-2, the benchmark's headline: decode steps of 8 rows
        _case("gpt2", "xl", "generate", [480, 301, 444, 512, 390, 505, 467, 350], 64,
              name="gpt2 xl, 8 chats"),
        # two whole contexts through the largest GPT-2
        _case("gpt2", "xl", "score", [1024, 1024], name="gpt2 xl, two contexts"),
        # the other designs, a batch of documents each
        _case("mapuvik", "1024", "score", [1024, 1024, 700, 1300], name="mapuvik, documents"),
        _case("gagotar", "2048", "score", [1024, 777, 247], name="gagotar, documents"),
        _case("semadra", "2048", "score", [1500, 1024, 900, 672], name="semadra, documents"),
        _case("rizitar", "1024", "score", [1024, 1024, 1024, 1024], name="rizitar, documents"),
        # one long document in one piece
        _case("senurax", "2048", "score", [4096], name="senurax, a long document"),
        # many short questions at once
        _case("kakilorn", "2048", "score", [137, 64, 501, 260, 33, 420, 198, 311, 84, 555, 290,
                                            195], name="kakilorn, questions"),
        # chats with one of the designs: decode steps over experts, latent rows and windows
        _case("semadra", "1024", "generate", [128, 300, 97, 210, 256, 180, 77, 240], 64,
              name="semadra, 8 chats"),
    ]


def _spread(rng: random.Random, low: float, high: float) -> int:
    """A whole number between the two, spread over its logarithm."""
    return round(math.exp(rng.uniform(math.log(low), math.log(high))))


def draw(rng: random.Random) -> dict:
    model = rng.choice(("gpt2",) * 3 + DESIGNS)
    if rng.random() < 0.15:  # the verification path runs small things
        size = "small" if model == "gpt2" else "1024"
        return _case(model, size, "score", [_spread(rng, 16, 300) for _ in
                                            range(rng.randint(1, 2))], dtype="float32")
    size = rng.choice(("small", "large", "xl") if model == "gpt2" else ("1024", "2048"))
    if rng.random() < 0.35:
        count = _spread(rng, 1, 32 if size in ("small", "1024") else 8)
        return _case(model, size, "generate", [_spread(rng, 16, 512) for _ in range(count)],
                     rng.randint(16, 48))
    longest = 1024 if model == "gpt2" else 3072
    prompts = [_spread(rng, 16, longest)]
    most = _spread(rng, prompts[0], 2048 if size in ("xl", "2048") else 4096)
    while len(prompts) < 24:
        more = _spread(rng, 16, longest)
        if sum(prompts) + more > most:
            break
        prompts.append(more)
    return _case(model, size, "score", prompts)


def tolerance(case: dict) -> dict:
    """About four times what the engine is off ``exact`` by: 1e-6 in float32, 3e-3 in bfloat16
    (the operands of every product and the cached rows are rounded to it) and more where a
    router may send a row whose two best experts score alike elsewhere."""
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 1e-3}
    routed = case["model"] in ("gagotar", "semadra", "rizitar", "senurax")
    return {"rel": 0.03 if routed else 0.015, "max": 0.9 if routed else 0.5, "differ": 0.01}


# ---- configurations --------------------------------------------------------------------------

def _lengths(case: dict) -> list[int]:
    return [int(n) for n in case["prompts"].split(",")]


def _config(case: dict) -> dict:
    """``config.json`` of the case's model."""
    if case["model"] == "gpt2":
        width, layers, heads = GPT2[case["size"]]
        return {"architectures": ["GPT2LMHeadModel"], "n_layer": layers, "n_embd": width,
                "n_head": heads, "n_inner": 4 * width, "vocab_size": 50257,
                "n_positions": 1024, "layer_norm_epsilon": EPS,
                "activation_function": "gelu_new", "tie_word_embeddings": True}
    width, heads = int(case["size"]), 16
    head, ff = width // heads, 4 * width
    full = {"heads": heads, "kv_heads": heads // 4, "dim": head, "vdim": head,
            "scale": head ** -0.5}
    dense = {"kind": "dense", "ff": ff}
    delta = {"heads": width // 64, "kv_heads": width // 64, "dim": 64, "vdim": 64, "conv": 4}
    channel = {**delta, "decay_rank": 64, "gate_rank": 64}
    memories = max(1, width // 256)

    def moe(expert: dict, router: dict, **more: object) -> dict:
        return {"kind": "moe", "expert": {"ff": ff // 4, **expert},
                "router": {"experts": 16, "top": 2, **router}, **more}

    def model(layers: list[dict], **more: object) -> dict:
        return {"architecture": case["model"].capitalize(), "vocab": 32000, "width": width,
                "norm": {"eps": EPS}, "layers": layers, **more}

    if case["model"] == "mapuvik":
        mixers = [("latent_attention", {
            "heads": heads, "dim": head, "rot_dim": head // 2, "vdim": head,
            "kv_rank": 256 - head // 2, "scale": (head + head // 2) ** -0.5,
            "mask": {"size": 1024}, "rot": {"base": 10000.0, "dims": head // 2}}),
            ("mamba2", {"heads": 2 * width // 64, "vdim": 64, "state": 128, "groups": 1,
                        "conv": 4, "norm_groups": 1}),
            ("mlstm", {"heads": memories, "dim": width // memories, "vdim": width // memories,
                       "gate_cap": 15.0})]
        return model([{"type": kind, "mixer": mixer, "mlp": dense}
                      for _ in range(2) for kind, mixer in mixers])
    if case["model"] == "gagotar":
        left = {**full, "mask": {"size": 384}, "rot": {
            "base": 500000.0, "dims": head,
            "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}}
        right = {"heads": memories, "dim": 128, "vdim": width // memories, "tau": 16.0,
                 "rank": 16}
        return model([{"type": "parallel", "mixer": {"left": left, "right": right},
                       "mlp": moe({"limit": 7.0}, {})}] * 6)
    if case["model"] == "semadra":
        latent = {"heads": heads, "dim": head, "vdim": head, "kv_rank": 256,
                  "q_rank": width // 2, "scale": head ** -0.5, "mask": {"size": 512}}
        experts = moe({}, {"scale": 2.5, "groups": {"count": 4, "keep": 2}},
                      shared={"ff": ff // 4})
        layers = []
        for at in (0, 3):
            layers += [{"type": "latent_attention", "mixer": latent,
                        "mlp": experts if at else dense},
                       {"type": "latent_attention", "mixer": {**latent, "kv_from": at},
                        "mlp": experts},
                       {"type": "attention", "mixer": {**full, "mask": {
                           "size": 512, "keep_first": 64}}, "mlp": experts}]
        return model(layers, embedding={"scale": width ** 0.5}, residual_mult=0.5,
                     token_side={"dim": 64})
    if case["model"] == "rizitar":
        attention = {**full, "mask": {"size": 512, "pool": 16}, "rot": {
            "base": 500000.0, "dims": head,
            "scaling": {"factor": 4.0, "original": 8192, "fast": 16.0, "slow": 1.0}}}
        memory = {"heads": width // 64, "dim": 64, "decay_rank": 64}
        return model([{"type": "attention", "mixer": attention, "mlp": dense},
                      {"type": "attention", "mixer": attention, "mlp": moe({}, {})},
                      {"type": "general_delta", "mixer": memory, "mlp": moe({}, {})}] * 2,
                     embedding={"scale": width ** 0.5}, token_side={"dim": 64})
    if case["model"] == "senurax":
        count = max(1, width // 128)
        retention = {"heads": count, "dim": 64, "vdim": 128,
                     "decay": [1.0 - 2.0 ** -(5 + i % 8) for i in range(count)],
                     "rot": {"dims": 64, "base": 10000.0}}
        left = {**full, "rot": {"dims": head, "base": 500000.0, "scaling": {"factor": 4.0}}}
        experts = moe({}, {"identity": 2, "scale": 1.5})
        ends = {"type": "retention", "mixer": retention, "mlp": dense}
        return model([ends, {"type": "channel_delta", "mixer": channel, "mlp": experts},
                      {"type": "parallel", "mixer": {"left": left, "right": delta},
                       "mlp": experts}, ends],
                     logit_softcap=30.0, loop={"start": 1, "stop": 3, "times": 2})
    latent = {"heads": heads, "dim": head, "rot_dim": head // 2, "vdim": head,
              "q_rank": width // 2, "kv_rank": 256 - head // 2,
              "scale": (head + head // 2) ** -0.5, "rot": {
                  "base": 500000.0, "dims": head // 2,
                  "scaling": {"factor": 8.0, "original": 8192, "fast": 16.0, "slow": 1.0}}}
    parallel = {"left": {**full, "mask": {"size": 512, "keep_first": 64}}, "right": delta,
                "left_scale": 0.5, "right_scale": 0.9}
    return model([{"type": kind, "mixer": mixer, "mlp": dense} for _ in range(2)
                  for kind, mixer in (("latent_attention", latent), ("parallel", parallel),
                                      ("channel_delta", channel))],
                 embedding={"scale": width ** 0.5}, logit_scale=0.5)


def _vocab(config: dict) -> int:
    return config.get("vocab") or config["vocab_size"]


# ---- weights ---------------------------------------------------------------------------------

Spec = tuple[str, tuple[int, ...], float, float]  # name, shape, mean, deviation


def _matrix(name: str, rows: int, cols: int, gain: float = 1.0) -> Spec:
    return name, (rows, cols), 0.0, gain / math.sqrt(cols)


def _around(name: str, size: int, mean: float = 1.0, deviation: float = 0.1) -> Spec:
    return name, (size,), mean, deviation


def _attention_specs(p: str, m: dict, width: int) -> Iterator[Spec]:
    yield _matrix(p + "q", m["heads"] * m["dim"], width)
    yield _matrix(p + "k", m["kv_heads"] * m["dim"], width)
    yield _matrix(p + "v", m["kv_heads"] * m["vdim"], width)
    yield _matrix(p + "o", width, m["heads"] * m["vdim"])


def _delta_specs(p: str, m: dict, width: int) -> Iterator[Spec]:
    inner = m["heads"] * m["vdim"]
    for name, rows in (("q", m["kv_heads"] * m["dim"]), ("k", m["kv_heads"] * m["dim"]),
                       ("v", inner)):
        yield _matrix(p + name, rows, width)
        yield f"{p}{name}.conv", (rows, m["conv"]), 0.0, m["conv"] ** -0.5
    yield _matrix(p + "b", m["heads"], width)
    yield _around(p + "A_log", m["heads"], -1.5, 1.0)
    decays = m["heads"]
    if "decay_rank" in m:
        decays *= m["dim"]
        for name, rank, rows in (("a", m["decay_rank"], decays), ("g", m["gate_rank"], inner)):
            yield _matrix(f"{p}{name}1", rank, width)
            yield _matrix(f"{p}{name}2", rows, rank)
    else:
        yield _matrix(p + "a", decays, width)
        yield _matrix(p + "g", inner, width)
    yield _around(p + "dt_bias", decays, -1.0, 1.0)
    yield _around(p + "norm", m["vdim"])
    yield _matrix(p + "o", width, inner)


def _latent_specs(p: str, m: dict, width: int) -> Iterator[Spec]:
    heads, rank, rot = m["heads"], m["kv_rank"], m.get("rot_dim", 0)
    if "q_rank" in m:
        yield _matrix(p + "dq", m["q_rank"], width)
        yield _around(p + "dq.norm", m["q_rank"])
        yield _matrix(p + "uq", heads * (m["dim"] + rot), m["q_rank"])
    else:
        yield _matrix(p + "q", heads * (m["dim"] + rot), width)
    if m.get("kv_from") is None:
        yield _matrix(p + "dkv", rank + rot, width)
        yield _around(p + "dkv.norm", rank)
    yield _matrix(p + "uk", heads * m["dim"], rank)
    yield _matrix(p + "uv", heads * m["vdim"], rank)
    yield _matrix(p + "o", width, heads * m["vdim"])


def _mixer_specs(design: str, kind: str, p: str, m: dict, width: int) -> Iterator[Spec]:
    if kind == "latent_attention":
        yield from _latent_specs(p, m, width)
        if design == "mapuvik":
            yield _matrix(p + "g", m["heads"] * m["vdim"], width)
        elif design == "kakilorn":
            yield _matrix(p + "g", m["heads"], width)
            yield _around(p + "sink", m["heads"], 0.0, 1.0)
    elif kind == "mamba2":
        inner, bc = m["heads"] * m["vdim"], 2 * m["groups"] * m["state"]
        yield _matrix(p + "in", 2 * inner + bc + m["heads"], width)
        yield p + "conv", (inner + bc, m["conv"]), 0.0, m["conv"] ** -0.5
        yield _around(p + "conv.b", inner + bc, 0.0)
        yield _around(p + "dt_bias", m["heads"], -1.5, 0.9)
        yield _around(p + "A_log", m["heads"], 0.2, 0.7)
        yield _around(p + "D", m["heads"], 1.0, 0.5)
        yield _around(p + "norm", inner)
        yield _matrix(p + "o", width, inner)
    elif kind == "mlstm":
        inner = m["heads"] * m["vdim"]
        for name, rows in (("q", m["heads"] * m["dim"]), ("k", m["heads"] * m["dim"]),
                           ("v", inner), ("g", inner), ("i", m["heads"]), ("f", m["heads"])):
            yield _matrix(p + name, rows, width)
        yield _around(p + "i.b", m["heads"], 0.0, 0.5)
        yield _around(p + "f.b", m["heads"], 2.5, 0.9)
        yield _around(p + "norm", inner)
        yield _matrix(p + "o", width, inner)
    elif kind == "general_delta":
        inner, rank = m["heads"] * m["dim"], m["decay_rank"]
        for name in "rkvga":
            yield _matrix(p + name, inner, width)
        yield _around(p + "a.b", inner, 0.0)
        yield _matrix(p + "w1", rank, width)
        yield _matrix(p + "w2", inner, rank)
        yield _around(p + "w0", inner, 0.0, 1.0)
        yield _around(p + "norm", inner)
        yield _matrix(p + "o", width, inner)
    elif kind == "retention":
        inner = m["heads"] * m["vdim"]
        for name, rows in (("q", m["heads"] * m["dim"]), ("k", m["heads"] * m["dim"]),
                           ("v", inner), ("g", inner)):
            yield _matrix(p + name, rows, width)
        yield _matrix(p + "o", width, inner)
    elif kind == "channel_delta":
        yield from _delta_specs(p, m, width)
    elif kind == "attention" and design == "semadra":
        yield from _attention_specs(p, m, width)
        yield _matrix(p + "g", m["heads"] * m["vdim"], width)
        yield _around(p + "q.norm", m["heads"] * m["dim"])
        yield _around(p + "k.norm", m["kv_heads"] * m["dim"])
    elif kind == "attention":  # rizitar: the values are the keys
        yield from (spec for spec in _attention_specs(p, m, width) if spec[0] != p + "v")
        yield _around(p + "q.norm", m["dim"])
        yield _around(p + "k.norm", m["dim"])
        yield _around(p + "sink", m["heads"], 0.0, 0.5)
    else:
        yield from _side_by_side_specs(design, p, m["left"], m["right"], width)


def _side_by_side_specs(design: str, p: str, left: dict, right: dict,
                        width: int) -> Iterator[Spec]:
    lp, rp = p + "left.", p + "right."
    yield from _attention_specs(lp, left, width)
    q, k = left["heads"] * left["dim"], left["kv_heads"] * left["dim"]
    if design == "kakilorn":
        yield _around(lp + "q.norm", left["dim"])
        yield _around(lp + "k.norm", left["dim"])
        yield _around(lp + "pb", left["heads"], -1.0, 1.0)
    if design != "gagotar":
        yield from _delta_specs(rp, right, width)
    else:
        for name, rows in (("q", q), ("k", k), ("v", left["kv_heads"] * left["vdim"])):
            yield _around(f"{lp}{name}.b", rows, 0.0)
        yield _around(lp + "q.norm", q)
        yield _around(lp + "k.norm", k)
        yield lp + "talk", (left["heads"], left["heads"]), 0.0, 0.3 * left["heads"] ** -0.5
        yield _around(lp + "temp", left["heads"], 1.2, 0.4)
        yield _matrix(lp + "g", left["heads"], width)
        qk, inner = right["heads"] * right["dim"], right["heads"] * right["vdim"]
        for name, rows in (("q", qk), ("k", qk), ("v", inner), ("g", inner)):
            yield _matrix(rp + name, rows, width)
        yield _matrix(rp + "a1", right["rank"], width)
        yield _matrix(rp + "a2", qk, right["rank"])
        yield _around(rp + "a2.b", qk, 3.0, 1.2)
        yield _around(rp + "norm", right["vdim"])
        yield _matrix(rp + "o", width, inner)
    if design != "kakilorn":
        yield _around(p + "left.out", width)
        yield _around(p + "right.out", width)


def _mlp_specs(design: str, p: str, mlp: dict, width: int) -> Iterator[Spec]:
    gated = design in ("gagotar", "semadra", "kakilorn") or \
        (design == "senurax" and mlp["kind"] == "moe")

    def unit(prefix: str, ff: int) -> Iterator[Spec]:
        if gated:
            yield _matrix(prefix + "gate", ff, width)
        yield _matrix(prefix + "up", ff, width)
        yield _matrix(prefix + "down", width, ff)

    if mlp["kind"] == "dense":
        yield from unit(p, mlp["ff"])
        if design == "rizitar":
            yield _around(p + "up.b", mlp["ff"], 0.0)
            yield _around(p + "down.b", width, 0.0)
            yield _around(p + "act", 2, 0.0, 0.5)
        return
    router = mlp["router"]
    outputs = router["experts"] + router.get("identity", 0)
    # (Semadra's routers read the stream as it is: scores that tell experts apart)
    yield _matrix(p + "router", outputs, width, 1.0 / STREAM[design] if design == "semadra" else 2.0)
    if design == "senurax":
        yield _around(p + "correction", outputs, 0.0, 0.2 / outputs)
    for e in range(router["experts"]):
        yield from unit(f"{p}e{e}.", mlp["expert"]["ff"])
    if "shared" in mlp:
        yield from unit(p + "shared.", mlp["shared"]["ff"])


def _specs(config: dict) -> Iterator[Spec]:
    """Every stored tensor of the model, under its checkpoint name."""
    if "n_embd" in config:
        d, inner, t = config["n_embd"], config["n_inner"], "transformer."
        yield t + "wte.weight", (config["vocab_size"], d), 0.0, 0.4
        yield t + "wpe.weight", (config["n_positions"], d), 0.0, 0.1
        small = 0.02 / math.sqrt(2 * config["n_layer"])
        for i in range(config["n_layer"]):
            b = f"{t}h.{i}."
            for ln in ("ln_1", "ln_2"):
                yield _around(f"{b}{ln}.weight", d)
                yield _around(f"{b}{ln}.bias", d, 0.0)
            for name, shape, std in (("attn.c_attn", (d, 3 * d), 0.02),
                                     ("attn.c_proj", (d, d), small),
                                     ("mlp.c_fc", (d, inner), 0.02),
                                     ("mlp.c_proj", (inner, d), small)):
                yield f"{b}{name}.weight", shape, 0.0, std
                yield _around(f"{b}{name}.bias", shape[1], 0.0, 0.02)
        yield _around(t + "ln_f.weight", d)
        yield _around(t + "ln_f.bias", d, 0.0)
        return
    design, width = config["architecture"].lower(), config["width"]
    one = 0.0 if design in ("mapuvik", "semadra") else 1.0  # norms stored as w or as 1 + w
    scale = config.get("embedding", {}).get("scale", 1.0)
    side = config.get("token_side", {}).get("dim", 0)
    yield "embed", (config["vocab"], width), 0.0, STREAM[design] / scale
    if side:
        yield "side.embed", (config["vocab"], side * len(config["layers"])), 0.0, 1.0
    if "loop" in config:
        yield "loop.in", (width, 2 * width), 0.0, 0.1 * width ** -0.5
        yield "loop.step", (config["loop"]["times"], width), 0.0, 0.5
    for index, layer in enumerate(config["layers"]):
        p = f"l{index}."
        yield _around(p + "norm1", width, one)
        if design != "mapuvik":
            yield _around(p + "norm2", width, one)
        if design == "gagotar":
            yield _around(p + "ls1", width, 0.5)
            yield _around(p + "ls2", width, 0.5)
        if design == "rizitar":
            yield _around(p + "norm1b", width)
            yield _around(p + "norm2b", width)
        yield from _mixer_specs(design, layer["type"], p + "mix.", layer["mixer"], width)
        yield from _mlp_specs(design, p + "mlp.", layer["mlp"], width)
        if side:
            yield _matrix(p + "side.gate", side, width)
            yield _matrix(p + "side.proj", width, side)
            yield _around(p + "side.norm", width)
    yield _around("final.norm", width, one)
    if design in ("mapuvik", "gagotar", "senurax"):
        yield "head", (config["vocab"], width), 0.0, 0.0  # filled from the embedding


def _successor(config: dict, token: int) -> int:
    """The greedy token behind ``token``: itself where the head is the token table, else the
    next one."""
    tied = "n_embd" in config or config["architecture"] in ("Semadra", "Rizitar", "Kakilorn")
    return token if tied else (token + 1) % _vocab(config)


def _weights(config: dict, dtype: str, seed: int) -> dict[str, torch.Tensor]:
    generator = torch.Generator("cuda").manual_seed(seed)
    out = {}
    for name, shape, mean, deviation in _specs(config):
        if name == "head":
            value = out["embed"].float().roll(1, 0) * (shape[1] ** -0.5)
        else:
            value = torch.randn(shape, generator=generator, device="cuda")
            value = value.mul_(deviation).add_(mean)
        if name.endswith(".talk"):
            value += torch.eye(shape[0], device="cuda")
        if name == "loop.in":  # a pass begins with the mean of the stream and the embeddings
            value += 0.5 * torch.eye(shape[0], device="cuda").repeat(1, 2)
        if name.endswith(".A_log"):
            value.clamp_(-3.0, 1.5)
        out[name] = value.to(torch.bfloat16) if dtype == "bfloat16" and len(shape) > 1 else value
    return out


def _prompts(case: dict, seed: int) -> list[list[int]]:
    rng = random.Random(seed)
    vocab = _vocab(_config(case))
    return [[rng.randrange(vocab) for _ in range(n)] for n in _lengths(case)]


# ---- a pass ----------------------------------------------------------------------------------

def prepare(case: dict, seed: int) -> dict:
    """An engine with its model, as a program keeps it, and the prompts."""
    config, lengths = _config(case), _lengths(case)
    rows = max(2048, sum(lengths) if case["use"] == "score" else 0)
    with tempfile.TemporaryDirectory() as folder:
        (Path(folder) / "config.json").write_text(json.dumps(config))
        llm = LLM.from_config(
            EngineConfig(model=folder, dtype=case["dtype"], device="cuda:0",
                         kv_reserve_tokens=sum(lengths) + len(lengths) * (case["new"] + 16),
                         max_context=max(lengths) + case["new"] if "n_embd" not in config
                         else None,
                         max_running=len(lengths), max_tokens_per_step=rows,
                         cuda_graph=case["use"] == "generate"),
            tensors=_weights(config, case["dtype"], seed))
    return {"llm": llm, "prompts": _prompts(case, seed), "new": case["new"], "use": case["use"]}


def _score(llm: LLM, sequences: list[list[int]]) -> torch.Tensor:
    entries = [StepEntry(f"scored-{i}", tokens, range(max(0, len(tokens) - SCORED), len(tokens)))
               for i, tokens in enumerate(sequences)]
    logits = llm.step(entries)
    for entry in entries:
        llm.release(entry.request_id)
    return logits


def _sample(lengths: list[int]) -> int:
    """How many of the generated sequences are scored: the first one or two."""
    return 2 if len(lengths) > 1 and sum(lengths[:2]) <= 1900 else 1


def run(state: dict) -> dict:
    llm, prompts = state["llm"], state["prompts"]
    if state["use"] == "score":
        return {"logits": _score(llm, prompts)}
    outputs = llm.generate(prompts, SamplingParams(temperature=0.0, max_tokens=state["new"],
                                                   ignore_eos=True))
    tokens = [list(output.outputs[0].token_ids) for output in outputs]
    count = _sample([len(prompt) for prompt in prompts])
    return {"tokens": torch.tensor(tokens),
            "logits": _score(llm, [prompt + new[:-1] for prompt, new
                                   in zip(prompts[:count], tokens)])}


def work(case: dict) -> dict:
    """Every weight that a step needs once a step, every cached row a decode step reads, the
    logits; two operations a weight and row, and attention's products."""
    config, lengths = _config(case), _lengths(case)
    size = 4 if case["dtype"] == "float32" else 2
    vocab, batch, new = _vocab(config), len(lengths), case["new"]
    gpt2 = "n_embd" in config
    layers = config["n_layer"] if gpt2 else len(config["layers"])
    width = config["n_embd"] if gpt2 else config["width"]
    share = 1.0 if gpt2 else 2.0 / 16  # of a layer's experts that a row meets
    plain = routed = 0
    for name, shape, _, _ in _specs(config):
        if len(shape) < 2 or name.split(".")[-1] == "embed" or "wpe" in name or "wte" in name \
                or name == "head":
            continue
        count = math.prod(shape)
        if ".mlp.e" in name:
            routed += count
        else:
            plain += count
    head = vocab * width
    kept = 2 * layers * width  # entries that attention goes over per key (about)

    def step(rows: int, wanted: int, keys: float) -> tuple[float, float]:
        touched = min(1.0, rows * share) if routed else 0.0
        flops = 2.0 * rows * (plain + routed * share) + 2.0 * wanted * head + \
            2.0 * rows * keys * kept
        return size * (plain + routed * touched + head) + 4.0 * wanted * vocab, flops

    def whole(sequences: list[int]) -> tuple[float, float]:
        rows = sum(sequences)
        keys = sum(n * n / 2 for n in sequences) / rows
        return step(rows, min(SCORED, min(sequences)) * len(sequences), keys)

    if case["use"] == "score":
        nbytes, flops = whole(lengths)
        return {"bytes": nbytes, "flops": flops}
    nbytes, flops = whole(lengths)
    mean = sum(lengths) / batch + new / 2
    a, b = step(batch, batch, mean)
    cached = size * kept * mean * batch if gpt2 else 0.0
    c, d = whole([n + new for n in lengths[:_sample(lengths)]])
    return {"bytes": nbytes + (new - 1) * (a + cached) + c, "flops": flops + (new - 1) * b + d}


# ---- the models in float64 ---------------------------------------------------------------------

Tensor = torch.Tensor
Weights = Callable[[str], Tensor]


def _rms(x: Tensor, weight: Tensor | None = None) -> Tensor:
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS)
    return y if weight is None else y * weight


def _unit(x: Tensor) -> Tensor:
    return x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)


def _silu(x: Tensor) -> Tensor:
    return x * torch.sigmoid(x)


def _gelu(x: Tensor) -> Tensor:
    return torch.nn.functional.gelu(x, approximate="tanh")


def _under(w: Weights, prefix: str) -> Weights:
    return lambda name: w(prefix + name)


def _visible(count: int, size: int = 0, keep: int = 0) -> Tensor:
    i, j = torch.arange(count, device="cuda")[:, None], torch.arange(count, device="cuda")
    return (j <= i) & ((i - j < (size or count)) | (j < keep))


def _softmax(scores: Tensor, seen: Tensor, sink: Tensor | None) -> Tensor:
    scores = scores.masked_fill(~seen, -math.inf)
    if sink is None:
        return torch.softmax(scores, -1)
    column = sink.expand(scores.shape[0], 1)
    return torch.softmax(torch.cat([scores, column], -1), -1)[:, :-1]


def _attend(q: Tensor, k: Tensor, v: Tensor, scale: float, seen: Tensor,
            sink: Tensor | None = None) -> Tensor:
    """``q`` [T, H, d], ``k`` [S, G, d], ``v`` [S, E, e]: H / G heads share a key head."""
    heads = q.shape[1]
    out = []
    for h in range(heads):
        weight = _softmax(q[:, h] @ k[:, h * k.shape[1] // heads].T * scale, seen,
                          None if sink is None else sink[h])
        out.append(weight @ v[:, h * v.shape[1] // heads])
    return torch.stack(out, 1)


def _frequencies(rot: dict) -> tuple[Tensor, float]:
    """The pairs' frequencies and the factor on cosine and sine."""
    dims, scaling = rot["dims"], rot.get("scaling")
    i = torch.arange(dims // 2, dtype=torch.float64, device="cuda")
    f = float(rot["base"]) ** (-2.0 * i / dims)
    if not scaling:
        return f, 1.0
    factor, original = scaling["factor"], scaling.get("original")
    if "low" in scaling:  # by wavelength
        s = (original * f / (2 * math.pi) - scaling["low"]) / (scaling["high"] - scaling["low"])
        s = s.clamp(0.0, 1.0)
        return (1.0 - s) * f / factor + s * f, 1.0
    if original is None:
        return f / factor, 1.0

    def pair(turns: float) -> float:
        return dims * math.log(original / (2 * math.pi * turns)) / (2 * math.log(rot["base"]))

    low = max(math.floor(pair(scaling["fast"])), 0)
    high = min(math.ceil(pair(scaling["slow"])), dims - 1)
    ramp = ((i - low) / max(high - low, 0.001)).clamp(0.0, 1.0)
    return f / factor * ramp + f * (1.0 - ramp), 0.1 * math.log(factor) + 1.0


def _turn(x: Tensor, rot: dict, halves: bool) -> Tensor:
    """``x`` [T, heads, d] turned by the position; pairs are entries half apart or neighbours."""
    f, gain = _frequencies(rot)
    dims = rot["dims"]
    angle = torch.arange(x.shape[0], dtype=torch.float64, device="cuda")[:, None, None] * f
    cos, sin = torch.cos(angle) * gain, torch.sin(angle) * gain
    first = slice(0, dims // 2) if halves else slice(0, dims, 2)
    second = slice(dims // 2, dims) if halves else slice(1, dims, 2)
    out = x.clone()
    out[..., first] = x[..., first] * cos - x[..., second] * sin
    out[..., second] = x[..., second] * cos + x[..., first] * sin
    return out


def _heads(x: Tensor, heads: int) -> Tensor:
    return x.reshape(x.shape[0], heads, -1)


def _memory(q: Tensor, k: Tensor, v: Tensor, g: Tensor) -> Tensor:
    """``S = g S + k v^T``, ``o = S^T q``, row by row; all [T, H, .]."""
    state = torch.zeros(k.shape[1], k.shape[2], v.shape[2], dtype=torch.float64, device="cuda")
    out = torch.empty_like(v)
    for t in range(q.shape[0]):
        state = g[t, :, :, None] * state + k[t, :, :, None] * v[t, :, None, :]
        out[t] = (q[t, :, None, :] @ state)[:, 0]
    return out


def _delta(q: Tensor, k: Tensor, v: Tensor, g: Tensor, write: Callable) -> Tensor:
    """As ``_memory``, with ``write(t, S, g S)`` in the place of ``k v^T``."""
    state = torch.zeros(k.shape[1], k.shape[2], v.shape[2], dtype=torch.float64, device="cuda")
    out = torch.empty_like(v)
    for t in range(q.shape[0]):
        faded = g[t, :, :, None] * state
        state = faded + write(t, state, faded)
        out[t] = (q[t, :, None, :] @ state)[:, 0]
    return out


def _conv(x: Tensor, weight: Tensor) -> Tensor:
    taps = weight.shape[1]
    padded = torch.cat([x.new_zeros(taps - 1, x.shape[1]), x])
    return sum(padded[i:i + x.shape[0]] * weight[:, i] for i in range(taps))


def _gated_delta(h: Tensor, w: Weights, m: dict) -> Tensor:
    heads, kv = m["heads"], m["kv_heads"]
    q, k, v = (_silu(_conv(h @ w(n).T, w(n + ".conv"))) for n in "qkv")
    q = _unit(_heads(q, kv)).repeat_interleave(heads // kv, 1) * m["dim"] ** -0.5
    k = _unit(_heads(k, kv)).repeat_interleave(heads // kv, 1)
    v, beta = _heads(v, heads), torch.sigmoid(h @ w("b").T)
    if "decay_rank" in m:
        raw = _heads((h @ w("a1").T) @ w("a2").T + w("dt_bias"), heads)
        gate = torch.sigmoid((h @ w("g1").T) @ w("g2").T)
    else:
        raw, gate = (h @ w("a").T + w("dt_bias"))[:, :, None], _silu(h @ w("g").T)
    g = torch.exp(-torch.exp(w("A_log"))[None, :, None] * torch.nn.functional.softplus(raw))

    def write(t: int, state: Tensor, faded: Tensor) -> Tensor:
        u = beta[t, :, None, None] * (v[t, :, None, :] - k[t, :, None, :] @ faded)
        return k[t, :, :, None] * u

    out = _delta(q, k, v, g.expand_as(k), write)
    return (_rms(out, w("norm")).flatten(1) * gate) @ w("o").T


def _latent(h: Tensor, c: Tensor, k_turned: Tensor | None, w: Weights, m: dict, q: Tensor,
            sink: Tensor | None = None) -> Tensor:
    """Latent attention from queries [T, H, dim + rot] and the latent rows."""
    count, heads, dim = h.shape[0], m["heads"], m["dim"]
    k = _heads(c @ w("uk").T, heads)
    if k_turned is not None:
        q = torch.cat([q[..., :dim], _turn(q[..., dim:], m["rot"], False)], -1)
        k = torch.cat([k, k_turned.expand(count, heads, -1)], -1)
    seen = _visible(count, m.get("mask", {}).get("size", 0))
    return _attend(q, k, _heads(c @ w("uv").T, heads), m["scale"], seen, sink)


def _mapuvik_mixer(kind: str, h: Tensor, w: Weights, m: dict) -> Tensor:
    heads = m["heads"]
    if kind == "latent_attention":
        down = h @ w("dkv").T
        c = _rms(down[:, :m["kv_rank"]], w("dkv.norm"))
        turned = _turn(down[:, None, m["kv_rank"]:], m["rot"], False)
        out = _latent(h, c, turned, w, m, _heads(h @ w("q").T, heads)).flatten(1)
        return (out * torch.sigmoid(h @ w("g").T)) @ w("o").T
    if kind == "mamba2":
        inner, n, groups = heads * m["vdim"], m["state"], m["groups"]
        z, xbc, dt = (h @ w("in").T).split([inner, inner + 2 * groups * n, heads], 1)
        xbc = _silu(_conv(xbc, w("conv")) + w("conv.b"))
        x = _heads(xbc[:, :inner], heads)
        b, c = (_heads(part, groups).repeat_interleave(heads // groups, 1)
                for part in xbc[:, inner:].chunk(2, 1))
        dt = torch.nn.functional.softplus(dt + w("dt_bias"))
        decay = torch.exp(-torch.exp(w("A_log")) * dt)[:, :, None].expand_as(b)
        y = _memory(c, b * dt[:, :, None], x, decay) + w("D")[:, None] * x
        y = _heads(y.flatten(1) * _silu(z), m["norm_groups"])
        return (_rms(y).flatten(1) * w("norm")) @ w("o").T
    q, k, v = (_heads(h @ w(n).T, heads) for n in "qkv")
    cap = m["gate_cap"]
    i = cap * torch.tanh((h @ w("i").T + w("i.b")) / cap)
    f = torch.nn.functional.logsigmoid(cap * torch.tanh((h @ w("f").T + w("f.b")) / cap))
    top, tops = torch.zeros_like(i[0]), []
    for t in range(h.shape[0]):
        top = torch.maximum(f[t] + top, i[t])
        tops.append(top)
    # sums not divided by exp(top): the gates' cap keeps them within 64 bits; the values'
    # last column of ones makes the normaliser
    sums = _memory(q * m["dim"] ** -0.5, k * torch.exp(i)[:, :, None],
                   torch.cat([v, torch.ones_like(v[..., :1])], -1),
                   torch.exp(f)[:, :, None].expand_as(k))
    below = sums[..., -1:].abs().clamp(min=1.0) + 1e-6 * torch.exp(torch.stack(tops))[:, :, None]
    out = _rms(sums[..., :-1] / below).flatten(1) * w("norm")
    return (out * torch.sigmoid(h @ w("g").T)) @ w("o").T


def _gagotar_mixer(h: Tensor, w: Weights, m: dict) -> Tensor:
    left, right = m["left"], m["right"]
    a, count = _under(w, "left."), h.shape[0]
    heads, kv, dim = left["heads"], left["kv_heads"], left["dim"]
    q = _turn(_heads(_rms(h @ a("q").T + a("q.b"), a("q.norm")), heads), left["rot"], True)
    k = _turn(_heads(_rms(h @ a("k").T + a("k.b"), a("k.norm")), kv), left["rot"], True)
    v = _heads(h @ a("v").T + a("v.b"), kv)
    # the heads' scores mixed by ``talk``: one query per head over all key heads side by side
    factor = (a("talk") * a("temp")).reshape(heads, kv, heads // kv)
    mixed = torch.einsum("hgr,tgrd->thgd", factor,
                         q.reshape(count, kv, heads // kv, dim)).flatten(2)
    block = torch.arange(count, device="cuda") // left["mask"]["size"]
    seen = _visible(count) & (block[:, None] == block)
    y = _attend(mixed, k.flatten(1)[:, None], v, left["scale"], seen)
    y = (y * torch.sigmoid(h @ a("g").T)[:, :, None]).flatten(1) @ a("o").T
    b, heads = _under(w, "right."), right["heads"]
    decay = torch.sigmoid((h @ b("a1").T) @ b("a2").T + b("a2.b")) ** (1.0 / right["tau"])
    z = _memory(_heads(h @ b("q").T, heads) * right["dim"] ** -0.5, _heads(h @ b("k").T, heads),
                _heads(h @ b("v").T, heads), _heads(decay, heads))
    z = (_rms(z, b("norm")).flatten(1) * _silu(h @ b("g").T)) @ b("o").T
    return 0.5 * (_rms(y, w("left.out")) + _rms(z, w("right.out")))


def _semadra_mixer(kind: str, h: Tensor, w: Weights, m: dict, latents: dict,
                   index: int) -> Tensor:
    heads = m["heads"]
    if kind == "latent_attention":
        if m.get("kv_from") is None:
            latents[index] = _rms(h @ w("dkv").T, w("dkv.norm"))
        q = _heads(_rms(h @ w("dq").T, w("dq.norm")) @ w("uq").T, heads)
        return _latent(h, latents[m.get("kv_from", index)], None, w, m, q).flatten(1) @ w("o").T
    q = _heads(_rms(h @ w("q").T, w("q.norm")), heads)
    k = _heads(_rms(h @ w("k").T, w("k.norm")), m["kv_heads"])
    seen = _visible(h.shape[0], m["mask"]["size"], m["mask"]["keep_first"])
    out = _attend(q, k, _heads(h @ w("v").T, m["kv_heads"]), m["scale"], seen).flatten(1)
    return (out * torch.sigmoid(h @ w("g").T)) @ w("o").T


def _rizitar_mixer(kind: str, h: Tensor, w: Weights, m: dict) -> Tensor:
    count, heads = h.shape[0], m["heads"]
    if kind == "attention":
        v = _heads(h @ w("k").T, m["kv_heads"])
        q = _turn(_rms(_heads(h @ w("q").T, heads), w("q.norm")), m["rot"], True)
        k = _turn(_rms(v, w("k.norm")), m["rot"], True)
        size, pool = m["mask"]["size"], m["mask"]["pool"]
        blocks = count // pool

        def pooled(x: Tensor) -> Tensor:
            means = x[:blocks * pool].reshape(blocks, pool, *x.shape[1:]).mean(1)
            return torch.cat([x, means])

        last = torch.arange(blocks, device="cuda") * pool + pool - 1
        far = last <= torch.arange(count, device="cuda")[:, None] - size
        seen = torch.cat([_visible(count, size), far], 1)
        return _attend(q, pooled(k), pooled(v), m["scale"], seen, w("sink")).flatten(1) @ w("o").T
    r, k, v = (_heads(h @ w(n).T, heads) for n in "rkv")
    raw = torch.tanh(h @ w("w1").T) @ w("w2").T + w("w0")
    g = _heads(torch.exp(-math.exp(-0.5) * torch.sigmoid(raw)), heads)
    u = _unit(k)
    au = _heads(torch.sigmoid(h @ w("a").T + w("a.b")), heads) * u

    def write(t: int, state: Tensor, faded: Tensor) -> Tensor:
        return k[t, :, :, None] * v[t, :, None, :] - \
            au[t, :, :, None] * (u[t, :, None, :] @ state)

    out = _rms(_delta(r, k, v, g, write)).flatten(1) * w("norm")
    return (out * torch.sigmoid(h @ w("g").T)) @ w("o").T


def _senurax_mixer(kind: str, h: Tensor, w: Weights, m: dict) -> Tensor:
    if kind == "channel_delta":
        return _gated_delta(h, w, m)
    if kind == "retention":
        heads = m["heads"]
        q, k = (_turn(_heads(h @ w(n).T, heads), m["rot"], True) for n in "qk")
        g = torch.tensor(m["decay"], dtype=torch.float64, device="cuda")[None, :, None]
        out = _memory(q, k * m["dim"] ** -0.5, _heads(h @ w("v").T, heads), g.expand_as(k))
        return (_rms(out).flatten(1) * _silu(h @ w("g").T)) @ w("o").T
    left, a = m["left"], _under(w, "left.")
    q = _turn(_heads(h @ a("q").T, left["heads"]), left["rot"], False)
    k = _turn(_heads(h @ a("k").T, left["kv_heads"]), left["rot"], False)
    y = _attend(q, k, _heads(h @ a("v").T, left["kv_heads"]), left["scale"],
                _visible(h.shape[0])).flatten(1) @ a("o").T
    z = _gated_delta(h, _under(w, "right."), m["right"])
    return 0.5 * (_rms(y, w("left.out")) + _rms(z, w("right.out")))


def _kakilorn_mixer(kind: str, h: Tensor, w: Weights, m: dict) -> Tensor:
    if kind == "channel_delta":
        return _gated_delta(h, w, m)
    if kind == "latent_attention":
        q = _heads(_rms(h @ w("dq").T, w("dq.norm")) @ w("uq").T, m["heads"])
        down = h @ w("dkv").T
        c = _rms(down[:, :m["kv_rank"]], w("dkv.norm"))
        turned = _turn(down[:, None, m["kv_rank"]:], m["rot"], False)
        out = _latent(h, c, turned, w, m, q, w("sink"))
        return (out * torch.sigmoid(h @ w("g").T)[:, :, None]).flatten(1) @ w("o").T
    left, a, count = m["left"], _under(w, "left."), h.shape[0]
    heads, kv = left["heads"], left["kv_heads"]
    q = _rms(_heads(h @ a("q").T, heads), a("q.norm"))
    k = _rms(_heads(h @ a("k").T, kv), a("k.norm"))
    v = _heads(h @ a("v").T, kv)
    seen = _visible(count, left["mask"]["size"], left["mask"]["keep_first"])
    at = torch.arange(count, dtype=torch.float64, device="cuda")
    out = []
    for i in range(heads):
        g = i * kv // heads
        score = q[:, i] @ k[:, g].T * left["scale"] - \
            2.0 ** (-8.0 * (i + 1) / heads) * (at[:, None] - at) + a("pb")[i]
        out.append(torch.sigmoid(score).masked_fill(~seen, 0.0) @ v[:, g])
    y = torch.cat(out, 1) @ a("o").T
    return m["left_scale"] * y + \
        m["right_scale"] * _gated_delta(h, _under(w, "right."), m["right"])


def _mlp(design: str, h: Tensor, w: Weights, mlp: dict) -> Tensor:
    def unit(x: Tensor, u: Weights) -> Tensor:
        up = x @ u("up").T
        if design == "mapuvik":
            return torch.nn.functional.gelu(up) @ u("down").T
        if design == "rizitar" and mlp["kind"] == "dense":
            z, (p, q) = up + u("up.b"), torch.nn.functional.softplus(u("act"))
            inner = torch.where(z > 0, p * z * z, (0.5 + q) * (torch.expm1(z.clamp(max=0)) - z))
            return (inner + 0.5 * z) @ u("down").T + u("down.b")
        if design == "rizitar" or (design == "senurax" and mlp["kind"] == "dense"):
            return torch.relu(up) ** 2 @ u("down").T
        gate = x @ u("gate").T
        if design == "gagotar":
            limit = mlp["expert"]["limit"]
            gate, up = gate.clamp(max=limit), up.clamp(-limit, limit)
            return (gate * torch.sigmoid(1.702 * gate) * (up + 1.0)) @ u("down").T
        return (_silu(gate) * up) @ u("down").T

    if mlp["kind"] == "dense":
        return unit(h, w)
    router = mlp["router"]
    experts, top = router["experts"], router["top"]
    z = h @ w("router").T
    if design == "gagotar":
        chosen = z.topk(top, -1).indices
        share = torch.softmax(z.gather(1, chosen), -1)
    elif design == "semadra":
        s = torch.sigmoid(z)
        grouped = s.reshape(h.shape[0], router["groups"]["count"], -1)
        best = grouped.topk(2, -1).values.sum(-1).topk(router["groups"]["keep"], -1).indices
        kept = torch.zeros(grouped.shape[:2], dtype=torch.bool, device="cuda")
        kept = kept.scatter_(1, best, True)[:, :, None].expand_as(grouped).flatten(1)
        chosen = s.masked_fill(~kept, -1.0).topk(top, -1).indices
        share = s.gather(1, chosen) * router["scale"]
    else:
        s = torch.softmax(z, -1)
        chosen = (s + w("correction") if design == "senurax" else s).topk(top, -1).indices
        share = s.gather(1, chosen)
        if design == "senurax":
            share = share / (share.sum(-1, keepdim=True) + 1e-20) * router["scale"]
    out = torch.zeros_like(h)
    for e in range(z.shape[1]):
        rows, place = (chosen == e).nonzero(as_tuple=True)
        y = h[rows] if e >= experts else unit(h[rows], _under(w, f"e{e}."))
        out[rows] += share[rows, place, None] * y
    return out + unit(h, _under(w, "shared.")) if "shared" in mlp else out


def _gpt2_rows(config: dict, w: Weights, tokens: Tensor) -> Tensor:
    d, heads = config["n_embd"], config["n_head"]
    norm = torch.nn.functional.layer_norm
    x = w("wte.weight")[tokens] + w("wpe.weight")[:tokens.shape[0]]
    seen = _visible(tokens.shape[0])
    for i in range(config["n_layer"]):
        u = _under(w, f"h.{i}.")
        h = norm(x, (d,), u("ln_1.weight"), u("ln_1.bias"), EPS)
        q, k, v = (_heads(part, heads) for part in
                   (h @ u("attn.c_attn.weight") + u("attn.c_attn.bias")).chunk(3, 1))
        y = _attend(q, k, v, (d // heads) ** -0.5, seen).flatten(1)
        x = x + y @ u("attn.c_proj.weight") + u("attn.c_proj.bias")
        h = norm(x, (d,), u("ln_2.weight"), u("ln_2.bias"), EPS)
        h = _gelu(h @ u("mlp.c_fc.weight") + u("mlp.c_fc.bias"))
        x = x + h @ u("mlp.c_proj.weight") + u("mlp.c_proj.bias")
    return norm(x, (d,), w("ln_f.weight"), w("ln_f.bias"), EPS)


def _design_rows(config: dict, w: Weights, tokens: Tensor) -> Tensor:
    design = config["architecture"].lower()
    one = 1.0 if design in ("mapuvik", "semadra") else 0.0
    behind = design in ("semadra", "kakilorn")  # norms on the sublayers' outputs alone
    factor = config.get("residual_mult", 1.0)
    x = x0 = w("embed")[tokens] * config.get("embedding", {}).get("scale", 1.0)
    latents: dict[int, Tensor] = {}
    order = [(i, None) for i in range(len(config["layers"]))]
    if "loop" in config:
        loop = config["loop"]
        again = [(i, n if i == loop["start"] else None) for n in range(loop["times"])
                 for i in range(loop["start"], loop["stop"])]
        order = order[:loop["start"]] + again + order[loop["stop"]:]
    for index, opens in order:
        if opens is not None:
            x = torch.cat([x, x0], 1) @ w("loop.in").T + w("loop.step")[opens]
        layer, u = config["layers"][index], _under(w, f"l{index}.")
        kind, m, mix = layer["type"], layer["mixer"], _under(u, "mix.")

        def mixed(h: Tensor) -> Tensor:
            if design == "mapuvik":
                return _mapuvik_mixer(kind, h, mix, m)
            if design == "gagotar":
                return _gagotar_mixer(h, mix, m)
            if design == "semadra":
                return _semadra_mixer(kind, h, mix, m, latents, index)
            return {"rizitar": _rizitar_mixer, "senurax": _senurax_mixer,
                    "kakilorn": _kakilorn_mixer}[design](kind, h, mix, m)

        ff = _under(u, "mlp.")
        if design == "mapuvik":
            h = _rms(x, one + u("norm1"))
            x = x + mixed(h) + _mlp(design, h, ff, layer["mlp"])
            continue
        if behind:
            x = x + factor * _rms(mixed(x), one + u("norm1"))
            x = x + factor * _rms(_mlp(design, x, ff, layer["mlp"]), one + u("norm2"))
        else:
            def joined(y: Tensor, post: str, scale: str) -> Tensor:
                if design == "rizitar":
                    return _rms(y, u(post))
                return y * u(scale) if design == "gagotar" else y

            x = x + joined(mixed(_rms(x, u("norm1"))), "norm1b", "ls1")
            y = _mlp(design, _rms(x, u("norm2")), ff, layer["mlp"])
            x = x + joined(y, "norm2b", "ls2")
        if "token_side" in config:
            dim = config["token_side"]["dim"]
            e = w("side.embed")[tokens, index * dim:(index + 1) * dim]
            y = (_gelu(x @ u("side.gate").T) * e) @ u("side.proj").T
            x = x + factor * _rms(y, u("side.norm"))
    return _rms(x, one + w("final.norm"))


def _logits(config: dict, weights: dict[str, Tensor], sequence: list[int]) -> Tensor:
    """Logits at the last places of a sequence."""
    tokens = torch.tensor(sequence, device="cuda")
    if "n_embd" in config:
        def w(name: str) -> Tensor:
            return weights["transformer." + name].double()

        return _gpt2_rows(config, w, tokens)[-SCORED:] @ w("wte.weight").T

    def w(name: str) -> Tensor:
        return weights[name].double()

    head = w("head" if "head" in weights else "embed")
    z = _design_rows(config, w, tokens)[-SCORED:] @ head.T * config.get("logit_scale", 1.0)
    cap = config.get("logit_softcap")
    return cap * torch.tanh(z / cap) if cap else z


@torch.no_grad()
def exact(case: dict, seed: int) -> dict:
    config = _config(case)
    weights = _weights(config, case["dtype"], seed)
    prompts = _prompts(case, seed)
    if case["use"] == "score":
        return {"logits": torch.cat([_logits(config, weights, p) for p in prompts])}
    tokens = []
    for prompt in prompts:
        chain = [prompt[-1]]
        for _ in range(case["new"]):
            chain.append(_successor(config, chain[-1]))
        tokens.append(chain[1:])
    count = _sample([len(prompt) for prompt in prompts])
    return {"tokens": torch.tensor(tokens),
            "logits": torch.cat([_logits(config, weights, prompt + new[:-1])
                                 for prompt, new in zip(prompts[:count], tokens)])}
