"""The work that users have this framework do, as cases that can be timed and whose results can be checked.

Three ways into the framework, over the decoders it serves:

* ``prompt``: the step function (``ModelRunner.step``) takes a prompt, whole or in portions, and gives the logits of its last
  token: time to first token;
* ``decode``: requests with a filled cache go on by a few tokens through captured decode steps (``DecodeGraphs``), each step
  queued behind the one before it as ``Engine.step`` queues them: the time between tokens;
* ``generate``: ``Engine.generate``, from prompts to all new tokens: admission, portions mixed with decoded tokens, captured
  steps, sampling.

Model sizes are those of the repository's own configurations (the 8B, 4B and 32B shapes of the Qwen3 decoder, its tiny model
with windowed layers, and the layer sizes of ``bench.py``'s comparison of designs for the Figalix and Damilix decoders), with
as many layers as keep a case's preparation short.  Weights are random but behave like trained ones where that matters to the
outcome: the layers' outputs are small beside the stream, a model is fairly sure of its next token, and a router's choice of
experts is not a matter of rounding.

``exact`` restates the decoders in plain 64-bit torch, whole sequences at a time, without the framework's code.
"""
import hashlib
import math

import numpy as np
import torch

import kirai_b200
from kirai_b200.engine.batch import StepEntry
from kirai_b200.engine.graphs import DecodeGraphs
from kirai_b200.engine.runner import ModelRunner
from kirai_b200.registry import config_from_dict
from kirai_b200.weights import loader

F64 = torch.float64
DEVICE = "cuda:0"
DECODE_STEPS = 8       # steps of one pass of a decode case
STEP_TOKENS = 2048     # tokens of one step, at most (the engine's default)
PAGE = 16

# ---------------------------------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------------------------------


def listed():
    return [
        # the smallest call: a tiny model in true 32-bit with windowed layers, four short prompts and twelve new tokens each;
        # nothing but launches and the host's own time
        {"name": "generate-tiny-f32", "kind": "generate", "model": "tiny", "layers": 3, "dtype": "float32", "requests": 4,
         "shortest": 3, "longest": 40, "new": 12, "portion": 0},
        # a short question to the 8B shape: time to its first token
        {"name": "prompt-8b-37", "kind": "prompt", "model": "8b", "layers": 36, "dtype": "bfloat16", "requests": 1,
         "shortest": 37, "longest": 37, "portion": 2048},
        # the headline prompt: 2,048 tokens on the 8B shape
        {"name": "prompt-8b-2048", "kind": "prompt", "model": "8b", "layers": 36, "dtype": "bfloat16", "requests": 1,
         "shortest": 2048, "longest": 2048, "portion": 2048},
        # a long document on the 32B shape's layers, in portions of 2,048 tokens
        {"name": "prompt-32b-8064", "kind": "prompt", "model": "32b", "layers": 4, "dtype": "bfloat16", "requests": 1,
         "shortest": 8064, "longest": 8064, "portion": 2048},
        # one user's conversation: the 8B shape, one request at a context of about 4,096
        {"name": "decode-8b-1", "kind": "decode", "model": "8b", "layers": 36, "dtype": "bfloat16", "requests": 1,
         "shortest": 4080, "longest": 4080, "temperature": 0.0, "top_p": 1.0},
        # the headline batch: eight requests at ragged contexts
        {"name": "decode-8b-8", "kind": "decode", "model": "8b", "layers": 36, "dtype": "bfloat16", "requests": 8,
         "shortest": 2317, "longest": 4080, "temperature": 0.0, "top_p": 1.0},
        # a full server: 64 requests of all lengths, sampled at a temperature inside a nucleus
        {"name": "decode-4b-64-sampled", "kind": "decode", "model": "4b", "layers": 12, "dtype": "bfloat16", "requests": 64,
         "shortest": 131, "longest": 1500, "temperature": 0.7, "top_p": 0.9},
        # requests of all lengths served together: portions of 512 tokens mixed with decoded tokens
        {"name": "serve-4b-16", "kind": "generate", "model": "4b", "layers": 12, "dtype": "bfloat16", "requests": 16,
         "shortest": 129, "longest": 1777, "new": 24, "portion": 512},
        # the true 32-bit path: what a user runs who checks results or a conversion, a prompt at the 4B shape's layers
        {"name": "prompt-4b-f32-515", "kind": "prompt", "model": "4b", "layers": 6, "dtype": "float32", "requests": 1,
         "shortest": 515, "longest": 515, "portion": 2048},
        # and generation in 32 bits: four short prompts
        {"name": "generate-4b-f32", "kind": "generate", "model": "4b", "layers": 6, "dtype": "float32", "requests": 4,
         "shortest": 21, "longest": 90, "new": 16, "portion": 0},
        # hybrid decoders at the larger of the compared sizes: a state space, attention under a window beside a matrix memory,
        # experts (Figalix); latent attention, gated linear attention, experts (Damilix)
        {"name": "generate-figalix", "kind": "generate", "model": "figalix", "layers": 8, "dtype": "bfloat16", "requests": 3,
         "shortest": 350, "longest": 1003, "new": 12, "portion": 0},
        {"name": "generate-damilix", "kind": "generate", "model": "damilix", "layers": 8, "dtype": "bfloat16", "requests": 3,
         "shortest": 350, "longest": 1003, "new": 12, "portion": 0},
    ]


def _between(rng, low, high):
    """A whole number, spread over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    which = rng.choice(["prompt", "prompt", "decode", "decode", "serve", "f32 prompt", "f32 generate", "tiny", "figalix", "damilix"])
    if which == "prompt":
        longest = _between(rng, 5, 6000)
        requests = rng.choice([1, 1, 2, 3])
        return {"kind": "prompt", "model": rng.choice(["8b", "4b", "32b"]), "layers": rng.randint(3, 8), "dtype": "bfloat16",
                "requests": requests, "shortest": max(3, longest // rng.randint(1, 4)), "longest": longest, "portion": 2048}
    if which == "decode":
        requests = _between(rng, 1, 64)
        longest = _between(rng, 100, min(6000, 64000 // requests))
        sampled = rng.random() < 0.4
        return {"kind": "decode", "model": rng.choice(["8b", "4b"]), "layers": rng.randint(4, 12), "dtype": "bfloat16",
                "requests": requests, "shortest": max(20, longest // rng.randint(1, 6)), "longest": longest,
                "temperature": rng.choice([0.6, 0.7, 0.8]) if sampled else 0.0, "top_p": rng.choice([0.9, 0.95]) if sampled else 1.0}
    if which == "serve":
        longest = _between(rng, 300, 2500)
        return {"kind": "generate", "model": rng.choice(["8b", "4b"]), "layers": rng.randint(4, 10), "dtype": "bfloat16",
                "requests": _between(rng, 3, 16), "shortest": max(20, longest // rng.randint(2, 9)), "longest": longest,
                "new": rng.randint(8, 24), "portion": rng.choice([256, 512])}
    if which == "f32 prompt":
        longest = _between(rng, 17, 800)
        return {"kind": "prompt", "model": rng.choice(["4b", "8b"]), "layers": rng.randint(2, 5), "dtype": "float32",
                "requests": rng.choice([1, 1, 2]), "shortest": max(9, longest // rng.randint(1, 3)), "longest": longest, "portion": 2048}
    if which == "f32 generate":
        longest = _between(rng, 9, 300)
        return {"kind": "generate", "model": rng.choice(["4b", "8b"]), "layers": rng.randint(2, 5), "dtype": "float32",
                "requests": _between(rng, 1, 8), "shortest": max(5, longest // rng.randint(1, 4)), "longest": longest,
                "new": rng.randint(6, 20), "portion": 0}
    if which == "tiny":
        longest = rng.randint(8, 60)
        return {"kind": "generate", "model": "tiny", "layers": rng.randint(2, 4), "dtype": rng.choice(["float32", "bfloat16"]),
                "requests": rng.randint(1, 6), "shortest": rng.randint(2, 8), "longest": longest, "new": rng.randint(6, 20), "portion": 0}
    longest = _between(rng, 60, 1300)
    return {"kind": "generate", "model": which, "layers": rng.choice([4, 8]), "dtype": "bfloat16", "requests": rng.randint(1, 4),
            "shortest": max(40, longest // rng.randint(1, 4)), "longest": longest, "new": rng.randint(4, 16), "portion": 0}


def _lengths(case):
    """The prompts' lengths (of a decode case: the tokens in the cache), spread evenly, not in order, the longest last."""
    n, low, high = case["requests"], case["shortest"], case["longest"]
    stride = next(k for k in (5, 3, 7, 11) if n % k)
    even = [high - (high - low) * (stride * i % n) // max(n - 1, 1) for i in range(n)]
    return even[1:] + even[:1]


# ---------------------------------------------------------------------------------------------------------------------
# configurations and weights
# ---------------------------------------------------------------------------------------------------------------------

_QWEN = {
    "8b": dict(hidden_size=4096, intermediate_size=12288, num_attention_heads=32, tie_word_embeddings=False),
    "4b": dict(hidden_size=2560, intermediate_size=9728, num_attention_heads=32, tie_word_embeddings=True),
    "32b": dict(hidden_size=5120, intermediate_size=25600, num_attention_heads=64, tie_word_embeddings=False),
}
_WIDE = dict(width=4096, heads=32, kv_heads=8, dim=128, vdim=128, experts=16, top=2, ff=1536, vocab=32000)
_STRETCHED = {"factor": 8.0, "original": 8192, "fast": 32.0, "slow": 1.0}


def _raw_config(case):
    """The config.json of a case's model."""
    model, layers = case["model"], case["layers"]
    if model == "tiny":
        return dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3", hidden_size=96, intermediate_size=160, num_hidden_layers=layers,
                    num_attention_heads=6, num_key_value_heads=2, head_dim=32, vocab_size=384, max_position_embeddings=512,
                    rms_norm_eps=1e-5, rope_theta=1000000.0, tie_word_embeddings=False, use_sliding_window=True, sliding_window=16,
                    max_window_layers=1)
    if model in _QWEN:
        return dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3", num_hidden_layers=layers, num_key_value_heads=8, head_dim=128,
                    vocab_size=151936, max_position_embeddings=40960, rms_norm_eps=1e-6, rope_theta=1000000.0, **_QWEN[model])
    s = _WIDE
    width, intermediate = s["width"], 2048
    if model == "figalix":
        state = {"heads": 2 * width // 64, "vdim": 64, "state": 128, "groups": 1, "conv": 4, "norm_groups": 1}
        left = {"heads": s["heads"], "kv_heads": s["kv_heads"], "dim": s["dim"], "vdim": s["vdim"], "scale": s["dim"] ** -0.5,
                "rot": {"base": 500000.0, "dims": s["dim"] // 2, "scaling": dict(_STRETCHED)}, "mask": {"size": 1024, "keep_first": 4}}
        right = {"heads": width // 256, "dim": 128, "vdim": 256, "gate_cap": 15.0}
        mixers = [("mamba2", state), ("parallel", {"left": left, "right": right})]
        mlps = [{"kind": "dense", "ff": intermediate},
                {"kind": "moe", "router": {"experts": s["experts"], "top": s["top"]}, "expert": {"ff": s["ff"]}, "shared": {"ff": s["ff"]}}]
        return {"architecture": "Figalix", "width": width, "vocab": s["vocab"], "norm": {"eps": 1e-6}, "residual_mult": 0.5, "logit_softcap": 30.0,
                "layers": [{"type": mixers[i % 2][0], "mixer": dict(mixers[i % 2][1]), "mlp": dict(mlps[i % 2])} for i in range(layers)]}
    lat = {"heads": 16, "dim": 64, "rot_dim": 64, "vdim": 64, "kv_rank": 192, "scale": 128 ** -0.5, "rot": {"base": 500000.0, "dims": 64}}
    stretched = dict(lat, rot=dict(lat["rot"], scaling=dict(_STRETCHED)))
    linear = {"heads": width // 256, "dim": 128, "vdim": 256, "tau": 16.0}
    mixers = [("latent_attention", stretched), ("gla", linear), ("latent_attention_2", lat), ("gla", linear)]
    experts = {"kind": "moe", "expert": {"ff": s["ff"]}, "shared": {"ff": s["ff"]},
               "router": {"experts": s["experts"], "identity": 2, "top": s["top"], "scale": 1.0}}
    mlps = [{"kind": "dense", "ff": intermediate}, experts, experts, experts]
    return {"architecture": "Damilix", "width": width, "vocab": s["vocab"], "norm": {"eps": 1e-6}, "token_side": {"dim": 256},
            "layers": [{"type": mixers[i % 4][0], "mixer": dict(mixers[i % 4][1]), "mlp": dict(mlps[i % 4])} for i in range(layers)]}


def _sizes(raw):
    """(width, vocabulary, layers) of a configuration."""
    if "hidden_size" in raw:
        return raw["hidden_size"], raw["vocab_size"], raw["num_hidden_layers"]
    return raw["width"], raw["vocab"], len(raw["layers"])


def _matrices(raw):
    """{name: (shape, share of its rows' values that a token needs, factor on the usual scale)} of every matrix that
    multiplies rows, the output head and embedding left out.  The usual scale keeps a normed row's values about one."""
    E, _, L = _sizes(raw)
    out = {}
    small = (2.0 * L) ** -0.5  # the layers' outputs together are about as large as the embedding
    if "hidden_size" in raw:
        H, G, d, I = raw["num_attention_heads"], raw["num_key_value_heads"], raw["head_dim"], raw["intermediate_size"]
        s = small * _embedding_scale(raw)
        for i in range(L):
            a, m = f"model.layers.{i}.self_attn.", f"model.layers.{i}.mlp."
            for name, rows in (("q", H * d), ("k", G * d), ("v", G * d)):
                out[a + name + "_proj.weight"] = ((rows, E), 1.0, 1.0)
            out[a + "o_proj.weight"] = ((E, H * d), 1.0, 2.0 * s)
            out[m + "gate_proj.weight"] = out[m + "up_proj.weight"] = ((I, E), 1.0, 1.0)
            out[m + "down_proj.weight"] = ((E, I), 1.0, 2.0 * s)
        return out
    back = small if raw["architecture"] == "Figalix" else 1.0
    for i, layer in enumerate(raw["layers"]):
        m, x, kind = layer["mixer"], f"l{i}.mix.", layer["type"]
        if kind == "mamba2":
            inner = m["heads"] * m["vdim"]
            out[x + "in"] = ((2 * inner + 2 * m["groups"] * m["state"] + m["heads"], E), 1.0, 1.0)
            out[x + "o"] = ((E, inner), 1.0, back)
        elif kind == "parallel":
            a, r = m["left"], m["right"]
            for name, rows in (("q", a["heads"] * a["dim"]), ("k", a["kv_heads"] * a["dim"]), ("v", a["kv_heads"] * a["vdim"]), ("g", a["heads"])):
                out[x + "left." + name] = ((rows, E), 1.0, 1.0)
            out[x + "left.o"] = ((E, a["heads"] * a["vdim"]), 1.0, 1.0)
            for name, rows in (("q", r["heads"] * r["dim"]), ("k", r["heads"] * r["dim"]), ("v", r["heads"] * r["vdim"]),
                               ("g", r["heads"] * r["vdim"]), ("i", r["heads"]), ("f", r["heads"])):
                out[x + "right." + name] = ((rows, E), 1.0, 1.0)
            out[x + "right.o"] = ((E, r["heads"] * r["vdim"]), 1.0, 1.0)
        elif kind == "gla":
            for name, rows in (("q", m["heads"] * m["dim"]), ("k", m["heads"] * m["dim"]), ("v", m["heads"] * m["vdim"]),
                               ("g", m["heads"] * m["vdim"]), ("a1", 16)):
                out[x + name] = ((rows, E), 1.0, 1.0)
            out[x + "a2"] = ((m["heads"] * m["dim"], 16), 1.0, 1.0)
            out[x + "o"] = ((E, m["heads"] * m["vdim"]), 1.0, 1.0)
        else:
            H = m["heads"]
            out[x + "q"] = ((H * (m["dim"] + m["rot_dim"]), E), 1.0, 1.0)
            out[x + "dkv"] = ((m["kv_rank"] + m["rot_dim"], E), 1.0, 1.0)
            out[x + "uk"], out[x + "uv"] = ((H * m["dim"], m["kv_rank"]), 1.0, 1.0), ((H * m["vdim"], m["kv_rank"]), 1.0, 1.0)
            out[x + "g"], out[x + "o"] = ((H, E), 1.0, 1.0), ((E, H * m["vdim"]), 1.0, 1.0)
        f, y = layer["mlp"], f"l{i}.mlp."
        if f["kind"] == "dense":
            out[y + "gate"] = out[y + "up"] = ((f["ff"], E), 1.0, 1.0)
            out[y + "down"] = ((E, f["ff"]), 1.0, 2.0 * back)
        else:
            n, identity = f["router"]["experts"], f["router"].get("identity", 0)
            out[y + "router"] = ((n + identity, E), 1.0, 1.0)
            for e in range(n):
                share = f["router"]["top"] / (n + identity)
                out[f"{y}e{e}.gate"] = out[f"{y}e{e}.up"] = ((f["expert"]["ff"], E), share, 1.0)
                out[f"{y}e{e}.down"] = ((E, f["expert"]["ff"]), share, 2.0 * back)
            out[y + "shared.gate"] = out[y + "shared.up"] = ((f["shared"]["ff"], E), 1.0, 1.0)
            out[y + "shared.down"] = ((E, f["shared"]["ff"]), 1.0, 2.0 * back)
            if raw["architecture"] == "Damilix":
                out[y + "shared.sg"] = ((1, E), 1.0, 1.0)
        if raw["architecture"] == "Damilix":
            side = raw["token_side"]["dim"]
            out[f"l{i}.side.gate"], out[f"l{i}.side.proj"] = ((side, E), 1.0, 1.0), ((E, side), 1.0, 1.0)
    return out


def _embedding_scale(raw):
    """Tokens are predicted by their embedding's own direction; this is the scale at which a logit comes out at about 16."""
    E = _sizes(raw)[0]
    return 24.0 / E if "hidden_size" in raw else 1.0


def _normal(seed, name, shape):
    generator = torch.Generator(device=DEVICE)
    generator.manual_seed(int.from_bytes(hashlib.sha256(f"{seed}/{name}".encode()).digest()[:8], "little") >> 1)
    return torch.randn(shape, generator=generator, device=DEVICE, dtype=torch.float32)


def _successors(raw, seed):
    """The token that the model is rather sure of after each token: another one where the head has a table of its own,
    the same one where it shares the embedding's."""
    V = _sizes(raw)[1]
    tied = raw.get("tie_word_embeddings", raw.get("architecture") == "Figalix")
    return torch.arange(V, device=DEVICE) if tied else torch.randperm(V, generator=torch.Generator().manual_seed(seed)).to(DEVICE)


def _weights(case, seed):
    """{name: tensor} of a case's model, made on the device, in the case's data type."""
    raw = _raw_config(case)
    dtype = getattr(torch, case["dtype"])
    E, V, L = _sizes(raw)
    w = {}

    def matrix(name, shape, scale):
        w[name] = (_normal(seed, name, shape) * scale).to(dtype)

    def vector(name, size, mean, spread):
        w[name] = (mean + spread * _normal(seed, name, (size,) if size else ())).to(dtype)

    for name, (shape, _, factor) in _matrices(raw).items():
        matrix(name, shape, factor * shape[1] ** -0.5)
    follow = _successors(raw, seed)
    table = _normal(seed, "embed", (V, E)) * _embedding_scale(raw)
    if "hidden_size" in raw:
        for i in range(L):
            base = f"model.layers.{i}."
            vector(base + "input_layernorm.weight", E, 1.0, 0.1)
            vector(base + "post_attention_layernorm.weight", E, 1.0, 0.1)
            vector(base + "self_attn.q_norm.weight", raw["head_dim"], 1.4, 0.1)
            vector(base + "self_attn.k_norm.weight", raw["head_dim"], 1.0, 0.1)
        vector("model.norm.weight", E, 1.0, 0.1)
        w["model.embed_tokens.weight"] = table.to(dtype)
        if not raw["tie_word_embeddings"]:
            w["lm_head.weight"] = torch.empty_like(w["model.embed_tokens.weight"]).index_copy_(0, follow, w["model.embed_tokens.weight"])
        return w
    for i, layer in enumerate(raw["layers"]):
        m, base, kind = layer["mixer"], f"l{i}.", layer["type"]
        x = base + "mix."
        if layer["mlp"]["kind"] == "moe":
            # tokens that know their experts: along each router's rows, two of a token's own choosing
            rows = w[base + "mlp.router"].float()
            rows = rows / rows.norm(dim=1, keepdim=True)
            order = _normal(seed, base + "choice", (V, rows.shape[0])).argsort(dim=1)
            table += 7.0 * rows[order[:, 0]] + 5.5 * rows[order[:, 1]]
        if raw["architecture"] == "Figalix":
            for norm in ("norm1", "norm2"):
                vector(base + norm, E, 1.0, 0.1)
                vector(base + norm + ".alpha", 0, 0.7, 0.02)
                vector(base + norm + ".b", E, 0.0, 0.02)
            if kind == "mamba2":
                inner, channels = m["heads"] * m["vdim"], m["heads"] * m["vdim"] + 2 * m["groups"] * m["state"]
                matrix(x + "conv", (channels, m["conv"]), 0.5)
                vector(x + "conv.b", channels, 0.0, 0.1)
                vector(x + "dt_bias", m["heads"], -4.0, 1.0)   # steps of 0.001 to 0.1
                vector(x + "A_log", m["heads"], 1.5, 0.7)      # decays of 1 to 16 to a step of 1
                vector(x + "D", m["heads"], 1.0, 0.1)
                vector(x + "norm", inner, 1.0, 0.1)
            else:
                r = m["right"]
                vector(x + "right.i.b", r["heads"], 0.0, 0.5)
                vector(x + "right.f.b", r["heads"], 4.0, 1.0)  # gates that keep
                vector(x + "right.norm", r["heads"] * r["vdim"], 1.0, 0.1)
                vector(x + "left.out", E, (2.0 * L) ** -0.5, 0.02)
                vector(x + "right.out", E, (2.0 * L) ** -0.5, 0.02)
        else:
            vector(base + "norm1", E, 0.3, 0.03)
            vector(base + "norm2", E, 0.3, 0.03)
            vector(base + "side.norm", E, 0.2, 0.02)
            if kind == "gla":
                vector(x + "a2.b", m["heads"] * m["dim"], 1.0, 1.0)
                vector(x + "norm", m["vdim"], 1.0, 0.1)
            else:
                vector(x + "dkv.norm", m["kv_rank"], 1.0, 0.1)
                vector(x + "sink", m["heads"], 0.0, 1.0)
            if layer["mlp"]["kind"] == "moe":
                vector(base + "mlp.correction", layer["mlp"]["router"]["experts"] + layer["mlp"]["router"]["identity"], 0.0, 0.01)
    w["embed"] = table.to(dtype)
    if raw["architecture"] == "Figalix":
        vector("final.norm", E, 40.0 / E, 4.0 / E)
        vector("final.norm.alpha", 0, 0.7, 0.02)
        vector("final.norm.b", E, 0.0, 1.0 / E)
    else:
        vector("embed.norm", E, 1.0, 0.1)
        vector("final.norm", E, 1.0, 0.1)
        matrix("side.embed", (V, raw["token_side"]["dim"] * L), 1.0)
        w["head"] = torch.empty_like(w["embed"]).index_copy_(0, follow, (table * (24.0 / E)).to(dtype))
    return w


def _prompts(case, seed):
    """Lists of token ids."""
    V = _sizes(_raw_config(case))[1]
    rng = np.random.RandomState(seed % (1 << 31))
    more = 1 if case["kind"] == "decode" else 0  # the token that the first decode step takes
    return [rng.randint(0, V, n + more).tolist() for n in _lengths(case)]


# ---------------------------------------------------------------------------------------------------------------------
# what is run
# ---------------------------------------------------------------------------------------------------------------------


def prepare(case, seed):
    raw = _raw_config(case)
    prompts = _prompts(case, seed)
    new = {"prompt": 0, "decode": DECODE_STEPS, "generate": case.get("new", 0)}[case["kind"]]
    room = sum(-(-(len(p) + new + 1) // PAGE) * PAGE for p in prompts) + 2 * PAGE

    def source(specs, device, ignorable):
        return loader.from_tensors(_weights(case, seed), specs, device, ignorable)

    runner = ModelRunner.build(config_from_dict(raw), source, dtype=case["dtype"], device=DEVICE, page_size=PAGE, max_tokens=room,
                               num_slots=len(prompts) + 1)
    state = {"case": case, "runner": runner, "prompts": prompts}
    if case["kind"] == "generate":
        state["engine"] = kirai_b200.Engine(runner=runner, max_new_tokens=case["new"], max_prefill_tokens=STEP_TOKENS,
                                            max_concurrent_requests=len(prompts), prefill_chunk=case["portion"] or None)
        state["params"] = kirai_b200.SamplingParams(temperature=0.0, max_new_tokens=case["new"], ignore_eos=True)
    if case["kind"] == "decode":
        requests = [runner.cache.open(i) for i in range(len(prompts))]
        for request, prompt in zip(requests, prompts):
            for first in range(0, len(prompt) - 1, STEP_TOKENS):
                runner.step([StepEntry(request, prompt[first : min(first + STEP_TOKENS, len(prompt) - 1)], [])])
            if not runner.cache.reserve(request, DECODE_STEPS):
                raise RuntimeError("no pages left")
        graphs = DecodeGraphs(runner)
        state.update(requests=requests, graphs=graphs, lengths=[r.length for r in requests],
                     draws=np.random.RandomState(seed % (1 << 31)).rand(DECODE_STEPS, len(requests)).tolist())
        _decode(state)  # captures the step, once, as a server does
    torch.cuda.empty_cache()  # what loading left over
    return state


def _prompt(state):
    runner, portion = state["runner"], state["case"]["portion"]
    requests = [runner.cache.open(i) for i in range(len(state["prompts"]))]
    rows = []
    for first in range(0, max(len(p) for p in state["prompts"]), portion):
        entries = [StepEntry(r, p[first : first + portion], [len(p) - first - 1] if len(p) <= first + portion else [])
                   for r, p in zip(requests, state["prompts"]) if len(p) > first]
        logits = runner.step(entries)
        if logits is not None:
            ends = [i for i, p in enumerate(state["prompts"]) if first < len(p) <= first + portion]
            rows += list(zip(ends, logits))
    for request in requests:
        runner.cache.close(request)
    return {"logits": torch.stack([row for _, row in sorted(rows, key=lambda r: r[0])])}


def _decode(state):
    case, cache, requests, lengths = state["case"], state["runner"].cache, state["requests"], state["lengths"]
    B = len(requests)
    tables = [cache.block_table_array(requests, g) for g in range(len(cache.groups))]
    graph, fresh = state["graphs"].get(B, max(t.shape[1] for t in tables), [n + 1 for n in lengths])
    slots, first = [r.slot for r in requests], [p[-1] for p in state["prompts"]]
    running, tokens = None, []
    for k in range(DECODE_STEPS):
        graph.load_inputs(first if k == 0 else None, [n + k for n in lengths], slots, tables, [case["temperature"]] * B, [case["top_p"]] * B,
                          state["draws"][k])
        if fresh and k == 0:
            graph.capture()
        step = graph.launch()  # queued behind the running one, whose tokens it takes on the device
        if running is not None:
            tokens.append(running.wait())
        running = step
    tokens.append(running.wait())
    return {"tokens": np.array(tokens), "logits": graph.logits_out}


def _generate(state):
    engine, prompts, new = state["engine"], state["prompts"], state["case"]["new"]
    engine.step_log = []
    outputs = engine.generate(prompts, state["params"])
    # the logits of the last request's last step, in the buffer of the captured step that made them
    lengths = [length for length, _ in engine.step_log[-1]]
    bucket = engine.graphs.batch_bucket(len(lengths))
    graph, fresh = engine.graphs.get(bucket, -(-(max(lengths) + 1) // PAGE), [n + 1 for n in lengths] + [1] * (bucket - len(lengths)))
    if fresh:
        raise RuntimeError("the last step was not a captured one")
    row = max(i for i, n in enumerate(lengths) if n == len(prompts[-1]) + new - 2)
    return {"tokens": np.array([o.token_ids for o in outputs]), "logits": graph.logits_out[row]}


def run(state):
    return {"prompt": _prompt, "decode": _decode, "generate": _generate}[state["case"]["kind"]](state)


# ---------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without, and what it may differ by
# ---------------------------------------------------------------------------------------------------------------------


def _layer_pairs(raw, first, count):
    """(pairs of query and key, key rows read) summed over the layers with attention, and multiply-adds per pair of them,
    for ``count`` new tokens behind ``first``; and the values that one token adds to the caches."""
    def seen(window, keep):
        total = 0
        for p in range(first, first + count):
            total += p + 1 if not window else min(p + 1, window) + max(0, min(keep, p + 1 - window))
        return total

    known = {}

    def add(flops, rows, window, keep, heads, width, row):
        if (window, keep) not in known:
            known[window, keep] = seen(window, keep)
        return flops + 4.0 * heads * width * known[window, keep], rows + row * min(first + count, (window + keep + count) if window else first + count)

    flops = rows = 0.0
    if "hidden_size" in raw:
        H, G, d = raw["num_attention_heads"], raw["num_key_value_heads"], raw["head_dim"]
        for i in range(raw["num_hidden_layers"]):
            window = raw["sliding_window"] if raw.get("use_sliding_window") and i >= raw["max_window_layers"] else 0
            flops, rows = add(flops, rows, window, 0, H, d, 2 * G * d)
        return flops, rows
    for layer in raw["layers"]:
        m = layer["mixer"]
        if layer["type"] == "mamba2":
            flops += 6.0 * m["heads"] * m["vdim"] * m["state"] * count
            rows += 2.0 * m["heads"] * m["vdim"] * m["state"] * 2  # a state of 32-bit values, read and written
        elif layer["type"] in ("parallel", "gla"):
            r = m.get("right", m)
            flops += 6.0 * r["heads"] * r["dim"] * r["vdim"] * count
            rows += 2.0 * r["heads"] * r["dim"] * r["vdim"] * 2
            if layer["type"] == "parallel":
                a = m["left"]
                flops, rows = add(flops, rows, a["mask"]["size"], a["mask"]["keep_first"], a["heads"], a["dim"], 2 * a["kv_heads"] * a["dim"])
        else:
            flops, rows = add(flops, rows, 0, 0, m["heads"], m["dim"] + m["rot_dim"], m["kv_rank"] + m["rot_dim"])
    return flops, rows


def work(case):
    raw = _raw_config(case)
    E, V, _ = _sizes(raw)
    size = 4 if case["dtype"] == "float32" else 2
    matrices = _matrices(raw)
    total = {"bytes": 0.0, "flops": 0.0}

    def step(runs, wanted):
        """One step over [(tokens before, new tokens)]."""
        tokens = sum(n for _, n in runs)
        for shape, share, _ in matrices.values():
            numbers = shape[0] * shape[1]
            total["flops"] += 2.0 * tokens * share * numbers
            total["bytes"] += size * numbers * min(1.0, share * tokens)
        total["flops"] += 2.0 * wanted * V * E
        total["bytes"] += (size * V * E if wanted else 0) + 4.0 * wanted * V + size * tokens * E
        for first, count in runs:
            flops, rows = _layer_pairs(raw, first, count)
            total["flops"] += flops
            total["bytes"] += size * rows

    lengths = _lengths(case)
    if case["kind"] == "prompt":
        for first in range(0, max(lengths), case["portion"]):
            runs = [(first, min(case["portion"], n - first)) for n in lengths if n > first]
            step(runs, sum(1 for n in lengths if first < n <= first + case["portion"]))
    elif case["kind"] == "decode":
        for k in range(DECODE_STEPS):
            step([(n + k, 1) for n in lengths], len(lengths))
    else:
        # prompts in as few full steps as hold them, then every request's tokens together
        waiting = [(first, min(STEP_TOKENS, n - first)) for n in lengths for first in range(0, n, STEP_TOKENS)]
        while waiting:
            taken, waiting = [waiting[0]], waiting[1:]
            while waiting and sum(n for _, n in taken) + waiting[0][1] <= STEP_TOKENS:
                taken, waiting = taken + [waiting[0]], waiting[1:]
            step(taken, sum(1 for first, n in taken if first + n in lengths))
        for k in range(case["new"] - 1):
            step([(n + k, 1) for n in lengths], len(lengths))
    return total


def tolerance(case):
    # against ``exact`` the logits are 5e-7 (tiny) to 2.4e-6 off in 32 bits, and 1.6e-3 to 5.4e-3 in bfloat16; tokens have not
    # differed.  About four times that
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 1e-4, "differ": 0.0}
    return {"rel": 0.02, "max": 0.2, "differ": 0.05}


# ---------------------------------------------------------------------------------------------------------------------
# the same in plain 64-bit torch, whole sequences at a time
# ---------------------------------------------------------------------------------------------------------------------


class _Wide:
    """Tensors by name, widened to 64 bits when asked for."""

    def __init__(self, tensors):
        self.tensors = tensors

    def __getitem__(self, name):
        return self.tensors[name].to(F64)


def _unit(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(z):
    return z * torch.sigmoid(z)


def _rotated(x, base, dims, scaling=None, neighbours=False):
    """x [T, heads, d] with its first ``dims`` columns rotated; angles are 32-bit products of 32-bit positions and
    frequencies, as in every implementation of these designs."""
    i = torch.arange(dims // 2, dtype=F64, device=x.device)
    f = base ** (-2.0 * i / dims)
    amplitude = 1.0
    if scaling:
        def index_of(turns):
            return dims * math.log(scaling["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))

        lo, hi = max(math.floor(index_of(scaling["fast"])), 0), min(math.ceil(index_of(scaling["slow"])), dims - 1)
        ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
        f = f / scaling["factor"] * ramp + f * (1.0 - ramp)
        amplitude = 0.1 * math.log(scaling["factor"]) + 1.0
    angle = (torch.arange(x.shape[0], dtype=torch.float32, device=x.device)[:, None] * f.float()[None, :]).to(F64)
    cos, sin = angle.cos()[:, None, :] * amplitude, angle.sin()[:, None, :] * amplitude
    a, b = (slice(0, dims, 2), slice(1, dims, 2)) if neighbours else (slice(0, dims // 2), slice(dims // 2, dims))
    y = x.clone()
    y[..., a], y[..., b] = x[..., a] * cos - x[..., b] * sin, x[..., b] * cos + x[..., a] * sin
    return y


def _attention(q, k, v, scale, window=0, keep=0, sink=None):
    """q [T, H, d], k [T, G, d], v [T, G, dv] -> [T, H dv]; row i sees j <= i, inside its window or among the kept first."""
    T, H = q.shape[:2]
    group = H // k.shape[1]
    out = torch.empty(T, H, v.shape[-1], dtype=F64, device=q.device)
    for lo in range(0, T, 1024):
        i = torch.arange(lo, min(lo + 1024, T), device=q.device)[:, None]
        j = torch.arange(int(i[-1]) + 1, device=q.device)[None, :]
        hidden = (j > i) | ((i - j >= window) & (j >= keep) if window else False)
        for g in range(k.shape[1]):
            heads = slice(g * group, (g + 1) * group)
            s = torch.einsum("thd,jd->htj", q[lo : lo + 1024, heads], k[: j.shape[1], g]) * scale
            s.masked_fill_(hidden[None], -math.inf)
            if sink is not None:
                s = torch.cat([s, sink[heads].view(-1, 1, 1).expand(-1, s.shape[1], 1)], dim=-1)
            p = torch.softmax(s, dim=-1)[..., : j.shape[1]]
            out[lo : lo + 1024, heads] = torch.einsum("htj,jd->thd", p, v[: j.shape[1], g])
    return out.reshape(T, -1)


def _qwen(raw, w, tokens, rows):
    E, _, L = _sizes(raw)
    H, G, d, eps = raw["num_attention_heads"], raw["num_key_value_heads"], raw["head_dim"], raw["rms_norm_eps"]
    x = w.tensors["model.embed_tokens.weight"][tokens].to(F64)
    T = x.shape[0]
    for i in range(L):
        a, base = f"model.layers.{i}.self_attn.", f"model.layers.{i}."
        n = _unit(x, eps) * w[base + "input_layernorm.weight"]
        q = _unit((n @ w[a + "q_proj.weight"].T).view(T, H, d), eps) * w[a + "q_norm.weight"]
        k = _unit((n @ w[a + "k_proj.weight"].T).view(T, G, d), eps) * w[a + "k_norm.weight"]
        v = (n @ w[a + "v_proj.weight"].T).view(T, G, d)
        window = raw["sliding_window"] if raw.get("use_sliding_window") and i >= raw["max_window_layers"] else 0
        o = _attention(_rotated(q, raw["rope_theta"], d), _rotated(k, raw["rope_theta"], d), v, d ** -0.5, window)
        if i == L - 1:  # only the wanted rows go on
            o, x = o[rows], x[rows]
        x = x + o @ w[a + "o_proj.weight"].T
        n = _unit(x, eps) * w[base + "post_attention_layernorm.weight"]
        x = x + (_silu(n @ w[base + "mlp.gate_proj.weight"].T) * (n @ w[base + "mlp.up_proj.weight"].T)) @ w[base + "mlp.down_proj.weight"].T
    head = "model.embed_tokens.weight" if raw["tie_word_embeddings"] else "lm_head.weight"
    return (_unit(x, eps) * w["model.norm.weight"]) @ w[head].T


def _gated(n, w, prefix):
    return (_silu(n @ w[prefix + "gate"].T) * (n @ w[prefix + "up"].T)) @ w[prefix + "down"].T


def _experts(n, w, mlp, prefix, scores, weights):
    """The sum of the chosen experts' outputs (beyond the last expert: the row itself) and the shared branch's."""
    out = torch.zeros_like(n)
    top = scores.topk(mlp["router"]["top"], dim=-1).indices
    chosen = weights(top)
    for e in range(mlp["router"]["experts"] + mlp["router"].get("identity", 0)):
        row, place = (top == e).nonzero(as_tuple=True)
        if row.numel():
            y = _gated(n[row], w, f"{prefix}e{e}.") if e < mlp["router"]["experts"] else n[row]
            out[row] += chosen[row, place][:, None] * y
    return out


def _figalix_memory(n, w, m, x, eps):
    T, H, d, dv, cap = n.shape[0], m["heads"], m["dim"], m["vdim"], m["gate_cap"]
    q, k, v = ((n @ w[x + name].T).view(T, H, -1) for name in "qkv")
    q = q * d ** -0.5
    take_log = cap * torch.tanh((n @ w[x + "i"].T + w[x + "i.b"]) / cap)
    keep_log = torch.nn.functional.logsigmoid(cap * torch.tanh((n @ w[x + "f"].T + w[x + "f.b"]) / cap))
    S, z, peak, rows = n.new_zeros(H, d, dv), n.new_zeros(H, d), n.new_zeros(H), []
    for t in range(T):
        top = torch.maximum(keep_log[t] + peak, take_log[t])
        keep, kt = torch.exp(keep_log[t] + peak - top)[:, None], torch.exp(take_log[t] - top)[:, None] * k[t]
        S = torch.baddbmm(S * keep[:, :, None], kt[:, :, None], v[t][:, None, :])
        z, peak = keep * z + kt, top
        bottom = torch.maximum((z * q[t]).sum(-1).abs(), torch.exp(-peak)) + 1e-6
        rows.append(torch.bmm(q[t][:, None, :], S)[:, 0] / bottom[:, None])
    o = _unit(torch.stack(rows), eps).reshape(T, -1) * w[x + "norm"] * torch.sigmoid(n @ w[x + "g"].T)
    return o @ w[x + "o"].T


def _figalix_state(n, w, m, x, eps):
    T, H, P, N, G = n.shape[0], m["heads"], m["vdim"], m["state"], m["groups"]
    inner = H * P
    proj = n @ w[x + "in"].T
    z, xbc, dt = proj[:, :inner], proj[:, inner : 2 * inner + 2 * G * N], proj[:, 2 * inner + 2 * G * N :]
    padded = torch.cat([xbc.new_zeros(m["conv"] - 1, xbc.shape[1]), xbc])
    xbc = _silu(w[x + "conv.b"] + sum(padded[j : j + T] * w[x + "conv"][:, j] for j in range(m["conv"])))
    u, B, C = xbc[:, :inner].view(T, H, P), xbc[:, inner : inner + G * N].view(T, G, N), xbc[:, inner + G * N :].view(T, G, N)
    B, C = (b.repeat_interleave(H // G, dim=1) for b in (B, C))
    dt = torch.nn.functional.softplus(dt + w[x + "dt_bias"], threshold=100.0)
    decay = torch.exp(-torch.exp(w[x + "A_log"]) * dt)
    S, rows = n.new_zeros(H, N, P), []
    for t in range(T):
        S = torch.baddbmm(S * decay[t][:, None, None], (dt[t][:, None] * B[t])[:, :, None], u[t][:, None, :])
        rows.append(torch.bmm(C[t][:, None, :], S)[:, 0])
    y = (torch.stack(rows) + w[x + "D"][:, None] * u).reshape(T, inner) * _silu(z)
    parts = m["norm_groups"]
    return (_unit(y.view(T, parts, -1), eps).reshape(T, inner) * w[x + "norm"]) @ w[x + "o"].T


def _figalix(raw, w, tokens, rows):
    eps, mult = raw["norm"]["eps"], raw["residual_mult"]

    def norm(x, name):
        return torch.tanh(w[name + ".alpha"] * x) * w[name] + w[name + ".b"]

    x = w.tensors["embed"][tokens].to(F64)
    T = x.shape[0]
    for i, layer in enumerate(raw["layers"]):
        m, mlp, base = layer["mixer"], layer["mlp"], f"l{i}."
        n, p = norm(x, base + "norm1"), base + "mix."
        if layer["type"] == "mamba2":
            y = _figalix_state(n, w, m, p, eps)
        else:
            a = m["left"]
            q, k, v = ((n @ w[p + "left." + name].T).view(T, heads, -1) for name, heads in (("q", a["heads"]), ("k", a["kv_heads"]), ("v", a["kv_heads"])))
            rot = a["rot"]
            o = _attention(_rotated(q, rot["base"], rot["dims"], rot["scaling"]), _rotated(k, rot["base"], rot["dims"], rot["scaling"]), v, a["scale"],
                           a["mask"]["size"], a["mask"]["keep_first"])
            o = o.view(T, a["heads"], -1) * torch.sigmoid(n @ w[p + "left.g"].T)[:, :, None]
            left = _unit(o.reshape(T, -1) @ w[p + "left.o"].T, eps) * w[p + "left.out"]
            y = 0.5 * (left + _unit(_figalix_memory(n, w, m["right"], p + "right.", eps), eps) * w[p + "right.out"])
        x = x + mult * y
        n, p = norm(x, base + "norm2"), base + "mlp."
        if mlp["kind"] == "dense":
            x = x + mult * _gated(n, w, p)
        else:
            scores = torch.softmax(n @ w[p + "router"].T, dim=-1)
            x = x + mult * (_experts(n, w, mlp, p, scores, lambda top: scores.gather(1, top)) + _gated(n, w, p + "shared."))
    logits = norm(x[rows], "final.norm") @ w["embed"].T
    return raw["logit_softcap"] * torch.tanh(logits / raw["logit_softcap"])


def _damilix(raw, w, tokens, rows):
    eps, side = raw["norm"]["eps"], raw["token_side"]["dim"]
    x = _unit(w.tensors["embed"][tokens].to(F64), eps) * w["embed.norm"]
    T = x.shape[0]
    for i, layer in enumerate(raw["layers"]):
        m, mlp, base = layer["mixer"], layer["mlp"], f"l{i}."
        p = base + "mix."
        if layer["type"] == "gla":
            q, k, v = ((x @ w[p + name].T).view(T, m["heads"], -1) for name in "qkv")
            keep = torch.exp(torch.nn.functional.logsigmoid((x @ w[p + "a1"].T) @ w[p + "a2"].T + w[p + "a2.b"]).view(T, m["heads"], -1) / m["tau"])
            S, out = x.new_zeros(m["heads"], m["dim"], m["vdim"]), []
            for t in range(T):
                S = torch.baddbmm(S * keep[t][:, :, None], k[t][:, :, None], v[t][:, None, :])
                out.append(torch.bmm(q[t][:, None, :] * m["dim"] ** -0.5, S)[:, 0])
            o = (_unit(torch.stack(out), eps) * w[p + "norm"]).reshape(T, -1) * _silu(x @ w[p + "g"].T)
        else:
            H, d = m["heads"], m["dim"]
            turn = (m["rot"]["base"], m["rot"]["dims"], m["rot"].get("scaling"), layer["type"] == "latent_attention")
            q, down = (x @ w[p + "q"].T).view(T, H, -1), x @ w[p + "dkv"].T
            latent = _unit(down[:, : m["kv_rank"]], eps) * w[p + "dkv.norm"]
            shared = _rotated(down[:, m["kv_rank"] :].reshape(T, 1, -1), *turn).expand(-1, H, -1)
            k = torch.cat([(latent @ w[p + "uk"].T).view(T, H, d), shared], dim=-1)
            q = torch.cat([q[..., :d], _rotated(q[..., d:], *turn)], dim=-1)
            o = _attention(q, k, (latent @ w[p + "uv"].T).view(T, H, -1), m["scale"], sink=w[p + "sink"])
            o = (o.view(T, H, -1) * torch.sigmoid(x @ w[p + "g"].T)[:, :, None]).reshape(T, -1)
        x = x + _unit(o @ w[p + "o"].T, eps) * w[base + "norm1"]
        p = base + "mlp."
        if mlp["kind"] == "dense":
            y = _gated(x, w, p)
        else:
            scores = torch.softmax(x @ w[p + "router"].T, dim=-1)

            def mix(top):
                picked = scores.gather(1, top)
                return picked / (picked.sum(-1, keepdim=True) + 1e-20) * mlp["router"]["scale"]

            y = _experts(x, w, mlp, p, scores + w[p + "correction"], mix) + torch.sigmoid(x @ w[p + "shared.sg"].T) * _gated(x, w, p + "shared.")
        x = x + _unit(y, eps) * w[base + "norm2"]
        own = w.tensors["side.embed"][tokens][:, i * side : (i + 1) * side].to(F64)
        gate = torch.nn.functional.gelu(x @ w[base + "side.gate"].T, approximate="tanh")
        x = x + _unit((gate * own) @ w[base + "side.proj"].T, eps) * w[base + "side.norm"]
    return (_unit(x[rows], eps) * w["final.norm"]) @ w["head"].T


def exact(case, seed):
    raw = _raw_config(case)
    w = _Wide(_weights(case, seed))
    follow = _successors(raw, seed)
    forward = {"Figalix": _figalix, "Damilix": _damilix}.get(raw.get("architecture"), _qwen)
    new = {"prompt": 1, "decode": DECODE_STEPS, "generate": case.get("new", 0)}[case["kind"]]
    sure = True
    tokens, last = [], []
    for prompt in _prompts(case, seed):
        # what follows is guessed and then checked, all of it in one pass over the sequence: a wrong guess begins a new one
        chain = torch.tensor(prompt, device=DEVICE)
        while True:
            while chain.numel() < len(prompt) + new - 1:
                chain = torch.cat([chain, follow[chain[-1:]]])
            rows = torch.arange(len(prompt) - 1, len(prompt) + new - 1, device=DEVICE)
            logits = forward(raw, w, chain, rows)
            best = logits.argmax(dim=-1)
            wrong = (best[:-1] != chain[len(prompt) :]).nonzero()
            if not wrong.numel():
                break
            at = int(wrong[0])
            chain = torch.cat([chain[: len(prompt) + at], best[at : at + 1]])
        if case.get("temperature"):
            # a nucleus that holds one token is that token, whatever is drawn
            sure = sure and bool((torch.softmax(logits / case["temperature"], dim=-1).max(dim=-1).values > case["top_p"]).all())
        tokens.append(best.tolist())
        last.append(logits[-1])
    last = torch.stack(last)
    if case["kind"] == "prompt":
        return {"logits": last}
    if case["kind"] == "decode":
        return {"tokens": np.array(tokens).T.copy(), "logits": last} if sure else {"tokens": None, "logits": None}
    return {"tokens": np.array(tokens), "logits": last[-1]}
