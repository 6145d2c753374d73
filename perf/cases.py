"""What the engine is timed on: passes through its public entry points, over the sizes its users bring.

A case names a model shape (the shapes of ``leone_b200.benchmark``), a dtype, and what is done with it:

``prompt``    one ``Engine.step`` that brings whole prompts of new requests and asks for logits; the requests end.
``decode``    requests that already hold a context get tokens through ``Engine.decode_logits`` (the captured
              decode step), then the cache is cut back to the context so that the pass can be repeated.
``mixed``     one ``Engine.step`` of a server between the two: decode rows beside a portion of a new prompt.
``serve``     a request's whole life: prompts in one step, then decoded tokens, then the requests end.
``generate``  ``generate()`` on an engine, token ids in and token ids out, greedy in 32 bits.
``sample``    ``Engine.sample``: one token per row of logits, with truncation stages.

Decoded tokens are given by the case and not fed back, so that a last bit of one logit cannot change the rest of the
pass; every pass returns the logits of every place that it asked for.
"""
import math

import numpy as np
import torch

from leone_b200 import generate
from leone_b200.engine.engine import Engine
from leone_b200.registry import config_from_dict, spec_from_config
from leone_b200.sampling.sampler import SamplingParams

DEVICE = "cuda"
DTYPES = {"bf16": torch.bfloat16, "fp32": torch.float32}


# -- shapes ---------------------------------------------------------------------------------------------
def _qwen3(layers, width, heads, kv_heads, dim, ff, vocab, tied, positions=40960, theta=1000000.0, eps=1e-6):
    return dict(architectures=["Qwen3ForCausalLM"], num_hidden_layers=layers, hidden_size=width,
                num_attention_heads=heads, num_key_value_heads=kv_heads, head_dim=dim, intermediate_size=ff,
                vocab_size=vocab, rope_theta=theta, rms_norm_eps=eps, max_position_embeddings=positions,
                tie_word_embeddings=tied)


def _sarizen(width, layers, heads, experts, top, expert_ff, shared_ff, window, vocab):
    latent = {"heads": heads, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512, "scale": 192 ** -0.5,
              "mask": {"size": window},
              "rot": {"base": 10000.0, "dims": 64,
                      "scaling": {"factor": 8.0, "original": 4096, "fast": 32.0, "slow": 1.0}}}
    lightning = {"heads": heads, "dim": 128, "vdim": 128,
                 "decay": [1.0 - 2.0 ** (-5.0 - 3.0 * h / max(heads - 1, 1)) for h in range(heads)]}
    moe = {"kind": "moe", "expert": {"ff": expert_ff}, "router": {"experts": experts, "top": top},
           "shared": {"ff": shared_ff}}
    return {"architecture": "Sarizen", "vocab": vocab, "width": width, "norm": {"eps": 1e-6}, "logit_scale": 1.0,
            "layers": [{"type": "lightning" if i % 4 else "latent_attention", "mixer": lightning if i % 4 else latent,
                        "mlp": moe if i else {"kind": "dense", "ff": top * expert_ff + shared_ff}}
                       for i in range(layers)]}


def _malapel(width, runs, heads, experts, top, expert_ff, window, chunk, vocab):
    def mix(kind, size=None):
        m = {"heads": heads, "kv_heads": heads // 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
             "rot": {"base": 1000000.0, "dims": 128}}
        return kind, dict(m, mask={"size": size}) if size else m
    kinds = [mix("attention_3", window), mix("attention", chunk), mix("attention_2"), mix("attention_2")]
    dense = {"kind": "dense", "ff": top * expert_ff, "limit": 7.0}
    moe = {"kind": "moe", "expert": {"ff": expert_ff},
           "router": {"experts": experts, "top": top, "scale": 2.0, "groups": {"count": 8, "keep": 4}}}
    return {"architecture": "Malapel", "vocab": vocab, "width": width, "norm": {"eps": 1e-6},
            "loop": {"start": 0, "stop": 2, "times": 2},
            "layers": [{"type": kinds[i % 4][0], "mixer": kinds[i % 4][1], "mlp": moe if i % 2 else dense}
                       for i in range(runs - 2)]}


def _kakirax(width, layers, heads, ff, vocab):
    attn = {"heads": heads, "kv_heads": heads // 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
            "rot": {"base": 500000.0, "dims": 128,
                    "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}}
    gla = {"heads": heads, "dim": 128, "vdim": 128, "tau": 16.0, "decay_rank": 16}
    return {"architecture": "Kakirax", "vocab": vocab, "width": width, "norm": {"eps": 1e-6}, "logit_softcap": 30.0,
            "embedding": {"scale": 8.0},
            "layers": [{"type": "attention" if i % 4 == 3 else "gla", "mixer": attn if i % 4 == 3 else gla,
                        "mlp": {"kind": "dense", "ff": ff}} for i in range(layers)]}


MODELS = {
    # 2 layers of width 64: what tests and first steps with the package run
    "tiny": _qwen3(2, 64, 4, 2, 16, 128, 256, True, positions=128, theta=10000.0),
    "qwen3-1.7b": _qwen3(28, 2048, 16, 8, 128, 6144, 151936, True),
    "qwen3-8b": _qwen3(36, 4096, 32, 8, 128, 12288, 151936, False),
    "sarizen-small": _sarizen(2048, 8, 16, 32, 4, 512, 1024, 1024, 32768),
    "sarizen-medium": _sarizen(4096, 8, 32, 64, 6, 1024, 2048, 2048, 65536),
    "malapel-small": _malapel(2048, 8, 16, 32, 4, 768, 1024, 1024, 32768),
    "malapel-medium": _malapel(4096, 8, 32, 64, 8, 1024, 2048, 2048, 65536),
    "kakirax-small": _kakirax(2048, 8, 16, 3072, 32768),
    "kakirax-medium": _kakirax(4096, 8, 32, 8192, 65536),
}


# -- the cases ------------------------------------------------------------------------------------------
def listed():
    return [
        # the smallest call there is: three short prompts through generate() on a model of two layers, where only
        # the host's path and the number of launches count
        {"name": "tiny-generate-fp32", "do": "generate", "model": "tiny", "dtype": "fp32", "requests": 3, "tokens": 13,
         "steps": 8},
        # the headline: eight conversations of 2,048 tokens decode together
        {"name": "8b-decode-8x2048", "do": "decode", "model": "qwen3-8b", "dtype": "bf16", "requests": 8, "tokens": 2048,
         "ragged": False, "steps": 16},
        # the headline's other half: a long prompt, of which the next token is wanted
        {"name": "8b-prompt-2048", "do": "prompt", "model": "qwen3-8b", "dtype": "bf16", "requests": 1, "tokens": 2048,
         "ragged": False, "want": 1},
        # a busy server of a small model: 64 requests with contexts of 64 to 2,048 tokens
        {"name": "1.7b-decode-64-ragged", "do": "decode", "model": "qwen3-1.7b", "dtype": "bf16", "requests": 64,
         "tokens": 2048, "ragged": True, "steps": 4},
        # the same server while a prompt arrives: 40 decode rows beside a portion of 987 tokens
        {"name": "1.7b-mixed-40+987", "do": "mixed", "model": "qwen3-1.7b", "dtype": "bf16", "requests": 40, "tokens": 1024,
         "ragged": True, "portion": 987},
        # a short question: 77 tokens until the first answer token, alone on the machine
        {"name": "1.7b-prompt-77", "do": "prompt", "model": "qwen3-1.7b", "dtype": "bf16", "requests": 1, "tokens": 77,
         "ragged": False, "want": 1},
        # the 32-bit path, which checks a model or a trace: logits at places of a prompt, and a few tokens after it
        {"name": "1.7b-fp32-prompt-509", "do": "prompt", "model": "qwen3-1.7b", "dtype": "fp32", "requests": 1, "tokens": 509,
         "ragged": False, "want": 16},
        {"name": "1.7b-fp32-decode-4x300", "do": "decode", "model": "qwen3-1.7b", "dtype": "fp32", "requests": 4, "tokens": 300,
         "ragged": False, "steps": 4},
        # a hybrid with linear attention, latent attention and routed experts reads a long prompt
        {"name": "sarizen-prompt-2048", "do": "prompt", "model": "sarizen-small", "dtype": "bf16", "requests": 1,
         "tokens": 2048, "ragged": False, "want": 16},
        # looped layers with three attention rules and routed experts: three prompts of unequal length in one step
        {"name": "malapel-prompts-3x900", "do": "prompt", "model": "malapel-small", "dtype": "bf16", "requests": 3,
         "tokens": 900, "ragged": True, "want": 16},
        # gated linear attention: eight requests from their prompts to their last tokens
        {"name": "kakirax-serve-8", "do": "serve", "model": "kakirax-small", "dtype": "bf16", "requests": 8, "tokens": 200,
         "ragged": True, "want": 1, "steps": 24},
        # a batch of rows sampled with top-k and top-p, as chat requests ask for it
        {"name": "sample-64-top-k-top-p", "do": "sample", "model": "tiny", "dtype": "fp32", "requests": 64, "vocab": 151936,
         "stages": "top_k=40,top_p=0.95", "temperature": 0.8},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["generate", "decode", "decode", "prompt", "prompt", "prompt", "mixed", "fp32", "fp32", "design",
                       "design", "design", "design", "sample"])
    if kind == "generate":
        return {"do": "generate", "model": "tiny", "dtype": "fp32", "requests": rng.randint(1, 6), "tokens": _log(rng, 2, 60),
                "steps": rng.randint(1, 16)}
    if kind == "sample":
        stages = rng.choice(["top_k=40,top_p=0.95", "top_p=0.9", "min_p=0.05", "top_k=%d" % _log(rng, 2, 200), "typical=0.9"])
        return {"do": "sample", "model": "tiny", "dtype": "fp32", "requests": _log(rng, 1, 64),
                "vocab": rng.choice([151936, 32768, _log(rng, 1000, 150000)]), "stages": stages,
                "temperature": round(rng.uniform(0.5, 1.2), 2)}
    if kind == "decode":
        model = rng.choice(["qwen3-1.7b", "qwen3-8b"])
        requests = _log(rng, 1, 64)
        tokens = _log(rng, 64, min(4096, (16384 if model == "qwen3-8b" else 65536) // requests))
        return {"do": "decode", "model": model, "dtype": "bf16", "requests": requests, "tokens": tokens,
                "ragged": rng.random() < 0.5, "steps": rng.randint(2, 8)}
    if kind == "prompt":
        requests = rng.choice([1, 1, 1, 2, 5])
        return {"do": "prompt", "model": rng.choice(["qwen3-1.7b", "qwen3-8b"]), "dtype": "bf16", "requests": requests,
                "tokens": _log(rng, 16, 2048 // requests), "ragged": requests > 1, "want": 1}
    if kind == "mixed":
        return {"do": "mixed", "model": "qwen3-1.7b", "dtype": "bf16", "requests": _log(rng, 2, 63),
                "tokens": _log(rng, 64, 1024), "ragged": True, "portion": _log(rng, 64, 1900)}
    if kind == "fp32":
        if rng.random() < 0.5:
            requests = rng.choice([1, 1, 3])
            return {"do": "prompt", "model": "qwen3-1.7b", "dtype": "fp32", "requests": requests,
                    "tokens": _log(rng, 8, 500 // requests), "ragged": requests > 1, "want": 4}
        return {"do": "decode", "model": "qwen3-1.7b", "dtype": "fp32", "requests": rng.randint(1, 8),
                "tokens": _log(rng, 16, 500), "ragged": rng.random() < 0.5, "steps": 2}
    model = rng.choice(["sarizen", "malapel", "kakirax"]) + rng.choice(["-small", "-small", "-medium"])
    if rng.random() < 0.6:
        requests = rng.choice([1, 1, 3])
        return {"do": "prompt", "model": model, "dtype": "bf16", "requests": requests, "tokens": _log(rng, 40, 2048 // requests),
                "ragged": requests > 1, "want": 8}
    return {"do": "serve", "model": model, "dtype": "bf16", "requests": _log(rng, 1, 16), "tokens": _log(rng, 8, 120),
            "ragged": True, "want": 1, "steps": rng.randint(4, 24)}


# -- inputs: tensors of a checkpoint, token ids -----------------------------------------------------------
def _tensor_table(cfg):
    """``(name, shape, mean, deviation)`` of every tensor of a checkpoint, in order.

    Token rows are of order one and output projections shrink with the depth, as in trained models, where a sublayer adds
    a small part of the stream; so bfloat16 rounding is not blown up from layer to layer, and a router's close call, which a
    last bit can turn, moves a token's logits by a little only.  The tiny model, which runs in 32 bits, is N(0, 0.02)
    throughout, like the package's own random weights."""
    if "architectures" in cfg:
        tiny = cfg["hidden_size"] < 256
        rows, out = (0.02, 0.02) if tiny else (1.0, 0.02 / math.sqrt(2 * cfg["num_hidden_layers"]))
        w, h, g, d, f = (cfg[k] for k in ("hidden_size", "num_attention_heads", "num_key_value_heads", "head_dim",
                                          "intermediate_size"))
        t = [("model.embed_tokens.weight", (cfg["vocab_size"], w), 0.0, rows), ("model.norm.weight", (w,), 1.0, 0.1)]
        if not cfg["tie_word_embeddings"]:
            t.append(("lm_head.weight", (cfg["vocab_size"], w), 0.0, 0.02))
        for i in range(cfg["num_hidden_layers"]):
            p = "model.layers.%d." % i
            t += [(p + "self_attn.%s_proj.weight" % n, s, 0.0, std)
                  for n, s, std in (("q", (h * d, w), 0.02), ("k", (g * d, w), 0.02), ("v", (g * d, w), 0.02), ("o", (w, h * d), out))]
            t += [(p + "mlp.%s_proj.weight" % n, s, 0.0, std)
                  for n, s, std in (("gate", (f, w), 0.02), ("up", (f, w), 0.02), ("down", (w, f), out))]
            t += [(p + "self_attn.%s_norm.weight" % n, (d,), 1.0, 0.1) for n in ("q", "k")]
            t += [(p + n + ".weight", (w,), 1.0, 0.1) for n in ("input_layernorm", "post_attention_layernorm")]
        return t
    arch, w, layers = cfg["architecture"], cfg["width"], cfg["layers"]
    out = 0.02 / math.sqrt(2 * len(layers))
    around = 0.0 if arch == "Malapel" else 1.0              # Malapel's gains are stored as their distance from one
    norm = lambda name, n=w: [(name, (n,), around, 0.1)] + ([(name + ".b", (n,), 0.0, 0.1)] if arch == "Kakirax" else [])  # noqa: E731
    t = [("embed", (cfg["vocab"], w), 0.0, 2.0 / cfg.get("embedding", {}).get("scale", 1.0))] + norm("final.norm")
    if arch != "Kakirax":
        t.append(("head", (cfg["vocab"], w), 0.0, 0.02))
    if arch == "Malapel":
        t += norm("embed.norm") + [("loop.in", (w, 2 * w), 0.0, 0.5 / math.sqrt(w))]
    for i, layer in enumerate(layers):
        m, f, p = layer["mixer"], layer["mlp"], "l%d." % i
        h, d, dv, g = m["heads"], m["dim"], m["vdim"], m.get("kv_heads", m["heads"])
        t += norm(p + "norm1") + norm(p + "norm2")
        p += "mix."
        if layer["type"] == "latent_attention":
            r, rank = m["rot_dim"], m["kv_rank"]
            t += [(p + "q", (h * (d + r), w), 0.0, 0.02), (p + "dkv", (rank + r, w), 0.0, 0.02),
                  (p + "dkv.norm", (rank,), 1.0, 0.1), (p + "uk", (h * d, rank), 0.0, 0.02),
                  (p + "uv", (h * dv, rank), 0.0, 0.02), (p + "sink", (h,), 0.0, 1.0), (p + "g", (h, w), 0.0, 0.02)]
        else:
            t += [(p + "q", (h * d, w), 0.0, 0.02), (p + "k", (g * d, w), 0.0, 0.02), (p + "v", (g * dv, w), 0.0, 0.02)]
        if layer["type"] == "lightning":
            t += [(p + "g", (h * dv, w), 0.0, 0.02), (p + "norm", (h * dv,), 1.0, 0.1)]
        if layer["type"] == "gla":
            rank = m["decay_rank"]
            t += [(p + "g", (h * dv, w), 0.0, 0.02), (p + "norm", (dv,), 1.0, 0.1), (p + "a1", (rank, w), 0.0, 0.02),
                  (p + "a2", (h * d, rank), 0.0, 0.02), (p + "a2.b", (h * d,), 0.0, 0.5)]
        if arch == "Kakirax" and layer["type"] == "attention":
            t += [(p + "g", (h * dv, w), 0.0, 0.02), (p + "q.norm", (d,), 1.0, 0.1), (p + "k.norm", (d,), 1.0, 0.1)]
        if arch == "Malapel" and layer["type"] == "attention":
            t += [(p + "q.norm", (h * d,), 1.0, 0.1), (p + "k.norm", (g * d,), 1.0, 0.1)]
        if layer["type"] == "attention_3":
            t.append((p + "pb", (h,), 0.0, 0.5))
        t.append((p + "o", (w, h * dv), 0.0, out))
        p = "l%d.mlp." % i
        gated = lambda q, n: [(q + "gate", (n, w), 0.0, 0.02), (q + "up", (n, w), 0.0, 0.02), (q + "down", (w, n), 0.0, out)]  # noqa: E731
        plain = lambda q, n: gated(q, n)[1:]                # noqa: E731
        if f["kind"] == "dense":
            t += (plain if arch == "Sarizen" else gated)(p, f["ff"])
        else:
            t.append((p + "router", (f["router"]["experts"], w), 0.0, 0.02))
            for e in range(f["router"]["experts"]):
                t += (gated if arch == "Sarizen" else plain)(p + "e%d." % e, f["expert"]["ff"])
            if "shared" in f:
                t += gated(p + "shared.", f["shared"]["ff"])
    return t


def _tensors(case, seed):
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    dtype = DTYPES[case["dtype"]]
    return {name: torch.empty(shape, dtype=dtype, device=DEVICE).normal_(mean, std, generator=gen)
            for name, shape, mean, std in _tensor_table(MODELS[case["model"]])}


def _vocab(case):
    cfg = MODELS[case["model"]]
    return cfg["vocab_size"] if "vocab_size" in cfg else cfg["vocab"]


def _lengths(case, seed):
    """Tokens each request brings (or holds): all the same, or spread between a thirty-second and the whole."""
    n, tokens = case["requests"], case["tokens"]
    if not case.get("ragged", True):
        return [tokens] * n
    rs = np.random.RandomState(seed % (1 << 31))
    return [int(v) for v in rs.randint(max(1, tokens // 32), tokens + 1, n)]


def _shape_seed(case):
    """Ragged lengths are part of the case, not of its inputs: every pass of a case does the same work."""
    return sum(ord(c) * (i + 1) for i, c in enumerate(case["model"])) + 131 * case["requests"] + case["tokens"]


def _tokens(case, seed):
    """Token ids: ``(prompts or contexts, given decode tokens [steps][requests], portion of a new prompt)``."""
    rs = np.random.RandomState((seed + 77) % (1 << 31))
    vocab = _vocab(case)
    prompts = [rs.randint(0, vocab, n).tolist() for n in _lengths(case, _shape_seed(case))]
    fed = rs.randint(0, vocab, (max(case.get("steps", 1), 1), case["requests"])).tolist()
    portion = rs.randint(0, vocab, case.get("portion", 1)).tolist()
    return prompts, fed, portion


def _places(case, n):
    """Which places of a prompt of ``n`` tokens give logits: the last one, or ``want`` places up to it."""
    want = min(case["want"], n)
    return sorted({n - 1 - (j * n) // want for j in range(want)})


def _logits_to_sample(case, seed):
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    return torch.empty((case["requests"], case["vocab"]), device=DEVICE).normal_(0.0, 3.0, generator=gen)


def _params(case, seed):
    stages = tuple((s.split("=")[0], float(s.split("=")[1])) for s in case["stages"].split(","))
    return [SamplingParams(case["temperature"], seed + i, stages) for i in range(case["requests"])]


# -- a pass ---------------------------------------------------------------------------------------------
def prepare(case, seed):
    prompts, fed, portion = _tokens(case, seed) if case["do"] != "sample" else ([], [], [])
    # token rows of one step, and what the cache has to hold at the end of a pass
    held = [len(p) + case.get("steps", 0) for p in prompts]
    rows = max(2048, case.get("portion", 0) + case.get("requests", 0))
    pages = sum(-(-n // 16) + 1 for n in held) + -(-case.get("portion", 0) // 16) + 1
    engine = Engine(spec_from_config(config_from_dict(MODELS[case["model"]])), _tensors(case, seed), dtype=DTYPES[case["dtype"]],
                    page_tokens=16, num_pages=pages + 8, max_requests=case["requests"] + 1, max_batch_tokens=rows)
    state = {"case": case, "engine": engine, "prompts": prompts, "fed": fed, "portion": portion}
    if case["do"] == "sample":
        state["logits"] = _logits_to_sample(case, seed)
        state["params"] = _params(case, seed)
        state["positions"] = [100 + 7 * i for i in range(case["requests"])]
    if case["do"] in ("decode", "mixed"):
        for rid, tokens in enumerate(prompts):
            for at in range(0, len(tokens), rows):
                engine.step([(rid, tokens[at:at + rows], [])])
    return state


def run(state):
    case, engine, prompts, fed = state["case"], state["engine"], state["prompts"], state["fed"]
    do = case["do"]
    if do == "generate":
        ids = generate(engine, prompts, case["steps"], temperature=0.0, eos_token_id=-1)
        return np.array(ids, dtype=np.int64)
    if do == "sample":
        return np.array(engine.sample(state["logits"], state["params"], state["positions"]), dtype=np.int64)
    rids = list(range(len(prompts)))
    if do == "decode":
        out = torch.stack([engine.decode_logits(rids, tokens).clone() for tokens in fed])
        for rid in rids:
            engine.cache.truncate(rid, len(prompts[rid]))
        return out
    if do == "mixed":
        entries = [(rid, [fed[0][rid]], [0]) for rid in rids]
        logits = engine.step(entries + [("new", state["portion"], [case["portion"] - 1])])
        engine.close("new")
        for rid in rids:
            engine.cache.truncate(rid, len(prompts[rid]))
        return logits
    logits = engine.step([(rid, p, _places(case, len(p))) for rid, p in zip(rids, prompts)])
    out = [logits]
    if do == "serve":
        out.append(torch.stack([engine.decode_logits(rids, tokens).clone() for tokens in fed]))
    for rid in rids:
        engine.close(rid)
    return out


# -- what a pass cannot do without ------------------------------------------------------------------------
def work(case):
    if case["do"] == "sample":
        n = case["requests"] * case["vocab"]
        return {"bytes": 4.0 * n, "flops": 10.0 * n}
    cfg, size = MODELS[case["model"]], 2 if case["dtype"] == "bf16" else 4
    lengths = _lengths(case, _shape_seed(case))
    table = _tensor_table(cfg)
    if "architectures" in cfg:
        layers, vocab, width = cfg["num_hidden_layers"], cfg["vocab_size"], cfg["hidden_size"]
        kinds = [("attention", cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"], cfg["head_dim"], None)] * layers
        times = [1] * layers
    else:
        vocab, width = cfg["vocab"], cfg["width"]
        times = [1] * len(cfg["layers"])
        for i in range(*((cfg["loop"]["start"], cfg["loop"]["stop"]) if "loop" in cfg else (0, 0))):
            times[i] = cfg["loop"]["times"]
        kinds = [(y["type"], y["mixer"]["heads"], y["mixer"].get("kv_heads", 1), y["mixer"]["dim"] + y["mixer"].get("rot_dim", 0),
                  y["mixer"]["vdim"], (y["mixer"].get("mask") or {}).get("size")) for y in cfg["layers"]]
    head = float(vocab * width)
    dense, experts = 0.0, 0.0                     # weights every token meets (a loop's as often as it runs), one expert's of all layers
    top = n_experts = 0
    for name, shape, _, _ in table:
        if len(shape) < 2 or "embed" in name or name in ("head", "lm_head.weight"):
            continue
        i = int(name.split(".")[0][1:]) if name[0] == "l" and name[1].isdigit() else None
        reps = 1 if i is None else times[i]
        if ".mlp.e" in name:
            if ".mlp.e0." in name:
                experts += reps * float(np.prod(shape))
                top, n_experts = cfg["layers"][i]["mlp"]["router"]["top"], cfg["layers"][i]["mlp"]["router"]["experts"]
        else:
            dense += reps * float(np.prod(shape)) * (2 if name == "loop.in" else 1)

    def step(new, before, logit_rows):
        """bytes, flops of one step in which request i brings new[i] tokens after before[i]."""
        n = sum(new)
        met = n_experts * (1.0 - (1.0 - top / n_experts) ** n) if n_experts else 0.0
        by = size * (dense + experts * met + head) + 4.0 * logit_rows * vocab
        fl = 2.0 * n * (dense + experts * top) + 2.0 * logit_rows * head
        for (kind, h, g, d, dv, limit), reps in zip(kinds, times):
            for k, b in zip(new, before):
                if kind in ("lightning", "gla"):
                    fl += reps * 4.0 * k * h * d * dv
                    by += reps * 8.0 * h * d * dv
                    continue
                seen = [min(b + j + 1, limit or b + j + 1) for j in (0, k // 2, k - 1)]
                pairs = k * (seen[0] + 2 * seen[1] + seen[2]) / 4.0
                fl += reps * 2.0 * pairs * h * (d + dv)
                by += reps * size * g * (d + dv) * (min(b, limit or b) + k)
        return by, fl

    do, steps = case["do"], case.get("steps", 1)
    passes = []
    if do in ("prompt", "serve", "generate"):
        passes.append(step(lengths, [0] * len(lengths), sum(len(_places(dict(case, want=case.get("want", 1)), n)) for n in lengths)))
    if do in ("serve", "generate", "decode"):
        for s in range(steps - (do == "generate")):
            passes.append(step([1] * len(lengths), [n + s for n in lengths], len(lengths)))
    if do == "mixed":
        passes.append(step([1] * len(lengths) + [case["portion"]], lengths + [0], len(lengths) + 1))
    return {"bytes": sum(p[0] for p in passes), "flops": sum(p[1] for p in passes)}


def tolerance(case):
    if case["do"] in ("generate", "sample"):
        return "exact"
    # About four times the distance from 64 bits that was seen: 1.3e-6 in 32 bits, 0.2 to 0.5 % in bfloat16 (the upper end
    # with 36 layers, or with routers whose close calls single tokens lose).
    if case["dtype"] == "fp32":
        return {"rel": 5e-6, "max": 1e-4}
    return {"rel": 0.02, "max": 0.5}


# -- the same in 64 bits ----------------------------------------------------------------------------------
def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _rotate(x, freqs, magnitude=1.0, adjacent=False):
    """``x``: [T, heads, dims], whole heads turned by position * frequency."""
    half = x.shape[-1] // 2
    ang = torch.arange(x.shape[0], dtype=torch.float64, device=x.device)[:, None, None] * freqs[None, None, :]
    c, s = torch.cos(ang) * magnitude, torch.sin(ang) * magnitude
    u, v = (x[..., 0::2], x[..., 1::2]) if adjacent else (x[..., :half], x[..., half:])
    a, b = u * c - v * s, v * c + u * s
    return torch.stack([a, b], -1).flatten(-2) if adjacent else torch.cat([a, b], -1)


def _freqs(rot):
    """Frequencies and magnitude: plain, with YaRN's blend (``fast``/``slow``) or scaled by wavelength (``low``/``high``)."""
    dims, base, sc = rot["dims"], float(rot["base"]), rot.get("scaling")
    f, mag = [base ** (-2.0 * i / dims) for i in range(dims // 2)], 1.0
    if sc and "fast" in sc:
        at = lambda turns: dims * math.log(sc["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))  # noqa: E731
        lo, hi = max(math.floor(at(sc["fast"])), 0), min(math.ceil(at(sc["slow"])), dims - 1)
        ramp = [min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0) for i in range(dims // 2)]
        f = [v / sc["factor"] * r + v * (1.0 - r) for v, r in zip(f, ramp)]
        mag = 0.1 * math.log(sc["factor"]) + 1.0
    elif sc:
        for i, v in enumerate(f):
            s = (sc["original"] * v / (2.0 * math.pi) - sc["low"]) / (sc["high"] - sc["low"])
            s = min(max(s, 0.0), 1.0)
            f[i] = (1.0 - s) * v / sc["factor"] + s * v
    return torch.tensor(f, dtype=torch.float64, device=DEVICE), mag


def _attend(q, k, v, scale, limit=None, chunk=None, rule="softmax", extra=None):
    """Causal attention, a key/value head at a time.  q: [T, H, d]; k, v: [T, G, .].  ``extra``: per head, the silent
    member's score (softmax) or what is added to every score (sigmoid)."""
    T, H, G = q.shape[0], q.shape[1], k.shape[1]
    p = torch.arange(T, device=q.device)
    hidden = p[None, :] > p[:, None]
    if limit:
        hidden = hidden | (p[:, None] - p[None, :] >= limit)
    if chunk:
        hidden = hidden | (p[:, None] // chunk != p[None, :] // chunk)
    out = []
    for h in range(H):
        s = q[:, h] @ k[:, h * G // H].t() * scale
        if rule == "sigmoid":
            w = torch.sigmoid(s + extra[h]).masked_fill_(hidden, 0.0)
        else:
            s = s.masked_fill_(hidden, float("-inf"))
            if extra is not None:
                s = torch.cat([s, extra[h].expand(T, 1)], 1)
            w = torch.softmax(s, -1)[:, :T]
        out.append(w @ v[:, h * G // H])
    return torch.stack(out, 1).flatten(1)


def _gated(h, W, p, act):
    return (act(h @ W(p + "gate").t()) * (h @ W(p + "up").t())) @ W(p + "down").t()


def _silu(x):
    return x * torch.sigmoid(x)


def _gelu(x):
    return 0.5 * x * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (x + 0.044715 * x ** 3)))


def _exact_mixer(kind, arch, h, W, m, eps):
    T, H, d, dv, G = h.shape[0], m["heads"], m["dim"], m["vdim"], m.get("kv_heads", m["heads"])
    if kind == "latent_attention":
        r, rank = m["rot_dim"], m["kv_rank"]
        f, mag = _freqs(m["rot"])
        q, dkv = (h @ W("q").t()).view(T, H, d + r), h @ W("dkv").t()
        c = _rms(dkv[:, :rank], eps) * W("dkv.norm")
        k_rot = _rotate(dkv[:, None, rank:], f, mag, True).expand(T, H, r)
        q = torch.cat([q[..., :d], _rotate(q[..., d:], f, mag, True)], -1)
        k = torch.cat([(c @ W("uk").t()).view(T, H, d), k_rot], -1)
        o = _attend(q, k, (c @ W("uv").t()).view(T, H, dv), m["scale"], m["mask"]["size"], extra=W("sink"))
        return (o.view(T, H, dv) * torch.sigmoid(h @ W("g").t())[:, :, None]).flatten(1) @ W("o").t()
    q, k, v = ((h @ W(n).t()).view(T, -1, e) for n, e in (("q", d), ("k", d), ("v", dv)))
    if kind == "lightning":
        q, k, v = _silu(q), _silu(k), _silu(v)
        p = torch.arange(T, device=h.device)
        gap = (p[:, None] - p[None, :]).double()
        o = torch.stack([((q[:, i] @ k[:, i].t()) * torch.where(gap >= 0, m["decay"][i] ** gap.clamp(min=0), 0.0)) @ v[:, i]
                         for i in range(H)], 1).flatten(1)
        return (_rms(o, eps) * W("norm") * torch.sigmoid(h @ W("g").t())) @ W("o").t()
    if kind == "gla":
        q = q * d ** -0.5
        a = torch.sigmoid(h @ W("a1").t() @ W("a2").t() + W("a2.b")).view(T, H, d) ** (1.0 / m["tau"])
        S, o = torch.zeros(H, d, dv, dtype=h.dtype, device=h.device), []
        for t in range(T):
            S = a[t][:, :, None] * S + k[t][:, :, None] * v[t][:, None, :]
            o.append(torch.matmul(q[t][:, None, :], S)[:, 0])
        o = (_rms(torch.stack(o), eps) * W("norm")).flatten(1)
        return (o * _silu(h @ W("g").t())) @ W("o").t()
    f, _ = _freqs(m["rot"])
    if arch == "Kakirax":
        q, k = _rms(q, eps) * W("q.norm"), _rms(k, eps) * W("k.norm")
        o = _attend(_rotate(q, f), _rotate(k, f), v, m["scale"])
        return (o * torch.sigmoid(h @ W("g").t())) @ W("o").t()
    if kind == "attention":
        q = (_rms(q.flatten(1), eps) * W("q.norm")).view(T, H, d)
        k = (_rms(k.flatten(1), eps) * W("k.norm")).view(T, G, d)
    q, k = _rotate(q, f), _rotate(k, f)
    if kind == "attention":
        o = _attend(q, k, v, m["scale"], chunk=m["mask"]["size"], extra=torch.zeros(H, dtype=h.dtype, device=h.device))
    elif kind == "attention_2":
        o = _attend(q, k, v, m["scale"])
    else:
        o = _attend(q, k, v, m["scale"], limit=m["mask"]["size"], rule="sigmoid", extra=W("pb"))
    return o @ W("o").t()


def _exact_ff(arch, h, W, f):
    square = lambda z: torch.clamp(z, min=0) ** 2           # noqa: E731
    if f["kind"] == "dense":
        if arch == "Sarizen":
            return square(h @ W("up").t()) @ W("down").t()
        if arch == "Kakirax":
            return _gated(h, W, "", _gelu)
        g, u = torch.clamp(h @ W("gate").t(), max=f["limit"]), torch.clamp(h @ W("up").t(), -f["limit"], f["limit"])
        return (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ W("down").t()
    r = f["router"]
    z = h @ W("router").t()
    score = torch.sigmoid(z) if arch == "Sarizen" else torch.softmax(z, -1)
    open_ = score
    if "groups" in r:
        n, count = r["experts"], r["groups"]["count"]
        best = torch.topk(score.view(-1, count, n // count).amax(-1), r["groups"]["keep"], -1).indices
        ok = torch.zeros(len(h), count, dtype=torch.bool, device=h.device).scatter_(1, best, True)
        open_ = score.masked_fill(~ok.repeat_interleave(n // count, 1), -1.0)
    value, chosen = torch.topk(open_, r["top"], -1)
    value = value * r.get("scale", 1.0)
    out = torch.zeros_like(h)
    for e in range(r["experts"]):
        row, at = torch.nonzero(chosen == e, as_tuple=True)
        if not len(row):
            continue
        w = value[row, at][:, None]
        if arch == "Sarizen":
            out[row] += _gated(w * h[row], W, "e%d." % e, _silu)
        else:
            out[row] += w * (square(h[row] @ W("e%d.up" % e).t()) @ W("e%d.down" % e).t())
    return out + _gated(h, W, "shared.", _silu) if "shared" in f else out


def _exact_logits(cfg, tensors, sequences, places):
    """Per sequence the logits of its places.  Layer by layer over all sequences, so that a layer's weights are widened once."""
    if "architectures" in cfg:
        w = lambda name: tensors[name + ".weight"].double()  # noqa: E731
        eps, H, G, d = cfg["rms_norm_eps"], cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"]
        f, _ = _freqs({"dims": d, "base": cfg["rope_theta"]})
        xs = [tensors["model.embed_tokens.weight"][torch.tensor(s, device=DEVICE)].double() for s in sequences]
        for i in range(cfg["num_hidden_layers"]):
            p = "model.layers.%d." % i
            Q, K, V, O = (w(p + "self_attn.%s_proj" % n) for n in "qkvo")
            gate, up, down = (w(p + "mlp.%s_proj" % n) for n in ("gate", "up", "down"))
            for j, x in enumerate(xs):
                h = _rms(x, eps) * w(p + "input_layernorm")
                q = _rms((h @ Q.t()).view(-1, H, d), eps) * w(p + "self_attn.q_norm")
                k = _rms((h @ K.t()).view(-1, G, d), eps) * w(p + "self_attn.k_norm")
                x = x + _attend(_rotate(q, f), _rotate(k, f), (h @ V.t()).view(-1, G, d), d ** -0.5) @ O.t()
                h = _rms(x, eps) * w(p + "post_attention_layernorm")
                xs[j] = x + (_silu(h @ gate.t()) * (h @ up.t())) @ down.t()
        xs = [(_rms(x[at], eps) * w("model.norm")) for x, at in zip(xs, places)]
        head = w("model.embed_tokens" if cfg["tie_word_embeddings"] else "lm_head")
        return [x @ head.t() for x in xs]
    arch, eps, layers = cfg["architecture"], cfg["norm"]["eps"], cfg["layers"]

    def norm(x, name):
        gain = tensors[name].double()
        if arch == "Kakirax":
            y = x - x.mean(-1, keepdim=True)
            return y / torch.sqrt((y * y).mean(-1, keepdim=True) + eps) * gain + tensors[name + ".b"].double()
        return _rms(x, eps) * (gain + 1.0 if arch == "Malapel" else gain)

    order = [(i, False) for i in range(len(layers))]
    if "loop" in cfg:
        a, b = cfg["loop"]["start"], cfg["loop"]["stop"]
        order = order[:a] + [(i, i == a) for _ in range(cfg["loop"]["times"]) for i in range(a, b)] + order[b:]
    out = []
    for s, at in zip(sequences, places):
        x = tensors["embed"][torch.tensor(s, device=DEVICE)].double() * cfg.get("embedding", {}).get("scale", 1.0)
        if arch == "Malapel":
            x = x0 = norm(x, "embed.norm")
        for i, first in order:
            y, p = layers[i], "l%d." % i
            part = lambda name, q="mix.": tensors[p + q + name].double()  # noqa: E731
            if first:
                x = torch.cat([x, x0], -1) @ tensors["loop.in"].double().t()
            a = _exact_mixer(y["type"], arch, norm(x, p + "norm1"), part, y["mixer"], eps)
            x2 = x if arch == "Sarizen" else x + a              # Sarizen's two branches read the same stream
            x = x + a + _exact_ff(arch, norm(x2, p + "norm2"), lambda name: part(name, "mlp."), y["mlp"])
        z = norm(x[at], "final.norm") @ tensors["embed" if arch == "Kakirax" else "head"].double().t()
        cap = cfg.get("logit_softcap")
        out.append(cap * torch.tanh(z / cap) if cap else z * cfg.get("logit_scale", 1.0))
    return out


def exact(case, seed):
    do = case["do"]
    if do in ("generate", "sample"):                          # whole numbers
        return None
    if work(dict(case, do="prompt", want=1))["flops"] > 4e14:
        return None                                           # more than about 20 seconds of 64-bit products
    prompts, fed, portion = _tokens(case, seed)
    tensors, cfg = _tensors(case, seed), MODELS[case["model"]]
    with torch.no_grad():
        if do == "mixed":
            got = _exact_logits(cfg, tensors, [p + [t] for p, t in zip(prompts, fed[0])] + [portion],
                                [[len(p)] for p in prompts] + [[len(portion) - 1]])
            return torch.cat(got)
        places = [_places(case, len(p)) if do != "decode" else [] for p in prompts]
        if do == "prompt":
            return [torch.cat(_exact_logits(cfg, tensors, prompts, places))]
        whole = [p + [t[j] for t in fed] for j, p in enumerate(prompts)]
        got = _exact_logits(cfg, tensors, whole, [a + list(range(len(p), len(p) + len(fed))) for a, p in zip(places, prompts)])
        later = torch.stack([g[len(a):] for g, a in zip(got, places)], 1)
        return later if do == "decode" else [torch.cat([g[:len(a)] for g, a in zip(got, places)]), later]
