"""The work this framework is asked to do, as cases that can be timed and checked: what goes in, one pass through the public
entry points, the bytes and operations a pass cannot do without, and what plain 64-bit arithmetic makes of the same inputs.

Three kinds of call, over two sorts of models:

  "tokens"   GGUF model: decoded tokens of one or more sequences behind a context that is already in the cache (the token that
             enters each step is given, so a pass ends where the last one did)
  "prompt"   GGUF model: one prompt, or the next part of one, then the first sampled token
  "folder"   model folder (layer list): sequences start, their prompts go through in one ragged step, some tokens follow one
             by one; logits of a few prompt rows, or of every sequence's last token

Weights are random in the formats and at the scales the formats are used with; every tensor comes from the seed.
"""
import math
import os
import sys

import numpy as np
import torch

PKG = os.path.join(os.getcwd(), "llama-fastapi-k8s-gpu_b200")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

F64 = torch.float64


def dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


# ---------------------------------------------------------------------------------------------------------------- the cases
def llama(width, heads, kv_heads, ff, vocab, layers, mix):
    return {"width": width, "heads": heads, "kv_heads": kv_heads, "ff": ff, "vocab": vocab, "layers": layers, "mix": mix}


def listed():
    wide = dict(width=4096, heads=32, kv_heads=8, ff=14336, vocab=32000)
    return [
        # one chat, answer streamed token by token: the framework's headline (8B shapes, Q4_K_M, 512-token prompt)
        {"name": "llama_token", "kind": "tokens", **wide, "layers": 4, "mix": "Q4_K_M", "seqs": 1, "context": 512, "steps": 8},
        # the same at the end of a long document (7B shapes at an 8k window)
        {"name": "llama_token_8k", "kind": "tokens", **wide, "layers": 2, "mix": "Q4_K_M", "seqs": 1, "context": 8100, "steps": 8},
        # a serving replica with 32 chats in flight (8B shapes, Q8_0)
        {"name": "llama_batch_32", "kind": "tokens", **wide, "layers": 4, "mix": "Q8_0", "seqs": 32, "context": 500, "steps": 8},
        # time to first token: a 512-token prompt
        {"name": "llama_prompt_512", "kind": "prompt", **wide, "layers": 4, "mix": "Q4_K_M", "past": 0, "prompt": 512},
        # the smallest call: a short question to a 1.1B-shaped Q4_0 model
        {"name": "llama_prompt_37", "kind": "prompt", **llama(2048, 32, 4, 5632, 32000, 2, "Q4_0"), "past": 0, "prompt": 37},
        # model folder, scoring or prompt of 2048 tokens: softmax attention with capped scores, experts by token id
        {"name": "zogurax_prompt", "kind": "folder", "family": "zogurax", "pattern": "ba", "width": 2048, "ff": 2048, "vocab": 32000,
         "dtype": "bfloat16", "prompts": "2048", "steps": 0},
        # the same model in a chat: a short prompt and an answer, one sequence
        {"name": "zogurax_chat", "kind": "folder", "family": "zogurax", "pattern": "ba", "width": 2048, "ff": 2048, "vocab": 32000,
         "dtype": "bfloat16", "prompts": "61", "steps": 24},
        # and served to 32 callers at once, prompts of different lengths
        {"name": "zogurax_batch_32", "kind": "folder", "family": "zogurax", "pattern": "ba", "width": 2048, "ff": 2048, "vocab": 32000,
         "dtype": "bfloat16", "prompts": ",".join(str(5 + 3 * i) for i in range(32)), "steps": 12},
        # latent attention (rotated, plain, and a layer that reads the plain one's latents) with gated units, 2048 tokens
        {"name": "fazovik_prompt", "kind": "folder", "family": "fazovik", "pattern": "rps", "width": 2048, "ff": 8192, "vocab": 32000,
         "dtype": "bfloat16", "prompts": "2048", "steps": 0},
        # window attention beside a selective scan, matrix memory, squared-ReLU unit, 2048 tokens at the largest width
        {"name": "goponex_prompt", "kind": "folder", "family": "goponex", "pattern": "mp", "width": 4096, "ff": 16384, "vocab": 32000,
         "dtype": "bfloat16", "prompts": "2048", "steps": 0},
        # parity runs: everything in 32 bits, two sequences of odd lengths
        {"name": "goponex_float32", "kind": "folder", "family": "goponex", "pattern": "mp", "width": 1024, "ff": 4096, "vocab": 8000,
         "dtype": "float32", "prompts": "301,158", "steps": 0},
    ]


def prompt_lengths(case):
    return [int(n) for n in case["prompts"].split(",")]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    shape = rng.choice([dict(width=4096, heads=32, kv_heads=8), dict(width=2048, heads=32, kv_heads=4), dict(width=2560, heads=20, kv_heads=5),
                        dict(width=3072, heads=24, kv_heads=8), dict(width=1024, heads=8, kv_heads=8)])
    gguf = {**shape, "ff": 256 * rng.randint(8, 56), "vocab": rng.choice([8000, 16384, 32000]), "layers": rng.randint(1, 3),
            "mix": rng.choice(["Q4_K_M", "Q8_0", "Q4_0"])}
    what = rng.choice(["tokens_1", "tokens_n", "prompt", "prompt", "folder", "folder", "folder", "folder"])
    if what == "tokens_1":
        return {"kind": "tokens", **gguf, "seqs": rng.randint(1, 2), "context": log_int(16, 8000), "steps": rng.randint(4, 8)}
    if what == "tokens_n":
        return {"kind": "tokens", **gguf, "seqs": rng.randint(3, 32), "context": log_int(16, 500), "steps": rng.randint(4, 8)}
    if what == "prompt":
        return {"kind": "prompt", **gguf, "past": rng.choice([0, 0, log_int(10, 2000)]), "prompt": log_int(8, 700)}
    family = rng.choice(["zogurax", "fazovik", "goponex"])
    pattern = {"zogurax": rng.choice(["b", "a", "ba"]), "fazovik": rng.choice(["r", "ps", "p"]), "goponex": rng.choice(["m", "p", "mp"])}[family]
    width = rng.choice([1024, 1280, 1536, 2048])
    case = {"kind": "folder", "family": family, "pattern": pattern, "width": width, "ff": 8 * rng.randint(64, 512), "vocab": rng.choice([4001, 8000, 32000]),
            "dtype": "bfloat16"}
    how = rng.choice(["prompt", "prompt", "chat", "many", "float32"])
    if how == "prompt":
        case.update(prompts=str(log_int(64, 2048)), steps=0)
    elif how == "chat":
        case.update(prompts=str(log_int(8, 200)), steps=rng.randint(8, 24))
    elif how == "many":
        case.update(prompts=",".join(str(log_int(4, 90)) for _ in range(rng.randint(2, 32))), steps=rng.randint(4, 12))
    else:
        case.update(width=rng.choice([512, 768, 1024]), dtype="float32", prompts=",".join(str(log_int(16, 300)) for _ in range(rng.randint(1, 3))), steps=0)
    return case


# ------------------------------------------------------------------------------------------------ GGUF weights (quant blocks)
BLOCK = {"Q4_0": (2, 32, 18), "Q8_0": (8, 32, 34), "Q4_K": (12, 256, 144), "Q6_K": (14, 256, 210), "F32": (0, 1, 4)}      # id, elements, bytes
UNIT = {"Q4_0": 4.611, "Q8_0": 73.91, "Q4_K": 258.6, "Q6_K": 347.0}       # standard deviation of random blocks with scale 1


def generator(seed, index):
    g = torch.Generator(device=dev())
    g.manual_seed(seed * 1000003 + index)
    return g


def f16_bytes(v):
    return v.to(torch.float16).view(torch.uint8).reshape(-1, 2)


def random_blocks(g, kind, n, k, std):
    """[n, bytes of a row]: random quants, block scales that make the values about N(0, std)."""
    _, be, bb = BLOCK[kind]
    nb = n * k // be
    b = torch.randint(0, 256, (nb, bb), dtype=torch.uint8, device=dev(), generator=g)
    d = (0.5 + torch.rand(nb, device=dev(), generator=g)) * (std / UNIT[kind])
    if kind in ("Q4_0", "Q8_0"):
        d = d * (2.0 * torch.randint(0, 2, (nb,), device=dev(), generator=g) - 1.0)
        b[:, 0:2] = f16_bytes(d)
    elif kind == "Q4_K":
        b[:, 0:2], b[:, 2:4] = f16_bytes(d), f16_bytes(7.5 * d)
    else:
        b[:, 192:208] = torch.randint(-32, 33, (nb, 16), dtype=torch.int8, device=dev(), generator=g).view(torch.uint8)
        b[:, 208:210] = f16_bytes(d)
    return b.reshape(n, k // be * bb)


def half(b, at):
    return b[:, at:at + 2].contiguous().view(torch.float16).to(F64)


def values(kind, rows, k):
    """The 64-bit values of quantised rows [n, bytes] as [n, k] (the block formats' definition)."""
    _, be, bb = BLOCK[kind]
    b = rows.reshape(-1, bb)
    if kind == "Q4_0":
        q = torch.cat([b[:, 2:] & 15, b[:, 2:] >> 4], 1).to(F64) - 8.0
        v = half(b, 0) * q
    elif kind == "Q8_0":
        v = half(b, 0) * b[:, 2:].contiguous().view(torch.int8).to(F64)
    elif kind == "Q4_K":
        s = b[:, 4:16].to(torch.int32)
        lo, hi = s[:, 8:12] & 15, s[:, 8:12] >> 4
        sc = torch.cat([s[:, 0:4] & 63, lo | ((s[:, 0:4] >> 6) << 4)], 1).to(F64)
        mn = torch.cat([s[:, 4:8] & 63, hi | ((s[:, 4:8] >> 6) << 4)], 1).to(F64)
        q = b[:, 16:].reshape(-1, 4, 1, 32)
        q = torch.cat([q & 15, q >> 4], 2).reshape(-1, 8, 32).to(F64)
        v = (half(b, 0) * sc)[:, :, None] * q - (half(b, 2) * mn)[:, :, None]
    else:
        ql, qh = b[:, 0:128].reshape(-1, 2, 2, 32).to(torch.int32), b[:, 128:192].reshape(-1, 2, 1, 32).to(torch.int32)
        low = torch.cat([ql & 15, ql >> 4], 2)                                  # quarters 0, 1 (low nibbles), 2, 3 (high)
        high = torch.cat([(qh >> (2 * i)) & 3 for i in range(4)], 2)
        q = (low | (high << 4)).to(F64) - 32.0
        sc = b[:, 192:208].contiguous().view(torch.int8).to(F64)
        v = half(b, 208)[:, :, None] * sc[:, :, None] * q.reshape(-1, 16, 16)
    return v.reshape(-1, k)


def gguf_tensors(case):
    """name -> (format, K, rows, standard deviation); the Q4_K_M mix keeps some layers' attn_v and ffn_down, and output, at Q6_K."""
    W, F, V, n = case["width"], case["ff"], case["vocab"], case["layers"]
    kv = W // case["heads"] * case["kv_heads"]
    base = {"Q4_K_M": "Q4_K"}.get(case["mix"], case["mix"])
    top = "Q8_0" if base == "Q8_0" else "Q6_K"
    out = {"token_embd.weight": (base, W, V, 0.02), "output_norm.weight": ("F32", W, 1, 0.0), "output.weight": (top, W, V, 0.02)}
    for i in range(n):
        p = f"blk.{i}."
        more = "Q6_K" if case["mix"] == "Q4_K_M" and i % 2 == 0 else base
        out.update({p + "attn_norm.weight": ("F32", W, 1, 0.0), p + "ffn_norm.weight": ("F32", W, 1, 0.0), p + "attn_q.weight": (base, W, W, 0.02),
                    p + "attn_k.weight": (base, W, kv, 0.02), p + "attn_v.weight": (more, W, kv, 0.02), p + "attn_output.weight": (base, W, W, 0.02),
                    p + "ffn_gate.weight": (base, W, F, 0.02), p + "ffn_up.weight": (base, W, F, 0.02), p + "ffn_down.weight": (more, F, W, 0.02)})
    return out


def gguf_weight(case, seed, index, spec):
    kind, k, n, std = spec
    g = generator(seed, index)
    if kind == "F32":
        return 0.5 + torch.rand(k, device=dev(), generator=g)
    return random_blocks(g, kind, n, k, std)


class Gguf:
    """A parsed model file in memory: what the loader hands to the engine."""

    class Tensor:
        def __init__(self, data, ggml_type, shape):
            self.data, self.ggml_type, self.shape = data, ggml_type, shape

    def __init__(self, case, seed):
        self.metadata = {"general.architecture": "llama", "llama.block_count": case["layers"], "llama.embedding_length": case["width"],
                         "llama.feed_forward_length": case["ff"], "llama.attention.head_count": case["heads"],
                         "llama.attention.head_count_kv": case["kv_heads"], "llama.attention.layer_norm_rms_epsilon": 1e-5, "llama.rope.freq_base": 5e5}
        self.tensors = {}
        for i, (name, spec) in enumerate(gguf_tensors(case).items()):
            w = gguf_weight(case, seed, i, spec).cpu().numpy()
            shape = (spec[1],) if spec[0] == "F32" else (spec[1], spec[2])
            self.tensors[name] = Gguf.Tensor(w, BLOCK[spec[0]][0], shape)


def token_lists(case, seed):
    """Per sequence, all its tokens: context or past, then what a pass brings."""
    g = np.random.default_rng([seed, 77])
    if case["kind"] == "tokens":
        lens = [case["context"] + case["steps"]] * case["seqs"]
        lens = [n - (5 * i) % 23 if n > 60 else n for i, n in enumerate(lens)]          # contexts of several chats differ
    elif case["kind"] == "prompt":
        lens = [case["past"] + case["prompt"]]
    else:
        lens = [p + case["steps"] for p in prompt_lengths(case)]
    return [[int(t) for t in g.integers(0, case["vocab"], size=n)] for n in lens]


# ------------------------------------------------------------------------------------------------------ model-folder weights
def folder_config(case):
    W, F, V = case["width"], case["ff"], case["vocab"]
    heads = max(2, W // 128)
    kv = max(1, heads // 4) if heads % 4 == 0 else 1
    if case["family"] == "zogurax":
        common = {"heads": heads, "kv_heads": kv, "dim": 128, "vdim": 128, "scale": 128 ** -0.5}
        mixers = {"a": dict(common, conv=4, softcap=30.0, q_temp={"coef": 0.1, "every": 1024}), "b": dict(common, softcap=50.0, q_temp={"coef": 0.2, "every": 512})}
        mlp = {"kind": "moe", "expert": {"ff": F // 2}, "router": {"experts": 8, "top": 2}, "shared": {"ff": F // 2}}
        layers = [{"type": "attention" if ch == "a" else "attention_2", "mixer": mixers[ch], "mlp": mlp} for ch in case["pattern"]]
        return {"architecture": "Zogurax", "layers": layers, "norm": {"eps": 1e-5}, "vocab": V, "width": W}
    if case["family"] == "fazovik":
        q_rank = 8 * (3 * W // 64)
        base = {"heads": heads, "dim": 128, "vdim": 128, "kv_rank": 512, "q_rank": q_rank}
        rot = dict(base, rot_dim=64, scale=192 ** -0.5, rot={"base": 1e4, "dims": 64, "scaling": {"factor": 8.0, "original": 4096, "fast": 32.0, "slow": 1.0}})
        layers = []
        for i, ch in enumerate(case["pattern"]):
            mix = rot if ch == "r" else dict(base, scale=128 ** -0.5, **({"kv_from": i - 1} if ch == "s" else {}))
            layers.append({"type": "latent_attention" if ch == "r" else "latent_attention_2", "mixer": mix, "mlp": {"kind": "dense", "ff": F}})
        return {"architecture": "Fazovik", "embedding": {"bigram": {"buckets": 4093, "mul_cur": 31, "mul_prev": 1009}}, "layers": layers,
                "norm": {"eps": 1e-5}, "vocab": V, "width": W}
    left = {"heads": heads, "kv_heads": kv, "dim": 128, "vdim": 128, "rot": {"base": 5e5, "dims": 64, "scaling": {"factor": 4.0, "fast": 16.0, "original": 8192, "slow": 2.0}},
            "mask": {"size": 1024, "keep_first": 4}, "scale": 128 ** -0.5}
    right = {"inner": 2 * W, "state": 16, "dt_rank": max(16, W // 16), "conv": 4}
    memory = {"heads": max(1, W // 256), "dim": 128, "vdim": 256, "gate_cap": 12.0}
    layers = [{"type": "mlstm", "mixer": memory, "mlp": None} if ch == "m" else
              {"type": "parallel", "mixer": {"left": left, "right": right}, "mlp": {"kind": "dense", "ff": F}} for ch in case["pattern"]]
    return {"architecture": "Goponex", "layers": layers, "norm": {"eps": 1e-5}, "postln_alpha": 1.0, "vocab": V, "width": W}


def folder_module(case):
    from llama_cpp import fazovik, goponex, zogurax
    return {"zogurax": zogurax, "fazovik": fazovik, "goponex": goponex}[case["family"]]


def folder_tensors(case, seed, shapes):
    """name -> bf16 tensor (int32 for tables of token ids)."""
    out = {}
    for i, (name, shape) in enumerate(shapes.items()):
        g = generator(seed, i)
        rand = lambda: torch.randn(shape, device=dev(), generator=g)
        uniform = lambda lo, hi: lo + (hi - lo) * torch.rand(shape, device=dev(), generator=g)
        leaf = name.rsplit(".", 1)[-1]
        if leaf == "table":
            first = torch.randint(0, 8, (shape[0], 1), device=dev(), generator=g)
            out[name] = ((first + 3 * torch.arange(shape[1], device=dev())) % 8).to(torch.int32)
            continue
        if leaf == "A_log":
            v = uniform(1.0, 16.0).log()
        elif name.endswith("dt.b"):
            v = uniform(0.001, 0.1).expm1().log()
        elif name.endswith("f.b"):
            v = uniform(3.0, 6.0)
        elif leaf == "conv":
            v = rand() * 0.4
        elif len(shape) == 2:
            v = rand() / math.sqrt(shape[1])
        elif leaf == "b":
            v = rand() * 0.05
        else:
            v = uniform(0.5, 1.5)
        out[name] = v.to(torch.bfloat16)
    return out


# ---------------------------------------------------------------------------------------------------------- prepare and run
def greedy():
    from llama_cpp.engine import SamplingSettings
    return SamplingSettings(temperature=0.0, repeat_penalty=1.0)


def prepare(case, seed):
    tokens = token_lists(case, seed)
    if case["kind"] == "folder":
        from llama_cpp.safetensors_file import STensor
        module = folder_module(case)
        cfg = folder_config(case)
        tensors = {}
        for name, t in folder_tensors(case, seed, module.tensor_shapes(cfg)).items():
            a = t.cpu().numpy() if t.dtype == torch.int32 else t.view(torch.int16).cpu().numpy().view(np.uint16)
            tensors[name] = STensor(name, "I32" if t.dtype == torch.int32 else "BF16", tuple(t.shape), a)
        longest = max(len(t) for t in tokens)
        engine = module.open_synthetic(cfg, tensors, n_ctx=longest + 16, max_seqs=len(tokens), dtype=case["dtype"],
                                       max_step_tokens=min(2048, max(64, sum(prompt_lengths(case)))))
        for slot, toks in enumerate(tokens):
            engine.ensure_pages(slot, len(toks))
        return {"case": case, "engine": engine, "tokens": tokens, "greedy": greedy()}
    from llama_cpp.engine import Engine
    engine = Engine(Gguf(case, seed), n_ctx=max(len(t) for t in tokens) + 16, max_seqs=len(tokens))
    brings = case["steps"] if case["kind"] == "tokens" else case["prompt"]
    for slot, toks in enumerate(tokens):
        engine.ensure_pages(slot, len(toks) + 1)
        engine.seq_begin(slot, 0, [], greedy())
        if len(toks) > brings:
            engine.prefill(slot, toks[:-brings])
    return {"case": case, "engine": engine, "tokens": tokens, "greedy": greedy()}


def prompt_rows(n):
    return sorted({max(0, n * i // 8 - 1) for i in range(1, 9)})


def run(state):
    case, engine, tokens = state["case"], state["engine"], state["tokens"]
    if case["kind"] == "tokens":
        n, slots, chosen = case["steps"], list(range(len(tokens))), []
        for s, toks in enumerate(tokens):
            engine.rewind(s, len(toks) - n, toks[-n], toks[-n - 64:-n])
        for i in range(n):
            chosen.append(engine.decode(slots))
            if i + 1 < n:
                for s, toks in enumerate(tokens):
                    engine.set_token(s, toks[i + 1 - n])
        return {"logits": np.stack([engine.logits(s) for s in slots]), "chosen": np.array(chosen, dtype=np.int64)}
    if case["kind"] == "prompt":
        toks, past = tokens[0], case["past"]
        engine.seq_begin(0, past, toks[:past][-64:], state["greedy"])
        engine.prefill(0, toks[past:])
        first = engine.sample(0)
        return {"logits": engine.logits(0)[None], "chosen": np.array([first], dtype=np.int64)}
    for s in range(len(tokens)):
        engine.seq_begin(s, 0, [], state["greedy"])
    steps, prompts = case["steps"], prompt_lengths(case)
    all_sample = [True] * len(tokens)
    if steps == 0:
        logits, first = engine.step([(s, t) for s, t in enumerate(tokens)], want=[prompt_rows(len(t)) for t in tokens], sample=all_sample)
        return {"logits": logits, "chosen": np.array(first, dtype=np.int64)}
    chosen = [engine.step([(s, t[:p]) for s, (t, p) in enumerate(zip(tokens, prompts))], sample=all_sample)[1]]
    for i in range(steps):
        last = i + 1 == steps
        logits, nxt = engine.step([(s, [t[p + i]]) for s, (t, p) in enumerate(zip(tokens, prompts))], want=[[0]] * len(tokens) if last else None, sample=all_sample)
        chosen.append(nxt)
    return {"logits": logits, "chosen": np.array(chosen, dtype=np.int64)}


# ----------------------------------------------------------------------------------------------------- bytes, operations, bars
def matrix_work(case):
    """(bytes of all matrices a pass needs, operations per token without the output map, the same of the output map)"""
    if case["kind"] != "folder":
        size, per_token, head = 0, 0, 0
        for name, (kind, k, n, _) in gguf_tensors(case).items():
            _, be, bb = BLOCK[kind]
            if name == "token_embd.weight":
                continue
            size += k * n // be * bb
            if name == "output.weight":
                head = 2 * k * n
            elif kind != "F32":
                per_token += 2 * k * n
        return size, per_token, head
    esz, size, per_token, head = 2, 0, 0, 0
    for name, shape in folder_module(case).tensor_shapes(folder_config(case)).items():
        leaf = name.rsplit(".", 1)[-1]
        if len(shape) != 2 or leaf in ("conv", "A_log", "table", "bigram") or (name == "embed" and case["family"] != "fazovik"):
            continue
        k = 2 * shape[0] * shape[1]
        if name in ("head", "embed"):
            head = k
            size += k // 2 * esz
        elif ".mlp.e" in name:
            share = min(1.0, 2 / 8) if len(prompt_lengths(case)) == 1 and case["steps"] else 1.0
            per_token += k * 2 // 8
            size += int(k // 2 * esz * share)
        else:
            per_token += k
            size += k // 2 * esz
    return size, per_token, head


def attention_pairs(case):
    """(query, key) pairs of one layer in a pass, and cached keys read."""
    if case["kind"] == "tokens":
        ctx = [len(t) for t in token_lists(case, 0)]
        n = case["steps"]
        pairs = sum(n * c - n * (n - 1) // 2 for c in ctx)
        return pairs, pairs
    if case["kind"] == "prompt":
        p, t = case["past"], case["prompt"]
        return t * p + t * (t + 1) // 2, p
    window = 1024 if case["family"] == "goponex" else 1 << 30
    total = read = 0
    for p in prompt_lengths(case):
        total += sum(min(i + 1, window) for i in range(p + case["steps"]))
        read += sum(min(p + i + 1, window) for i in range(case["steps"]))
    return total, read


def work(case):
    size, per_token, head = matrix_work(case)
    pairs, read = attention_pairs(case)
    if case["kind"] != "folder":
        hd = case["width"] // case["heads"]
        tokens = case["steps"] * case["seqs"] if case["kind"] == "tokens" else case["prompt"]
        heads_out = tokens if case["kind"] == "tokens" else 1
        passes = case["steps"] if case["kind"] == "tokens" else 1
        kv = 4 * case["kv_heads"] * hd * case["layers"]
        return {"bytes": passes * size + kv * (read + tokens) + 4 * case["vocab"] * heads_out,
                "flops": tokens * per_token + heads_out * head + 4 * case["heads"] * hd * case["layers"] * pairs}
    W = case["width"]
    heads = max(2, W // 128)
    prompt_tokens = sum(prompt_lengths(case))
    tokens = prompt_tokens + case["steps"] * len(prompt_lengths(case))
    rows = sum(len(prompt_rows(p)) for p in prompt_lengths(case)) if case["steps"] == 0 else (case["steps"] + 1) * len(prompt_lengths(case))
    layers = len(case["pattern"]) if case["family"] != "goponex" else case["pattern"].count("p")
    pair_ops = {"zogurax": 4 * 128, "goponex": 4 * 128, "fazovik": 4 * 128 + 2 * 64}[case["family"]] * heads
    row_bytes = {"zogurax": 4 * 128 * max(1, heads // 4), "goponex": 4 * 128 * max(1, heads // 4), "fazovik": 2 * 576}[case["family"]]
    scan = 0
    if case["family"] == "goponex":          # scan: decay, write, read of 16 states per channel; memory: write and read of 128 x 256 per head
        scan = tokens * (case["pattern"].count("p") * 2 * W * 16 * 6 + case["pattern"].count("m") * max(1, W // 256) * 128 * 256 * 5)
    return {"bytes": (case["steps"] + 1) * size + layers * row_bytes * (read + tokens) + 2 * W * tokens + 4 * case["vocab"] * rows,
            "flops": tokens * per_token + rows * head + layers * pair_ops * pairs + scan}


def tolerance(case):
    # about four times the distance from exact() that was measured: 32-bit products 1.0e-6 to 1.6e-6; model folders in bf16
    # 0.003 to 0.0054 (activations rounded to bf16 ahead of every product); GGUF models 0.001 to 0.0026 (f16 cache and activations)
    if case["kind"] == "folder" and case["dtype"] == "float32":
        return {"rel": 1e-5, "differ": 0.05}
    if case["kind"] == "folder":
        return {"rel": 2e-2, "differ": 0.25}
    return {"rel": 1e-2, "differ": 0.25}


# ------------------------------------------------------------------------------------------------ the same in plain 64 bits
def rms(x, w=None, eps=1e-5):
    y = x / ((x * x).mean(-1, keepdim=True) + eps).sqrt()
    return y if w is None else y * w


def layer_norm(x, w, b=None, eps=1e-5):
    c = x - x.mean(-1, keepdim=True)
    y = c / ((c * c).mean(-1, keepdim=True) + eps).sqrt() * w
    return y if b is None else y + b


def rotate_pairs(x, cos, sin, dims):
    """x [T, heads, d]: entries 2i and 2i + 1 of the first `dims` are one pair."""
    u, v = x[..., 0:dims:2], x[..., 1:dims:2]
    c, s = cos[:, None, :], sin[:, None, :]
    return torch.cat([torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2), x[..., dims:]], -1)


def turns(rot, T):
    dims, base = rot["dims"], rot["base"]
    i = torch.arange(dims // 2, dtype=F64, device=dev())
    f, mag = base ** (-2.0 * i / dims), 1.0
    sc = rot.get("scaling")
    if sc:
        corr = lambda t: dims * math.log(sc["original"] / (2.0 * math.pi * t)) / (2.0 * math.log(base))
        lo, hi = max(math.floor(corr(sc["fast"])), 0), min(math.ceil(corr(sc["slow"])), dims - 1)
        ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
        f, mag = f / sc["factor"] * ramp + f * (1.0 - ramp), 0.1 * math.log(sc["factor"]) + 1.0
    a = torch.arange(T, dtype=F64, device=dev())[:, None] * f
    return a.cos() * mag, a.sin() * mag


def attend(q, k, v, scale, visible, softcap=0.0, extra=0.0):
    """q [T, H, d], k [T, G, d], v [T, G, dv] -> [T, H * dv], one head at a time."""
    group, outs = q.shape[1] // k.shape[1], []
    for h in range(q.shape[1]):
        s = q[:, h] @ k[:, h // group].T * scale
        if softcap > 0.0:
            s = softcap * (s / softcap).tanh()
        s = s.masked_fill(~visible, -math.inf)
        m = s.amax(-1, keepdim=True)
        p = (s - m).exp()
        outs.append(p @ v[:, h // group] / (p.sum(-1, keepdim=True) + extra * (-m).exp()))
    return torch.cat(outs, -1)


def causal(T, window=None, keep=0):
    i = torch.arange(T, device=dev())
    ok = i[None, :] <= i[:, None]
    return ok if window is None else ok & ((i[:, None] - i[None, :] < window) | (i[None, :] < keep))


def gguf_logits(case, seed, rows_of):
    """Logits of the wanted rows of every sequence, all layers for all tokens; weights one tensor at a time."""
    specs = gguf_tensors(case)
    index = {name: i for i, name in enumerate(specs)}

    def weight(name):
        w = gguf_weight(case, seed, index[name], specs[name])
        return w.to(F64) if specs[name][0] == "F32" else values(specs[name][0], w, specs[name][1])

    seqs = token_lists(case, seed)
    H, G = case["heads"], case["kv_heads"]
    hd = case["width"] // H
    kind = specs["token_embd.weight"]
    table = gguf_weight(case, seed, index["token_embd.weight"], kind)
    xs = [values(kind[0], table[torch.tensor(t, device=dev())], kind[1]) for t in seqs]
    cut = np.cumsum([0] + [len(t) for t in seqs])
    x = torch.cat(xs)
    rot = [turns({"dims": hd, "base": 5e5}, len(t)) for t in seqs]
    for i in range(case["layers"]):
        p = f"blk.{i}."
        h = rms(x, weight(p + "attn_norm.weight"))
        q, k, v = (h @ weight(p + n).T for n in ("attn_q.weight", "attn_k.weight", "attn_v.weight"))
        outs = []
        for s, t in enumerate(seqs):
            a, b = cut[s], cut[s + 1]
            qs, ks, vs = q[a:b].reshape(-1, H, hd), k[a:b].reshape(-1, G, hd), v[a:b].reshape(-1, G, hd)
            outs.append(attend(rotate_pairs(qs, *rot[s], hd), rotate_pairs(ks, *rot[s], hd), vs, hd ** -0.5, causal(len(t))))
        x = x + torch.cat(outs) @ weight(p + "attn_output.weight").T
        h = rms(x, weight(p + "ffn_norm.weight"))
        u = torch.nn.functional.silu(h @ weight(p + "ffn_gate.weight").T) * (h @ weight(p + "ffn_up.weight").T)
        x = x + u @ weight(p + "ffn_down.weight").T
    rows = torch.cat([x[cut[s] + torch.tensor(rows_of(len(t)), device=dev())] for s, t in enumerate(seqs)])
    return rms(rows, weight("output_norm.weight")) @ weight("output.weight").T


def shift_conv(u, taps):
    """Causal convolution of every channel: u [T, C], taps [C, n]."""
    n = taps.shape[1]
    pad = torch.cat([u.new_zeros(n - 1, u.shape[1]), u])
    return sum(pad[j:j + u.shape[0]] * taps[:, j] for j in range(n))


def zogurax_layers(cfg, w, tokens):
    T, W = len(tokens), cfg["width"]
    ids = torch.tensor(tokens, device=dev())
    angle = torch.arange(T, dtype=F64, device=dev())[:, None] * 10000.0 ** (-2.0 * torch.arange((W + 1) // 2, dtype=F64, device=dev()) / W)
    x = w["embed"][ids] + torch.stack([angle.sin(), angle.cos()], -1).flatten(1)[:, :W]
    for li, L in enumerate(cfg["layers"]):
        p, m = f"l{li}.", L["mixer"]
        a, H, G, d = p + "mix.", m["heads"], m["kv_heads"], m["dim"]
        h = layer_norm(x, w[p + "norm1"])
        q, k, v = (h @ w[a + n].T for n in "qkv")
        conv = L["type"] == "attention"
        if conv:
            q, k, v = (shift_conv(t, w[a + n + ".conv"]) for t, n in ((q, "q"), (k, "k"), (v, "v")))
            q, k = rms(q, w[a + "q.norm"]), rms(k, w[a + "k.norm"])
        else:
            q, k, v = (t + w[a + n + ".b"] for t, n in ((q, "q"), (k, "k"), (v, "v")))
        pos = torch.arange(T, dtype=F64, device=dev())
        q = q * (1.0 + m["q_temp"]["coef"] * (((pos + 1.0) / m["q_temp"]["every"]).floor() + 1.0).log())[:, None]
        o = attend(q.reshape(T, H, d), k.reshape(T, G, d), v.reshape(T, G, d), m["scale"], causal(T), m["softcap"], 0.0 if conv else 1.0)
        if conv:
            o = (o.reshape(T, H, d) * (h @ w[a + "g"].T).sigmoid()[:, :, None]).reshape(T, H * d)
        y = o @ w[a + "o"].T
        if not conv:
            y = y + w[a + "o.b"]
        e = p + "mlp."
        unit = lambda z, pre: (z @ w[pre + "up"].T).clamp(min=0.0).square() @ w[pre + "down"].T
        y = y + (h @ w[e + "shared.sg"].T).sigmoid() * unit(h, e + "shared.")
        table = w[e + "table"].long()[ids]
        for n in range(L["mlp"]["router"]["experts"]):
            hits = (table == n).sum(-1)
            rows = hits.nonzero()[:, 0]
            if len(rows):
                y[rows] += unit(h[rows], f"{e}e{n}.") * hits[rows, None] / table.shape[1]
        x = x + y
    return layer_norm(x, w["final.norm"]), w["head"]


def fazovik_layers(cfg, w, tokens):
    T, bg = len(tokens), cfg["embedding"]["bigram"]
    ids = torch.tensor(tokens, device=dev())
    pair = torch.cat([ids.new_tensor([bg["buckets"]]), (ids[:-1] * bg["mul_prev"] + ids[1:] * bg["mul_cur"]) % bg["buckets"]])
    x = w["embed"][ids] + w["bigram"][pair]
    latents = {}
    for li, L in enumerate(cfg["layers"]):
        p, m = f"l{li}.", L["mixer"]
        a, H, d, rank = p + "mix.", m["heads"], m["dim"], m["kv_rank"]
        h = layer_norm(x, w[p + "norm1"], w[p + "norm1.b"])
        q = (rms(h @ w[a + "dq"].T, w[a + "dq.norm"]) @ w[a + "uq"].T).reshape(T, H, -1)
        src = m.get("kv_from", li)
        if src == li:
            down = h @ w[a + "dkv"].T
            latents[li] = rms(down[:, :rank], w[a + "dkv.norm"])
        c = latents[src]
        k, v = (c @ w[a + "uk"].T).reshape(T, H, d), (c @ w[a + "uv"].T).reshape(T, H, -1)
        if "rot_dim" in m:
            cs = turns(m["rot"], T)
            q = torch.cat([q[..., :d], rotate_pairs(q[..., d:], *cs, m["rot"]["dims"])], -1)
            kr = rotate_pairs(down[:, None, rank:], *cs, m["rot"]["dims"])
            k = torch.cat([k, kr.expand(T, H, kr.shape[-1])], -1)
        o = attend(q, k, v, m["scale"], causal(T))
        if "rot_dim" in m:
            o = (o.reshape(T, H, -1) * (h @ w[a + "g"].T).sigmoid()[:, :, None]).reshape(T, -1)
        y = o @ w[a + "o"].T
        h = layer_norm(x, w[p + "norm2"], w[p + "norm2.b"])
        g = torch.nn.functional.gelu(h @ w[p + "mlp.gate"].T, approximate="tanh")
        x = x + y + (g * (h @ w[p + "mlp.up"].T)) @ w[p + "mlp.down"].T
    return layer_norm(x, w["final.norm"], w["final.norm.b"]), w["embed"]


def matrix_memory(h, w, a, m):
    T, H, d, dv, cap = h.shape[0], m["heads"], m["dim"], m["vdim"], m["gate_cap"]
    q, k, v = ((h @ w[a + n].T).reshape(T, H, -1) for n in "qkv")
    q = q * d ** -0.5
    ig = cap * ((h @ w[a + "i"].T + w[a + "i.b"]) / cap).tanh()
    fg = torch.nn.functional.logsigmoid(cap * ((h @ w[a + "f"].T + w[a + "f.b"]) / cap).tanh())
    # log of the largest weight so far, starting at 0: m_t = max(f_t + m_(t-1), i_t) = F_t + max(0, max_s<=t (i_s - F_s))
    F = fg.cumsum(0)
    top = F + (ig - F).cummax(0).values.clamp(min=0.0)
    out = torch.empty(T, H, dv, dtype=F64, device=h.device)
    ok = causal(T)
    for n in range(H):
        weight = (F[:, None, n] - F[None, :, n] + ig[None, :, n] - top[:, None, n]).masked_fill(~ok, -math.inf).exp()
        s = weight * (q[:, n] @ k[:, n].T)
        out[:, n] = s @ v[:, n] / (torch.maximum(s.sum(-1).abs(), (-top[:, n]).exp()) + 1e-6)[:, None]
    o = rms(out).reshape(T, H * dv) * w[a + "norm"] * (h @ w[a + "g"].T).sigmoid()
    return o @ w[a + "o"].T


def selective_scan(h, w, a, m):
    T, inner, N, R = h.shape[0], m["inner"], m["state"], m["dt_rank"]
    x, z = (h @ w[a + "in"].T).split(inner, -1)
    x = torch.nn.functional.silu(shift_conv(x, w[a + "conv"]) + w[a + "conv.b"])
    dt, B, C = (x @ w[a + "x"].T).split([R, N, N], -1)
    dt = torch.nn.functional.softplus(dt @ w[a + "dt"].T + w[a + "dt.b"], threshold=60.0)
    A = -w[a + "A_log"].exp()
    S, y = torch.zeros(inner, N, dtype=F64, device=h.device), torch.empty(T, inner, dtype=F64, device=h.device)
    for t in range(T):
        S = (dt[t][:, None] * A).exp() * S + (dt[t] * x[t])[:, None] * B[t]
        y[t] = S @ C[t]
    return ((y + w[a + "D"] * x) * torch.nn.functional.silu(z)) @ w[a + "o"].T


def goponex_layers(cfg, w, tokens):
    T = len(tokens)
    x = w["embed"][torch.tensor(tokens, device=dev())]
    for li, L in enumerate(cfg["layers"]):
        p = f"l{li}."
        a = p + "mix."
        if L["type"] == "mlstm":
            y = matrix_memory(x, w, a, L["mixer"])
        else:
            m = L["mixer"]["left"]
            H, G, d = m["heads"], m["kv_heads"], m["dim"]
            q, k = (x @ w[a + "left.q"].T).reshape(T, H, d), (x @ w[a + "left.k"].T).reshape(T, G, d)
            cs = turns(m["rot"], T)
            qr, kr = (rotate_pairs(rms(t, w[a + "left." + n + ".norm"]), *cs, m["rot"]["dims"]) for t, n in ((q, "q"), (k, "k")))
            left = attend(qr, kr, k, m["scale"], causal(T, m["mask"]["size"], m["mask"]["keep_first"])) @ w[a + "left.o"].T
            right = selective_scan(x, w, a + "right.", L["mixer"]["right"])
            y = 0.5 * (rms(left, w[a + "left.out"]) + rms(right, w[a + "right.out"]))
        x = layer_norm(cfg["postln_alpha"] * x + y, w[p + "norm1"])
        if L["mlp"]:
            u = (x @ w[p + "mlp.up"].T + w[p + "mlp.up.b"]).clamp(min=0.0).square()
            x = layer_norm(cfg["postln_alpha"] * x + u @ w[p + "mlp.down"].T + w[p + "mlp.down.b"], w[p + "norm2"])
    return layer_norm(x, w["final.norm"]), w["head"]


def exact(case, seed):
    with torch.no_grad():
        if case["kind"] != "folder":
            return {"logits": gguf_logits(case, seed, lambda n: [n - 1]).cpu().numpy(), "chosen": None}
        cfg = folder_config(case)
        w = {n: (t if t.dtype == torch.int32 else t.to(F64)) for n, t in folder_tensors(case, seed, folder_module(case).tensor_shapes(cfg)).items()}
        layers = {"zogurax": zogurax_layers, "fazovik": fazovik_layers, "goponex": goponex_layers}[case["family"]]
        out = []
        for toks in token_lists(case, seed):
            x, head = layers(cfg, w, toks)
            rows = prompt_rows(len(toks)) if case["steps"] == 0 else [len(toks) - 1]
            out.append(x[torch.tensor(rows, device=x.device)] @ head.T)
        return {"logits": torch.cat(out).cpu().numpy(), "chosen": None}
