"""What the speed of this framework is measured on: its models through their public entry points, and its memory-bound ops.

A case is a dict of plain values. `prepare` gives what a serving or scoring program holds before a call (a loaded model, an engine
or position ids, and new token ids or activations made from the seed), `run` is one call of it, `exact` the same in 64 bits with
plain torch. Models have the sizes of the benchmarks (GPT-2 small and large, BERT-base, the sequence designs at width 1024
and 2048) and random weights. Unlike freshly initialised ones, their next-token choice is peaked, as a trained model's is: the row
of the head that meets a token's embedding is that embedding (GPT-2: tied) or its image under a fixed permutation (sequence
models), and the embeddings are large enough in the stream for it, so that a greedy choice is not decided by rounding.
"""
import math

import numpy as np
import torch
import torch.nn.functional as F

import applegpu_runtime_b200 as gpu
from applegpu_runtime_b200 import _lib, seqbench
from applegpu_runtime_b200.generate import Gpt2Decoder

_TORCH = {"float32": torch.float32, "float16": torch.float16, "bfloat16": torch.bfloat16}
_MODELS = {}                     # loaded models: a program loads its weights once and serves many requests


def listed():
    return [
        # scoring / prompt processing of a batch of full contexts, logits of every position: the headline benchmark
        {"name": "gpt2_8x1024_bf16", "kind": "gpt2", "dtype": "bfloat16", "batch": 8, "seq": 1024},
        # the same in float32 on short sequences
        {"name": "gpt2_8x128_f32", "kind": "gpt2", "dtype": "float32", "batch": 8, "seq": 128},
        # greedy generation for a batch of prompts: prompt, then one captured step per token
        {"name": "gpt2_generate_8x64+50", "kind": "gpt2_generate", "dtype": "bfloat16", "batch": 8, "prompt": 64, "new": 50},
        # a large model with int8 weights
        {"name": "gpt2_large_int8_32x512", "kind": "gpt2_int8", "dtype": "bfloat16", "batch": 32, "seq": 512},
        # encoding a corpus
        {"name": "bert_256x512_bf16", "kind": "bert", "dtype": "bfloat16", "batch": 256, "seq": 512},
        # prompts of the sequence models, next-token logits
        {"name": "gedenex_w1024_8x1024", "kind": "gedenex", "width": 1024, "dtype": "bfloat16", "batch": 8, "prompt": 1024, "new": 0, "each": False},
        {"name": "rurunex_w2048_8x1024", "kind": "rurunex", "width": 2048, "dtype": "bfloat16", "batch": 8, "prompt": 1024, "new": 0, "each": False},
        # prompts of an odd length, half precision
        {"name": "rurunex_w1024_3x777_f16", "kind": "rurunex", "width": 1024, "dtype": "float16", "batch": 3, "prompt": 777, "new": 0, "each": False},
        # one user's greedy answer behind a short prompt; a batch's behind long ones
        {"name": "gedenex_w2048_1x128+48", "kind": "gedenex", "width": 2048, "dtype": "bfloat16", "batch": 1, "prompt": 128, "new": 48, "each": False},
        {"name": "rurunex_w1024_8x1024+48", "kind": "rurunex", "width": 1024, "dtype": "bfloat16", "batch": 8, "prompt": 1024, "new": 48, "each": False},
        # a few tokens with the logits of each on the host, where a caller samples
        {"name": "gedenex_w1024_1x9+4_logits", "kind": "gedenex", "width": 1024, "dtype": "bfloat16", "batch": 1, "prompt": 9, "new": 4, "each": True},
        # the bandwidth-bound ops as a user's own layer calls them: layer_norm, causal softmax of scores, gelu behind a bias
        {"name": "ops_8192x768_bf16", "kind": "ops", "dtype": "bfloat16", "rows": 8192, "width": 768, "maps": 96, "len": 1024},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["gpt2", "gpt2", "gpt2_generate", "gpt2_int8", "bert", "gedenex", "gedenex", "gedenex", "rurunex", "rurunex", "rurunex", "ops"])
    if kind == "gpt2":               # up to the benchmark's 8192 rows, contexts up to the model's 1024
        seq = _log(rng, 16, 1024)
        return {"kind": kind, "dtype": rng.choice(["bfloat16", "bfloat16", "float16", "float32"]), "batch": rng.randint(1, max(1, min(32, 8192 // seq))), "seq": seq}
    if kind == "gpt2_generate":      # up to the 16 sequences that a step takes
        return {"kind": kind, "dtype": rng.choice(["bfloat16", "bfloat16", "float16", "float32"]), "batch": rng.randint(1, 16), "prompt": _log(rng, 8, 512), "new": _log(rng, 8, 64)}
    if kind == "gpt2_int8":
        return {"kind": kind, "dtype": "bfloat16", "batch": rng.randint(1, 32), "seq": _log(rng, 32, 512)}
    if kind == "bert":
        return {"kind": kind, "dtype": rng.choice(["bfloat16", "bfloat16", "float16"]), "batch": _log(rng, 1, 256), "seq": _log(rng, 16, 512)}
    if kind == "ops":
        n = _log(rng, 64, 1024)
        return {"kind": kind, "dtype": rng.choice(["bfloat16", "float32", "float16"]), "rows": _log(rng, 64, 16384), "width": rng.choice([768, 1024, 1280, 2048]), "maps": rng.randint(1, 96), "len": n}
    prompt = _log(rng, 4, 2048)
    new = 0 if rng.random() < 0.5 else _log(rng, 2, 48)
    return {"kind": kind, "width": rng.choice([1024, 2048]), "dtype": rng.choice(["bfloat16", "bfloat16", "float16"]), "batch": rng.randint(1, max(1, min(16, 8192 // prompt))),
            "prompt": prompt, "new": new, "each": bool(new) and new <= 16 and rng.random() < 0.3}


# ── weights ─────────────────────────────────────────────────────────────────
def _sizes(case):
    return gpu.GPT2_LARGE if case["kind"] == "gpt2_int8" else gpu.BERT_BASE if case["kind"] == "bert" else gpu.GPT2_SMALL


def _transformer_weights(case):
    """{name: float32 tensor on the GPU}, every value one that the model's type holds."""
    cfg, g, w = _sizes(case), torch.Generator("cuda").manual_seed(7), {}
    d, n_layer, dt = cfg["n_embd"], cfg["n_layer"], _TORCH[case["dtype"]]

    def put(name, std, *shape, mean=0.0):
        w[name] = (torch.randn(shape, generator=g, device="cuda") * std + mean).to(dt).float()

    def norm(name):
        put(name + ".weight", 0.05, d, mean=1.0)
        put(name + ".bias", 0.02, d)

    if case["kind"] == "bert":
        for n, k in (("word", cfg["vocab_size"]), ("position", cfg["n_positions"]), ("token_type", cfg["type_vocab"])):
            put(f"embeddings.{n}_embeddings.weight", 0.02, k, d)
        norm("embeddings.LayerNorm")
        for i in range(n_layer):
            p = f"encoder.layer.{i}."
            for n, o, k in (("attention.self.query", d, d), ("attention.self.key", d, d), ("attention.self.value", d, d), ("attention.output.dense", d, d),
                            ("intermediate.dense", cfg["d_ff"], d), ("output.dense", d, cfg["d_ff"])):
                put(p + n + ".weight", 0.02, o, k)
                put(p + n + ".bias", 0.02, o)
            norm(p + "attention.output.LayerNorm")
            norm(p + "output.LayerNorm")
        return w
    p = "transformer."
    put(p + "wte.weight", 0.1, cfg["vocab_size"], d)
    put(p + "wpe.weight", 0.02, cfg["n_positions"], d)
    back = 0.02 / math.sqrt(2 * n_layer)                  # the projections into the stream, as GPT-2 initialises them
    for i in range(n_layer):
        h = f"{p}h.{i}."
        norm(h + "ln_1")
        norm(h + "ln_2")
        for n, k, o, std in (("attn.c_attn", d, 3 * d, 0.02), ("attn.c_proj", d, d, back), ("mlp.c_fc", d, 4 * d, 0.02), ("mlp.c_proj", 4 * d, d, back)):
            put(h + n + ".weight", std, k, o)
            put(h + n + ".bias", 0.02 if std == 0.02 else back, o)
    norm(p + "ln_f")
    return w


def _seq_config(case):
    return (seqbench.config_of if case["kind"] == "gedenex" else seqbench.rurunex_config_of)(case["width"])


def _next_of(vocab):
    """The token that the head prefers behind each token."""
    return np.random.default_rng(3).permutation(vocab)


def _seq_weights(case):
    """{name: float32 array}; the matrices are rounded where they are used."""
    cfg = _seq_config(case)
    if case["kind"] == "gedenex":
        w = gpu.init_gedenex_weights(cfg, seed=0)
        w["embed"] *= np.float32(100.0)
        scale = 0.01
    else:
        w = gpu.init_rurunex_weights(cfg, seed=0, ranks={"channel_delta": 128})
        w["embed"] *= np.float32(5.0)
        scale = 0.2
    w["head"][_next_of(cfg["vocab"])] = w["embed"] * np.float32(scale)
    return w


def _model(case):
    key = (case["kind"].replace("_generate", ""), case.get("width"), case["dtype"])
    if key in _MODELS:
        return _MODELS[key]
    if case["kind"] in ("gedenex", "rurunex"):
        m = (gpu.load_gedenex if case["kind"] == "gedenex" else gpu.load_rurunex)(_seq_config(case), _seq_weights(case), case["dtype"])
    else:
        w = _transformer_weights(case)
        if case["kind"] == "bert":
            m = gpu.load_bert_state_dict(w, gpu.BERT_BASE, case["dtype"])
        elif case["kind"] == "gpt2_int8":
            m = gpu.quantize_gpt2_linears(gpu.load_gpt2_state_dict(w, gpu.GPT2_LARGE, case["dtype"], fold_layer_norms=False))
            for name in list(m["weights"]):
                if name.endswith((".c_attn.weight", ".c_fc.weight", ".c_proj.weight")):
                    del m["weights"][name]
        else:
            m = gpu.load_gpt2_state_dict(w, gpu.GPT2_SMALL, case["dtype"])
        del w
        torch.cuda.empty_cache()
    _MODELS[key] = m
    return m


# ── preparation ─────────────────────────────────────────────────────────────
def _ids(case, seed):
    n = case["seq"] if "seq" in case else case["prompt"]
    vocab = _seq_config(case)["vocab"] if "width" in case and case["kind"] != "ops" else _sizes(case)["vocab_size"]
    return np.random.default_rng(seed).integers(0, vocab, (case["batch"], n)).astype(np.int32)


def _activations(case, seed):
    """layer_norm's rows, gain and bias; scores; a feed-forward's rows and bias: float32 values that the case's type holds."""
    g, dt = torch.Generator("cuda").manual_seed(seed), _TORCH[case["dtype"]]
    r, d, m, n = case["rows"], case["width"], case["maps"], case["len"]

    def draw_(*shape):
        return torch.randn(shape, generator=g, device="cuda").to(dt)
    return draw_(r, d), draw_(d) * 0.1 + 1, draw_(d), draw_(m, n, n), draw_(r, 4 * d), draw_(4 * d)


def prepare(case, seed):
    gpu.init_backend()
    state = dict(case)
    if case["kind"] == "ops":
        state["tensors"] = [gpu.from_torch(t) for t in _activations(case, seed)]
        return state
    state["model"] = _model(case)
    ids = _ids(case, seed)
    if case["kind"] in ("gedenex", "rurunex"):
        state["ids"] = ids                                # the engine takes token ids from the host
        state["engine"] = state["model"].engine(slots=case["batch"], max_len=case["prompt"] + case["new"] + 1)
        return state
    if case["kind"] == "bert":
        state["ids"] = ids
        return state
    B, T = ids.shape
    state["shape"] = np.zeros((B, T), np.int64)
    state["ids"] = (gpu.from_numpy(ids.reshape(-1)), gpu.from_numpy(np.tile(np.arange(T, dtype=np.int32), B)))
    if case["kind"] == "gpt2_generate":
        state["decoder"] = Gpt2Decoder(state["model"], B, T + case["new"])
    return state


# ── one pass ────────────────────────────────────────────────────────────────
class _Memory:
    """Device memory of a tensor for torch to look at in place."""

    def __init__(self, keep, ptr, shape, strides, size):
        self.keep = keep
        self.__cuda_array_interface__ = {"shape": shape, "strides": tuple(s * size for s in strides), "typestr": "<i%d" % size, "data": (ptr, False), "version": 3}


def _seen(t, shape, dtype):
    """A result [.., columns] as a torch tensor over the same memory; its rows may lie further apart than they are long."""
    L, flat, size, keep = _lib.load(), (int(np.prod(shape[:-1])), shape[-1]), {"float32": 4}.get(dtype, 2), [t]

    def at(x):
        return int(L.applegpu_ffi_device_ptr(x.id) or 0)

    def row(i):
        r = t
        for dim, j in enumerate(np.unravel_index(i, shape[:-1])):
            r = gpu.slice(r, dim, int(j), int(j) + 1)
        keep.append(r)
        return at(r)
    ptr, pitch = at(t), flat[1]
    if not ptr:                                           # rows with a pitch
        ptr = row(0)
        pitch = (row(1) - ptr) // size
    if not ptr:
        raise RuntimeError(L.applegpu_ffi_last_error())
    return torch.as_tensor(_Memory(keep, ptr, flat, (pitch, 1), size), device="cuda").view(_TORCH[dtype])


def run(state):
    kind = state["kind"]
    if kind == "ops":
        x, gain, shift, scores, h, bias = state["tensors"]
        out = [gpu.layer_norm(x, gain, shift, 1e-5), gpu.softmax_causal(scores), gpu.gelu(gpu.add_bias(h, bias))]
        r, d, m, n = state["rows"], state["width"], state["maps"], state["len"]
        return [_seen(t.eval(), s, state["dtype"]) for t, s in zip(out, ((r, d), (m, n, n), (r, 4 * d)))]
    if kind == "bert":
        B, T = state["ids"].shape
        return _seen(gpu.bert_forward(state["model"], state["ids"], compiled=True), (B, T, gpu.BERT_BASE["n_embd"]), state["dtype"])
    if kind in ("gpt2", "gpt2_int8"):
        logits, _ = gpu.gpt2_forward(state["model"], state["shape"], device_ids=state["ids"], compiled=True)
        return _seen(logits, (state["batch"], state["seq"], _sizes(state)["vocab_size"]), state["dtype"])
    if kind == "gpt2_generate":
        logits, kv = gpu.gpt2_forward(state["model"], state["shape"], device_ids=state["ids"], last_only=True, compiled=True)
        first = gpu.argmax(logits)
        state["decoder"].prefill(kv, first, state["prompt"])
        rest = state["decoder"].steps(state["new"] - 1)
        return {"logits": logits.to_numpy(), "first": first.to_numpy(), "rest": rest}
    eng, n = state["engine"], state["batch"]
    eng.reset(0, n)
    logits, tok = eng.forward(state["ids"], pick=True)
    if not state["new"]:
        return {"logits": logits, "tokens": tok}
    if state["each"]:
        all_logits, tokens = [logits], [tok]
        for _ in range(state["new"]):
            logits, tok = eng.forward(tok[:, None], pick=True)
            all_logits.append(logits)
            tokens.append(tok)
        return {"logits": np.stack(all_logits), "tokens": np.stack(tokens)}
    tokens = eng.decode(state["new"], 0, n)
    after, last = eng.forward(tokens[-1][:, None], pick=True)
    return {"logits": np.stack([logits, after]), "tokens": np.concatenate([tok[None], tokens, last[None]])}


# ── what a pass has to do ───────────────────────────────────────────────────
def work(case):
    kind, e = case["kind"], {"float32": 4}.get(case["dtype"], 2)
    if kind == "ops":
        r, d, m, n = case["rows"], case["width"], case["maps"], case["len"]
        return {"bytes": e * (2 * r * d + 2 * d + m * (n * (n + 1) // 2 + n * n) + 8 * r * d + 4 * d), "flops": 0}
    if "seq" in case or kind == "gpt2_generate":
        c = _sizes(case)
        d, L, V = c["n_embd"], c["n_layer"], c["vocab_size"]
        B, T = case["batch"], case.get("seq", case.get("prompt"))
        per_token = 24 * d * d * L
        if kind == "bert":
            return {"bytes": e * (12 * d * d * L + B * T * d), "flops": B * T * (per_token + 4 * T * d * L)}
        weights = (1 if kind == "gpt2_int8" else e) * 12 * d * d * L + e * V * d
        if kind != "gpt2_generate":
            return {"bytes": weights + e * B * T * V, "flops": B * T * (per_token + 2 * d * V) + 2 * B * T * (T + 1) * d * L}
        n, steps = case["new"], case["new"] - 1           # every step reads the weights and the keys and values so far
        cache = 2 * e * L * B * d * (steps * T + steps * (steps + 1) // 2)
        return {"bytes": (1 + steps) * weights + cache, "flops": B * (T * per_token + 2 * d * V) + 2 * B * T * (T + 1) * d * L + steps * B * (per_token + 2 * d * V + 4 * T * d * L)}
    cfg = _seq_config(case)
    W, V, B, P, n = case["width"], cfg["vocab"], case["batch"], case["prompt"], case["new"] + bool(case["new"] and not case["each"])
    steps = n
    weights = mixing = state = cache = 0
    loop = cfg.get("loop")
    for i, layer in enumerate(cfg["layers"]):
        times = loop["times"] if loop and loop["start"] <= i < loop["stop"] else 1
        m, t = layer["mixer"], layer["type"]
        H, dim, vdim = m["heads"], m["dim"], m["vdim"]
        mat = 3 * W * layer["mlp"]["ff"] + W * H * vdim
        if t == "latent_attention":
            r = m["kv_rank"]
            mat += W * (H * (dim + m["rot_dim"]) + r + m["rot_dim"]) + r * H * (dim + vdim)
            mixing += times * H * (P + 1) * (dim + m["rot_dim"] + vdim)          # the unmasked half, per token
            cache += times * (r + m["rot_dim"])
        elif t == "attention":
            G, win = m["kv_heads"], min(m["mask"]["size"], P)
            mat += W * H * dim + (0 if m.get("kv_from") is not None else W * G * (dim + vdim))
            mixing += 2 * H * min((P + 1) / 2, win) * (dim + vdim)
            cache += G * (dim + vdim) * min(1.0, win / P)
        else:
            G = m.get("kv_heads", H)
            mat += W * (2 * G * dim + H * vdim + (128 if t == "channel_delta" else H * vdim))
            mixing += times * 4 * H * dim * vdim
            state += times * H * dim * vdim * 8                                  # read and written, 32 bits
        weights += mat * times
    flops = B * P * (2 * weights + mixing) + B * (2 * V * W) + steps * B * (2 * weights + mixing + 2 * V * W)
    return {"bytes": (1 + steps) * (e * (weights + V * W) + B * state) + steps * B * cache * P * e + 4 * B * V * (1 + (steps if case["each"] else bool(steps))), "flops": flops}


def tolerance(case):
    """About four times what the results differ from 64 bits by: 0.009 to 0.014 over the 12 to 36 layers of the 16-bit transformers,
    0.002 to 0.006 in the sequence models, whose stream is float32, an eighth of that in float16, 3.5e-6 in float32; 0.0026 for one op."""
    dt = case["dtype"]
    if case["kind"] == "ops":
        return {"rel": {"float32": 1e-5, "float16": 1.5e-3}.get(dt, 1e-2), "max": {"float32": 1e-4, "float16": 0.01}.get(dt, 0.05)}
    if dt == "float32":
        return {"rel": 2e-5, "max": 2e-4}
    if dt == "float16":
        return {"rel": 5e-3, "max": 0.05}
    return {"rel": 0.02 if case["kind"] in ("gedenex", "rurunex") else 0.03, "max": 0.2}


# ── the same in 64 bits ─────────────────────────────────────────────────────
def _causal_attention(q, k, v):
    T, S = q.shape[-2], k.shape[-2]
    out = torch.empty(*q.shape[:-1], v.shape[-1], dtype=q.dtype, device=q.device)
    for b in range(q.shape[0]):
        s = q[b] @ k[b].transpose(-1, -2) / math.sqrt(q.shape[-1])
        s = s.masked_fill(torch.ones(T, S, dtype=torch.bool, device=q.device).triu(S - T + 1), float("-inf"))
        out[b] = torch.softmax(s, -1) @ v[b]
    return out


def _as_int8(w):
    """A [in, out] weight through one int8 scale per output, as 64-bit numbers."""
    top = w.abs().amax(0, keepdim=True)
    scale = torch.where(top > 0, top / 127.0, torch.ones_like(top))
    q = w / scale
    return (torch.sign(q) * torch.floor(q.abs() + 0.5)).clamp(-128, 127).double() * scale.double()


def _gpt2_exact(case, ids):
    c, w = _sizes(case), _transformer_weights(case)
    d, H = c["n_embd"], c["n_head"]
    for k in list(w):
        w[k] = _as_int8(w[k]) if case["kind"] == "gpt2_int8" and k.endswith((".c_attn.weight", ".c_fc.weight", ".c_proj.weight")) else w[k].double()
    B, T = ids.shape
    p = "transformer."
    x = w[p + "wte.weight"][ids] + w[p + "wpe.weight"][torch.arange(T, device="cuda")]
    for i in range(c["n_layer"]):
        h = f"{p}h.{i}."
        y = F.layer_norm(x, (d,), w[h + "ln_1.weight"], w[h + "ln_1.bias"], 1e-5) @ w[h + "attn.c_attn.weight"] + w[h + "attn.c_attn.bias"]
        q, k, v = (t.reshape(B, T, H, d // H).transpose(1, 2) for t in y.split(d, -1))
        a = _causal_attention(q, k, v).transpose(1, 2).reshape(B, T, d)
        x = x + a @ w[h + "attn.c_proj.weight"] + w[h + "attn.c_proj.bias"]
        y = F.layer_norm(x, (d,), w[h + "ln_2.weight"], w[h + "ln_2.bias"], 1e-5) @ w[h + "mlp.c_fc.weight"] + w[h + "mlp.c_fc.bias"]
        x = x + F.gelu(y, approximate="tanh") @ w[h + "mlp.c_proj.weight"] + w[h + "mlp.c_proj.bias"]
    return F.layer_norm(x, (d,), w[p + "ln_f.weight"], w[p + "ln_f.bias"], 1e-5), w[p + "wte.weight"]


def _bert_exact(case, ids):
    c = _sizes(case)
    w = {k: t.double() for k, t in _transformer_weights(case).items()}
    d, H, eps = c["n_embd"], c["n_head"], c["eps"]
    out = []
    for part in ids.split(32):
        B, T = part.shape
        x = w["embeddings.word_embeddings.weight"][part] + w["embeddings.position_embeddings.weight"][:T] + w["embeddings.token_type_embeddings.weight"][0]
        x = F.layer_norm(x, (d,), w["embeddings.LayerNorm.weight"], w["embeddings.LayerNorm.bias"], eps)
        for i in range(c["n_layer"]):
            p = f"encoder.layer.{i}."

            def lin(t, n):
                return F.linear(t, w[p + n + ".weight"], w[p + n + ".bias"])
            q, k, v = (lin(x, "attention.self." + n).reshape(B, T, H, d // H).transpose(1, 2) for n in ("query", "key", "value"))
            a = (torch.softmax(q @ k.transpose(-1, -2) / math.sqrt(d // H), -1) @ v).transpose(1, 2).reshape(B, T, d)
            x = F.layer_norm(x + lin(a, "attention.output.dense"), (d,), w[p + "attention.output.LayerNorm.weight"], w[p + "attention.output.LayerNorm.bias"], eps)
            x = F.layer_norm(x + lin(F.gelu(lin(x, "intermediate.dense")), "output.dense"), (d,), w[p + "output.LayerNorm.weight"], w[p + "output.LayerNorm.bias"], eps)
        out.append(x)
    return torch.cat(out).reshape(-1, d)


def _rms(x, eps):
    return x / torch.sqrt(x.square().mean(-1, keepdim=True) + eps)


def _angles(rot, T):
    """cos and sin [T, pairs] of YaRN-scaled rotary positions."""
    n, i = rot["dims"], torch.arange(rot["dims"] // 2, dtype=torch.float64, device="cuda")
    freq, s = float(rot["base"]) ** (-2.0 * i / n), rot["scaling"]

    def pair(turns):
        return n * math.log(s["original"] / (2 * math.pi * turns)) / (2 * math.log(rot["base"]))
    lo, hi = max(math.floor(pair(s["fast"])), 0), min(math.ceil(pair(s["slow"])), n - 1)
    ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0, 1)
    a = torch.arange(T, dtype=torch.float64, device="cuda")[:, None] * (freq / s["factor"] * ramp + freq * (1 - ramp))
    amp = 0.1 * math.log(s["factor"]) + 1.0
    return torch.cos(a) * amp, torch.sin(a) * amp


def _attend(q, k, v, scale, window=0, cap=0.0):
    """q [B, T, H, d], k and v [B, T, G, ..]."""
    T, H = q.shape[1], q.shape[2]
    t = torch.arange(T, device="cuda")
    hidden = t[None, :] > t[:, None]
    if window:
        hidden = hidden | (t[None, :] <= t[:, None] - window)
    out = []
    for b in range(q.shape[0]):
        kk, vv = (x[b].repeat_interleave(H // x.shape[2], 1).transpose(0, 1) for x in (k, v))
        s = q[b].transpose(0, 1) @ kk.transpose(-1, -2) * scale
        s = cap * torch.tanh(s / cap) if cap else s
        out.append((torch.softmax(s.masked_fill(hidden, float("-inf")), -1) @ vv).transpose(0, 1).reshape(T, -1))
    return torch.stack(out)


def _mlstm(h, w, p, m, eps):
    B, T, _ = h.shape
    H, d, e, cap = m["heads"], m["dim"], m["vdim"], m["gate_cap"]
    q, k, v = (h @ w[p + n].T for n in "qkv")
    q, k, v = q.reshape(B, T, H, d) * d ** -0.5, k.reshape(B, T, H, d), v.reshape(B, T, H, e)
    li = cap * torch.tanh((h @ w[p + "i"].T + w[p + "i.b"]) / cap)
    lf = F.logsigmoid(cap * torch.tanh((h @ w[p + "f"].T + w[p + "f.b"]) / cap))
    S, n, mx = h.new_zeros(B, H, d, e), h.new_zeros(B, H, d), h.new_zeros(B, H)
    out = h.new_empty(B, T, H, e)
    for t in range(T):
        mn = torch.maximum(lf[:, t] + mx, li[:, t])
        keep, kt = torch.exp(lf[:, t] + mx - mn), k[:, t] * torch.exp(li[:, t] - mn)[..., None]
        S.mul_(keep[..., None, None]).addcmul_(kt[..., None], v[:, t][:, :, None])
        n.mul_(keep[..., None]).add_(kt)
        den = torch.maximum((n * q[:, t]).sum(-1).abs(), torch.exp(-mn)) + 1e-6
        out[:, t] = (q[:, t][:, :, None] @ S)[:, :, 0] / den[..., None]
        mx = mn
    return _rms(out, eps).reshape(B, T, H * e) * w[p + "norm"] * torch.sigmoid(h @ w[p + "g"].T)


def _latent(h, w, p, m, eps):
    B, T, _ = h.shape
    H, d, rd, e, r = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
    c, s = _angles(m["rot"], T)

    def turn(x):                                          # neighbouring entries are a pair; x [B, T, heads, rd]
        u, v = x[..., 0::2], x[..., 1::2]
        return torch.stack([u * c[:, None] - v * s[:, None], v * c[:, None] + u * s[:, None]], -1).reshape(x.shape)
    q, down = (h @ w[p + "q"].T).reshape(B, T, H, d + rd), h @ w[p + "dkv"].T
    lat = _rms(down[..., :r], eps) * w[p + "dkv.norm"]
    kr = turn(down[..., r:].reshape(B, T, 1, rd)).expand(B, T, H, rd)
    q, k = torch.cat([q[..., :d], turn(q[..., d:])], -1), torch.cat([(lat @ w[p + "uk"].T).reshape(B, T, H, d), kr], -1)
    return _attend(q, k, (lat @ w[p + "uv"].T).reshape(B, T, H, e), m["scale"])


def _decayed(q, k, v, decay, beta):
    """Matrix states with a decay per key channel, with the delta rule where beta is given."""
    B, T, H, d = q.shape
    S, out = q.new_zeros(B, H, d, v.shape[-1]), torch.empty_like(v)
    for t in range(T):
        S.mul_(decay[:, t][..., None])
        u = v[:, t] if beta is None else (v[:, t] - (k[:, t][:, :, None] @ S)[:, :, 0]) * beta[:, t][..., None]
        S.addcmul_(k[:, t][..., None], u[:, :, None])
        out[:, t] = (q[:, t][:, :, None] @ S)[:, :, 0]
    return out


def _gla(h, w, p, m, eps):
    B, T, _ = h.shape
    H, d, e = m["heads"], m["dim"], m["vdim"]
    q, k, v = (h @ w[p + n].T for n in "qkv")
    decay = torch.exp(F.logsigmoid(h @ w[p + "a1"].T @ w[p + "a2"].T + w[p + "a2.b"]) / m["tau"]).reshape(B, T, H, d)
    o = _decayed(q.reshape(B, T, H, d) * d ** -0.5, k.reshape(B, T, H, d), v.reshape(B, T, H, e), decay, None)
    return (_rms(o, eps) * w[p + "norm"]).reshape(B, T, H * e) * F.silu(h @ w[p + "g"].T)


def _delta(h, w, p, m, eps):
    B, T, _ = h.shape
    H, G, d, e = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    parts = []
    for n in "qkv":
        taps = w[p + n + ".conv"]
        x = F.pad(h @ w[p + n].T, (0, 0, taps.shape[1] - 1, 0))
        parts.append(F.silu(sum(x[:, i:i + T] * taps[:, i] for i in range(taps.shape[1]))))

    def unit(x):
        x = x.reshape(B, T, G, d)
        return (x / torch.sqrt(x.square().sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 2)
    step = F.softplus(h @ w[p + "a1"].T @ w[p + "a2"].T + w[p + "dt_bias"]).reshape(B, T, H, d)
    decay = torch.exp(-torch.exp(w[p + "A_log"])[:, None] * step)
    o = _decayed(unit(parts[0]) * d ** -0.5, unit(parts[1]), parts[2].reshape(B, T, H, e), decay, torch.sigmoid(h @ w[p + "b"].T))
    return (_rms(o, eps) * w[p + "norm"]).reshape(B, T, H * e) * torch.sigmoid(h @ w[p + "g1"].T @ w[p + "g2"].T)


def _grouped(h, w, p, m, eps, source):
    B, T, _ = h.shape
    H, G, d, e = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    c, s = _angles(m["rot"], T)

    def turn(x):                                          # halves are a pair
        u, v = x.chunk(2, -1)
        return torch.cat([u * c[:, None] - v * s[:, None], v * c[:, None] + u * s[:, None]], -1)
    q = turn(_rms((h @ w[p + "q"].T).reshape(B, T, H, d), eps) * w[p + "q.norm"])
    if source is None:
        source = turn(_rms((h @ w[p + "k"].T).reshape(B, T, G, d), eps) * w[p + "k.norm"]), (h @ w[p + "v"].T).reshape(B, T, G, e)
    return _attend(q, *source, m["scale"], m["mask"]["size"], m["softcap"]), source


def _seq_exact(case, ids, rows):
    """Logits [len(rows), batch, vocab] of the tokens `ids` at the positions `rows`."""
    cfg, dt = _seq_config(case), _TORCH[case["dtype"]]
    w = {}
    for k, a in _seq_weights(case).items():
        t = torch.from_numpy(a).cuda()
        w[k] = (t.to(dt) if t.ndim == 2 and not k.endswith((".conv", "loop.step")) else t).double()
    eps, layers = cfg["norm"]["eps"], cfg["layers"]
    emb = w["embed"][ids]
    if case["kind"] == "gedenex":
        lo, hi, times = cfg["loop"]["start"], cfg["loop"]["stop"], cfg["loop"]["times"]
        x = emb
        for i, turn in [(i, None) for i in range(lo)] + [(i, t) for t in range(times) for i in range(lo, hi)] + [(i, None) for i in range(hi, len(layers))]:
            if turn is not None and i == lo:
                x = x + w["loop.step"][turn] + (emb if turn else 0)
            p, m, mlp = f"l{i}.", layers[i]["mixer"], layers[i]["mlp"]
            y = (_mlstm if layers[i]["type"] == "mlstm" else _latent)(_rms(x, eps) * w[p + "norm1"], w, p + "mix.", m, eps) @ w[p + "mix.o"].T
            h = _rms(x, eps) * w[p + "norm2"]
            g, u = (h @ w[p + "mlp.gate"].T).clamp(max=mlp["limit"]), (h @ w[p + "mlp.up"].T).clamp(-mlp["limit"], mlp["limit"])
            x = x + y + (g * torch.sigmoid(1.702 * g) * (u + 1)) @ w[p + "mlp.down"].T
        return ((_rms(x, eps) * w["final.norm"])[:, rows] @ w["head"].T).transpose(0, 1)
    x, kept = emb * cfg["embedding"]["scale"], {}
    for i, layer in enumerate(layers):
        p, m = f"l{i}.", layer["mixer"]
        h = _rms(x, eps) * (1 + w[p + "norm1"])
        if layer["type"] == "attention":
            y, kept[i] = _grouped(h, w, p + "mix.", m, eps, kept.get(m.get("kv_from")))
        else:
            y = (_gla if layer["type"] == "gla" else _delta)(h, w, p + "mix.", m, eps)
        x = x + _rms(y @ w[p + "mix.o"].T, eps) * (1 + w[p + "norm1b"])
        h = _rms(x, eps) * (1 + w[p + "norm2"])
        y = (F.silu(h @ w[p + "mlp.gate"].T) * (h @ w[p + "mlp.up"].T)) @ w[p + "mlp.down"].T
        x = x + _rms(y, eps) * (1 + w[p + "norm2b"])
    return ((_rms(x, eps) * (1 + w["final.norm"]))[:, rows] @ w["head"].T * cfg["logit_scale"]).transpose(0, 1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "ops":
        x, gain, shift, scores, h, bias = (t.double() for t in _activations(case, seed))
        n = case["len"]
        scores.masked_fill_(torch.ones(n, n, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
        return [F.layer_norm(x, (case["width"],), gain, shift, 1e-5), torch.softmax(scores, -1).reshape(-1, n), F.gelu(h + bias, approximate="tanh")]
    ids = torch.from_numpy(_ids(case, seed)).long().cuda()
    if kind == "bert":
        return _bert_exact(case, ids)
    if kind in ("gpt2", "gpt2_int8"):
        x, head = _gpt2_exact(case, ids)
        return x.reshape(-1, x.shape[-1]) @ head.T
    if kind == "gpt2_generate":                          # tokens are checked between two versions, the prompt's logits here
        x, head = _gpt2_exact(case, ids)
        return {"logits": x[:, -1] @ head.T, "first": None, "rest": None}
    P, n = case["prompt"], case["new"]
    follow = torch.from_numpy(_next_of(_seq_config(case)["vocab"])).cuda()
    steps = n + (0 if case["each"] or not n else 1)
    seq = ids
    for _ in range(steps):
        seq = torch.cat([seq, follow[seq[:, -1:]]], 1)
    rows = list(range(P - 1, P + n)) if case["each"] else [P - 1] + ([P + n] if n else [])
    logits = _seq_exact(case, seq, rows)
    return {"logits": logits if n else logits[0], "tokens": None}
