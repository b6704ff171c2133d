"""Performance cases of dnet_b200: what a serving program has it do, through its public entry points.

Two families of entry points exist, and both are measured.

Llama-like shards (``LlamaRingModel`` / ``Qwen2RingModel`` / ``MixtralRingModel``, libdnet_b200.so):
  * ``layer``   one decoder layer on a chunk of tokens behind a context (``apply_single_layer``): the unit of which a shard
                of any number of layers is made.  Few tokens (a user's turn, a draft), short and ragged prompts, chunks
                of long prompts; 16-bit and quantised KV caches; dense and sparse-expert feed-forwards.
  * ``prompt``  a whole prompt through several layers and the head (``embed`` + ``window_forward`` + ``head_logits``).
  * ``token``   one decoded token through the fused step (``dn_shard_step``), with the head.
Layer-list models (``SequenceBatcher`` over ``SeqMixRingModel``, libdnet_b200_seq.so):
  * ``batch``   one step that brings ragged prompts of several requests (admit, step, finish).
  * ``turns``   several requests decoded together: a short prompt each, then steps of one token per request.

Sizes are those of the repository's benchmarks: Llama-3-8B, Qwen2.5-32B, Mixtral-8x7B and the layer-list sizes "1k" - "4k".
Weights are random with the scales of trained ones (projections N(0, 1 / fan_in)), tokens and activations are synthetic.
Routers are decisive, as trained ones are: a token's input leans towards the experts that are to be its own.
"""
from __future__ import annotations

import ctypes
import math

import torch

from dnet_b200 import _cabi
from dnet_b200.core.models.llama import LlamaRingModel, MixtralRingModel, Qwen2RingModel
from dnet_b200.core.models.seqmix import BokenexRingModel, MoputarRingModel
from dnet_b200.shard.batching import SequenceBatcher

DEV = "cuda"
BF = torch.bfloat16
F64 = torch.float64
HD = 128

LLAMA = {
    "llama8b": dict(hidden_size=4096, num_attention_heads=32, num_key_value_heads=8, head_dim=HD, intermediate_size=14336,
                    vocab_size=128256, rms_norm_eps=1e-5, rope_theta=500000.0, model_type="llama"),
    "qwen32b": dict(hidden_size=5120, num_attention_heads=40, num_key_value_heads=8, head_dim=HD, intermediate_size=27648,
                    vocab_size=152064, rms_norm_eps=1e-6, rope_theta=1000000.0, model_type="qwen2"),
    "mixtral8x7b": dict(hidden_size=4096, num_attention_heads=32, num_key_value_heads=8, head_dim=HD, intermediate_size=14336,
                        vocab_size=32000, rms_norm_eps=1e-5, rope_theta=1000000.0, model_type="mixtral", num_local_experts=8,
                        num_experts_per_tok=2),
}
CLASSES = {"llama": LlamaRingModel, "qwen2": Qwen2RingModel, "mixtral": MixtralRingModel}
SEQ_SIZES = {
    "1k": dict(width=1024, heads=8, kv_heads=2, ff=4096),
    "2k": dict(width=2048, heads=16, kv_heads=4, ff=8192),
    "4k": dict(width=4096, heads=32, kv_heads=8, ff=14336),
}
SEQ_VOCAB = 32768


def listed():
    return [
        # one decoded token, early in a conversation: the headline workload (a shard of 8 layers and the head)
        dict(name="token", kind="token", model="llama8b", layers=8, context=512, kv_bits=0),
        # one decoded token deep in a document, with the cache that requests get by default (8 bit)
        dict(name="token_q8_deep", kind="token", model="llama8b", layers=2, context=8192, kv_bits=8),
        # a handful of tokens behind a context: the end of a chunked prompt, a short follow-up, a draft to be checked
        dict(name="layer_3_tokens", kind="layer", model="llama8b", context=256, tokens=3, kv_bits=0),
        # a question
        dict(name="layer_short_prompt", kind="layer", model="llama8b", context=0, tokens=45, kv_bits=0),
        # a page or two of text, first to last: embedding, layers, head
        dict(name="prompt_2048", kind="prompt", model="llama8b", layers=2, tokens=2048, kv_bits=0),
        # one chunk of a long document, other head counts (groups of 5) and q / k / v biases
        dict(name="layer_long_chunk", kind="layer", model="qwen32b", context=8192, tokens=512, kv_bits=0),
        # a ragged prompt behind earlier turns, with the default 8-bit cache
        dict(name="layer_q8_prompt", kind="layer", model="llama8b", context=1024, tokens=777, kv_bits=8),
        # sparse experts: one decoded token, and a prompt
        dict(name="experts_token", kind="layer", model="mixtral8x7b", context=512, tokens=1, kv_bits=0),
        dict(name="experts_prompt", kind="layer", model="mixtral8x7b", context=0, tokens=500, kv_bits=0),
        # layer-list models: prompts of four requests in one step (block-masked attention, shared keys, delta rule, 4 streams)
        dict(name="batch_moputar", kind="batch", family="moputar", size="4k", sequences=4, tokens=2048),
        # ... and four requests answered token by token
        dict(name="turns_moputar", kind="turns", family="moputar", size="4k", sequences=4, prompt=24, steps=12),
        # sigmoid attention beside routed and dense feed-forwards, three requests of a smaller model
        dict(name="batch_bokenex", kind="batch", family="bokenex", size="2k", sequences=3, tokens=1000),
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["token", "layer", "layer", "layer", "layer", "prompt", "batch", "batch", "turns"])
    if kind == "token":
        return dict(kind=kind, model="llama8b", layers=rng.randint(1, 8), context=_log(rng, 8, 8000), kv_bits=rng.choice([0, 0, 8, 4]))
    if kind == "layer":
        model = rng.choice(["llama8b", "llama8b", "qwen32b", "mixtral8x7b"])
        bits = rng.choice([0, 0, 8, 4]) if model == "llama8b" else 0
        return dict(kind=kind, model=model, context=_log(rng, 1, 8192) - 1, tokens=_log(rng, 1, 500 if model == "mixtral8x7b" else 1500), kv_bits=bits)
    if kind == "prompt":
        return dict(kind=kind, model="llama8b", layers=rng.randint(1, 2), tokens=_log(rng, 5, 2048), kv_bits=rng.choice([0, 0, 8]))
    family = rng.choice(["moputar", "bokenex"])
    size = rng.choice(["1k", "2k", "4k"])
    if kind == "batch":
        n = rng.randint(1, 4)
        return dict(kind=kind, family=family, size=size, sequences=n, tokens=max(2 * n, _log(rng, 20, 2048)))
    return dict(kind=kind, family=family, size=size, sequences=rng.randint(1, 4), prompt=_log(rng, 4, 60), steps=rng.randint(4, 12))


# -- inputs ------------------------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _normal(g, shape, std=1.0, mean=0.0):
    return torch.empty(shape, dtype=torch.float32, device=DEV).normal_(mean, std, generator=g).to(BF)


def _llama_config(case):
    cfg = dict(LLAMA[case["model"]])
    cfg.update(num_hidden_layers=case.get("layers", 1), tie_word_embeddings=False, torch_dtype="bfloat16")
    return cfg


def _llama_weights(cfg, layers, g, with_api):
    H, nh, nk, F = cfg["hidden_size"], cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["intermediate_size"]
    w = {}
    for i in range(layers):
        p = f"model.layers.{i}."
        for name, rows, cols in (("q", nh * HD, H), ("k", nk * HD, H), ("v", nk * HD, H), ("o", H, nh * HD)):
            w[f"{p}self_attn.{name}_proj.weight"] = _normal(g, (rows, cols), cols ** -0.5)
            if cfg["model_type"] == "qwen2" and name != "o":
                w[f"{p}self_attn.{name}_proj.bias"] = _normal(g, (rows,), 0.3)
        for name in ("input_layernorm", "post_attention_layernorm"):
            w[f"{p}{name}.weight"] = _normal(g, (H,), 0.1, 1.0)
        mlp = (("gate", "w1", F, H), ("up", "w3", F, H), ("down", "w2", H, F))
        if cfg.get("num_local_experts"):
            w[f"{p}block_sparse_moe.gate.weight"] = _normal(g, (cfg["num_local_experts"], H), H ** -0.5)
            for e in range(cfg["num_local_experts"]):
                for _, name, rows, cols in mlp:
                    w[f"{p}block_sparse_moe.experts.{e}.{name}.weight"] = _normal(g, (rows, cols), cols ** -0.5)
        else:
            for name, _, rows, cols in mlp:
                w[f"{p}mlp.{name}_proj.weight"] = _normal(g, (rows, cols), cols ** -0.5)
    if with_api:
        w["model.embed_tokens.weight"] = _normal(g, (cfg["vocab_size"], H))
        w["model.norm.weight"] = _normal(g, (H,), 0.1, 1.0)
        w["lm_head.weight"] = _normal(g, (cfg["vocab_size"], H), H ** -0.5)
    return w


def _lean(g, x, router, top, low):
    """x [T, W] and, for each row, `top` distinct experts towards whose router rows it leans"""
    pick = torch.rand(x.shape[0], router.shape[0], generator=g, device=DEV).argsort(1)[:, :top]
    x = x.float()
    for j in range(top):
        x += (low + 1.2 * j) * router[pick[:, j]].float()
    return x.to(BF)


def _llama_inputs(case, seed):
    """config, weights, and the activations (``layer``) or token ids (``prompt``, ``token``) of context and call together"""
    g = _gen(seed)
    cfg = _llama_config(case)
    with_api = case["kind"] != "layer"
    w = _llama_weights(cfg, cfg["num_hidden_layers"], g, with_api)
    n = case.get("context", 0) + case.get("tokens", 1)
    if with_api:
        return cfg, w, torch.randint(0, cfg["vocab_size"], (n,), generator=g, device=DEV, dtype=torch.int32)
    x = _normal(g, (n, cfg["hidden_size"]))
    if cfg.get("num_local_experts"):
        x = _lean(g, x, w["model.layers.0.block_sparse_moe.gate.weight"], cfg["num_experts_per_tok"], 5.5)
    return cfg, w, x


def _ragged(case):
    """lengths of a batch's prompts: of unlike size, together `tokens`"""
    n, total = case["sequences"], case["tokens"]
    parts = [1 + (7 * i + 3) % 5 for i in range(n)]
    lens = [max(1, total * p // sum(parts)) for p in parts]
    lens[0] += total - sum(lens)
    return lens


def _seq_config(case):
    sz = SEQ_SIZES[case["size"]]
    W, H, G, ff = sz["width"], sz["heads"], sz["kv_heads"], sz["ff"]
    base = {"heads": H, "kv_heads": G, "dim": HD, "vdim": HD, "conv": 4}
    dense = {"kind": "dense", "ff": ff}
    if case["family"] == "moputar":
        att = {**base, "scale": HD ** -0.5, "rot": {"base": 500000.0, "dims": 64}, "mask": {"size": 1024}}
        layers = [{"type": "attention", "mixer": att, "mlp": dense},
                  {"type": "attention", "mixer": {**att, "kv_from": 0}, "mlp": dense},
                  {"type": "delta", "mixer": base, "mlp": dense}]
        return {"architecture": "Moputar", "vocab": SEQ_VOCAB, "width": W, "streams": 4, "norm": {"eps": 1e-5}, "embedding": {"scale": 1.0},
                "layers": layers}
    mx = {**base, "scale": HD ** -0.5, "mask": {"size": 1024}}
    moe = {"kind": "moe", "router": {"experts": 16, "top": 4, "scale": 2.0}, "expert": {"ff": ff // 4}}
    return {"architecture": "Bokenex", "vocab": SEQ_VOCAB, "width": W, "norm": {"eps": 1e-5}, "residual_mult": 0.4, "max_positions": 4096,
            "layers": [{"type": "attention", "mixer": mx, "mlp": moe}, {"type": "attention", "mixer": mx, "mlp": dense}]}


def _seq_shapes(cfg):
    """name -> shape of a checkpoint, as the families' files name them"""
    W, V, S = cfg["width"], cfg["vocab"], int(cfg.get("streams", 0))
    bok = cfg["architecture"] == "Bokenex"
    out = {"embed": (V, W), "head": (V, W), "final.norm": () if bok else (W,)}
    if bok:
        out["pos"] = (cfg["max_positions"], W)
    for i, L in enumerate(cfg["layers"]):
        p, mx, mlp = f"l{i}.", L["mixer"], L["mlp"]
        H, G, d, J = mx["heads"], mx["kv_heads"], mx["dim"], mx["conv"]
        att = L["type"] == "attention"
        own = mx.get("kv_from") is None
        rows = {"q": (H if att else G) * d, "k": G * d, "v": (G if att else H) * d}
        out[p + "norm1"] = () if bok else (W,)
        for c in "qkv" if own else "q":
            out[f"{p}mix.{c}"], out[f"{p}mix.{c}.conv"] = (rows[c], W), (rows[c], J)
        out[p + "mix.o"] = (W, H * d)
        if bok:
            out[p + "mix.q.norm"] = out[p + "mix.k.norm"] = (d,)
            out[p + "mix.r1"] = out[p + "mix.r2"] = out[p + "mix.pb"] = (H,)
        elif att:
            out[p + "mix.q.norm"] = (rows["q"],)
            if own:
                out[p + "mix.k.norm"] = (rows["k"],)
        else:
            out[p + "mix.a"] = out[p + "mix.b"] = (H, W)
            out[p + "mix.g"] = (H * d, W)
            out[p + "mix.A_log"] = out[p + "mix.dt_bias"] = (H,)
            out[p + "mix.norm"] = (d,)
        if not bok:
            out[p + "norm2"] = (W,)
        if mlp["kind"] == "moe":
            out[p + "mlp.router"] = (mlp["router"]["experts"], W)
            for e in range(mlp["router"]["experts"]):
                out[f"{p}mlp.e{e}.up"], out[f"{p}mlp.e{e}.down"] = (mlp["expert"]["ff"], W), (W, mlp["expert"]["ff"])
        else:
            out[p + "mlp.up"], out[p + "mlp.down"] = (mlp["ff"], W), (W, mlp["ff"])
            if not bok:
                out[p + "mlp.gate"] = (mlp["ff"], W)
        for q in ("hc1", "hc2") if S else ():
            out[f"{p}{q}.in"] = out[f"{p}{q}.out"] = (S,)
            out[f"{p}{q}.mix"] = (S, S)
    return out


def _seq_weights(cfg, g):
    S = int(cfg.get("streams", 0))
    bok = cfg["architecture"] == "Bokenex"
    w = {}
    for name, shape in _seq_shapes(cfg).items():
        leaf = name.split(".", 1)[-1] if name[0] == "l" and name[1].isdigit() else name
        if leaf in ("norm1", "norm2", "final.norm"):
            t = _normal(g, shape, 0.1, 1.0 if bok else 0.0)
        elif leaf in ("mix.q.norm", "mix.k.norm", "mix.norm"):
            t = _normal(g, shape, 0.1, 1.0)
        elif leaf.endswith(".conv"):
            t = _normal(g, shape, 0.5)
        elif leaf == "mix.A_log":
            t = _normal(g, shape, 0.5, -1.0)
        elif leaf == "mix.dt_bias":
            t = _normal(g, shape, 0.5)
        elif leaf in ("mix.r1", "mix.r2"):
            t = _normal(g, shape, 0.1, 0.4).abs()
        elif leaf == "mix.pb":
            t = _normal(g, shape, 0.5, -4.0)
        elif leaf.endswith(".in"):
            t = _normal(g, shape, 0.1, 1.0 / S)
        elif leaf.endswith(".out"):
            t = _normal(g, shape, 0.1, 0.5)
        elif leaf.endswith(".mix"):
            t = (torch.eye(S, device=DEV) * 0.9 + 0.1 / S).to(BF)
        elif name in ("embed", "pos"):
            t = _normal(g, shape, 1.0 if name == "embed" else 0.3)
        else:
            t = _normal(g, shape, shape[-1] ** -0.5)
        w[name] = t
    if bok:
        w["embed"] = _lean(g, w["embed"], w["l0.mlp.router"], cfg["layers"][0]["mlp"]["router"]["top"], 5.5)
    return w


def _seq_inputs(case, seed):
    """config, weights, and per request its tokens (``turns``: prompt and answer together)"""
    g = _gen(seed)
    cfg = _seq_config(case)
    w = _seq_weights(cfg, g)
    if case["kind"] == "batch":
        lens = _ragged(case)
    else:
        lens = [max(1, case["prompt"] - 3 * i) + case["steps"] for i in range(case["sequences"])]
    toks = [torch.randint(0, SEQ_VOCAB, (n,), generator=g, device=DEV).tolist() for n in lens]
    return cfg, w, toks


# -- what is timed -------------------------------------------------------------------------------------------------------
def prepare(case, seed):
    if "model" in case:
        cfg, w, given = _llama_inputs(case, seed)
        n, ctx = len(given), case.get("context", 0)
        layers = list(range(cfg["num_hidden_layers"]))
        model = CLASSES[cfg["model_type"]](cfg, layers, kv_pool_pages=(n + 63) // 64 + 1, kv_bits=case["kv_bits"])
        model.load_weights(w)
        kv = model.make_cache(max_tokens=(n + 63) // 64 * 64)
        st = dict(case=case, model=model, kv=kv, weights=w, layers=layers)
        if ctx:      # the earlier turns or chunks
            x = model.embed(given[:ctx]) if case["kind"] == "token" else given[:ctx].clone()
            model.window_forward(layers, x, kv)
            kv.advance(ctx, torch.cuda.current_stream().cuda_stream)
        st["given"] = given[ctx:].contiguous()
        if case["kind"] == "token":
            st["token"] = int(given[ctx])
            st["array"] = (ctypes.c_int32 * len(layers))(*layers)
        return st
    cfg, w, toks = _seq_inputs(case, seed)
    cls = MoputarRingModel if case["family"] == "moputar" else BokenexRingModel
    total = sum((len(t) + 63) // 64 for t in toks)
    model = cls(cfg, dtype="bfloat16", kv_pool_pages=total + 4, max_seqs=4, max_batch_tokens=2048)
    model.load_weights(w)
    return dict(case=case, model=model, batcher=SequenceBatcher(model), tokens=toks, weights=w)


def run(st):
    case, model = st["case"], st["model"]
    kind = case["kind"]
    if kind == "layer":
        s = torch.cuda.current_stream().cuda_stream
        st["kv"].seek(case["context"], s)
        return model.apply_single_layer(0, st["given"].clone(), st["kv"])
    if kind == "prompt":
        s = torch.cuda.current_stream().cuda_stream
        st["kv"].seek(0, s)
        x = model.embed(st["given"])
        model.window_forward(st["layers"], x, st["kv"])
        return x, model.head_logits(x, want_f32=True, want_bf16=False)[0]
    if kind == "token":
        s = torch.cuda.current_stream().cuda_stream
        x = torch.empty(1, model.hidden_size, dtype=BF, device=DEV)
        logits = torch.empty(model.vocab_size, dtype=torch.float32, device=DEV)
        st["kv"].seek(case["context"], s)
        st["kv"].set_token(st["token"], s)
        _cabi.check(_cabi.load().dn_shard_step(model._h, st["array"], len(st["layers"]), x.data_ptr(), st["kv"]._h, 1, 1, None, None,
                                               logits.data_ptr(), 1, s))
        return x, logits
    b, toks = st["batcher"], st["tokens"]
    if kind == "batch":
        out = b.step([(f"r{i}", t, [len(t) - 1]) for i, t in enumerate(toks)])
    else:
        k = case["steps"]
        out = [b.step([(f"r{i}", t[:-k], [len(t) - k - 1]) for i, t in enumerate(toks)])]
        for j in range(k):
            out.append(b.step([(f"r{i}", [t[len(t) - k + j]], [0]) for i, t in enumerate(toks)]))
    for i in range(len(toks)):
        b.finish(f"r{i}")
    return out


# -- what a pass cannot do without -----------------------------------------------------------------------------------------
def _seen(first, count, block=0):
    """keys that the queries at positions first .. first + count - 1 see together (block: only those of their own block)"""
    if not block:
        return count * first + count * (count + 1) // 2
    return sum(p % block + 1 for p in range(first, first + count))


def work(case):
    if "model" in case:
        cfg = _llama_config(case)
        H, nh, nk, F, E = cfg["hidden_size"], cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["intermediate_size"], cfg.get("num_local_experts", 0)
        L, ctx, T = cfg["num_hidden_layers"], case.get("context", 0), case.get("tokens", 1)
        att = (2 * nh + 2 * nk) * HD * H
        row = 2 * nk * (HD * 2 if not case["kv_bits"] else HD * case["kv_bits"] // 8 + 8)
        if E:
            k = cfg["num_experts_per_tok"]
            touched = E * (1 - (1 - k / E) ** T)
            ff_read, ff_flops = 3 * F * H * touched + E * H, T * (3 * F * H * k + E * H)
        else:
            ff_read, ff_flops = 3 * F * H, T * 3 * F * H
        nbytes = L * (2 * (att + ff_read) + row * (ctx + T))
        flops = L * (2 * (T * att + ff_flops) + 4 * nh * HD * _seen(ctx, T))
        if case["kind"] == "layer":
            nbytes += 4 * T * H
        else:
            nbytes += 2 * cfg["vocab_size"] * H + 4 * cfg["vocab_size"] + 4 * T * H
            flops += 2 * cfg["vocab_size"] * H
        return {"bytes": nbytes, "flops": flops}
    cfg = _seq_config(case)
    W, V = cfg["width"], cfg["vocab"]
    if case["kind"] == "batch":
        steps = [[(0, n) for n in _ragged(case)]]
    else:
        lens = [max(1, case["prompt"] - 3 * i) for i in range(case["sequences"])]
        steps = [[(0, n) for n in lens]] + [[(n + j, 1) for n in lens] for j in range(case["steps"])]
    nbytes = flops = 0
    for entries in steps:
        N = sum(n for _, n in entries)
        nbytes += 2 * N * W + 2 * V * W + 4 * len(entries) * V
        flops += 2 * len(entries) * V * W
        for i, L in enumerate(cfg["layers"]):
            mx, mlp = L["mixer"], L["mlp"]
            H, G, d = mx["heads"], mx["kv_heads"], mx["dim"]
            if L["type"] == "attention":
                m = (2 * H + (2 * G if mx.get("kv_from") is None else 0)) * d * W
                seen = [_seen(p, n, mx["mask"]["size"]) for p, n in entries]
                flops += 4 * H * d * sum(seen)
                nbytes += 4 * G * d * sum(min(p + n, mx["mask"]["size"]) for p, n in entries)
            else:
                m = (2 * G + 3 * H) * d * W + 2 * H * W
                flops += 8 * H * d * d * N
                nbytes += 8 * H * d * d * len(entries)
            flops += 2 * N * m
            if mlp["kind"] == "moe":
                E, k, f = mlp["router"]["experts"], mlp["router"]["top"], mlp["expert"]["ff"]
                nbytes += 4 * f * W * E * (1 - (1 - k / E) ** N) + 2 * E * W
                flops += 2 * N * (2 * f * W * k + E * W)
            else:
                n_mat = 2 if cfg["architecture"] == "Bokenex" else 3
                m += n_mat * mlp["ff"] * W
                flops += 2 * N * n_mat * mlp["ff"] * W
            nbytes += 2 * m
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # bf16 storage between the operations: measured against the sums in 64 bits, a layer is off by 4e-3 (2-norm), 8 layers and the
    # head by 1.2e-2, the layer-list models (fp32 residual) by 3e-3; two orders of the sums differ by less than that
    if case["kind"] in ("token", "prompt"):
        return {"rel": 0.03, "max": 0.3}
    return {"rel": 0.015 if case["kind"] == "layer" else 0.012, "max": 0.3}


# -- the same in 64 bits -----------------------------------------------------------------------------------------------------
def _rms(x, eps):
    return x / torch.sqrt(x.pow(2).mean(-1, keepdim=True) + eps)


def _rope(x, theta):
    """x [T, heads, HD], rotated by halves; angles of the positions 0 .. T - 1"""
    half = HD // 2
    inv = (theta ** (-(2.0 * torch.arange(half, dtype=F64, device=DEV)) / HD)).float()
    ang = (torch.arange(x.shape[0], device=DEV, dtype=torch.float32)[:, None] * inv[None]).to(F64)
    c, s = ang.cos()[:, None], ang.sin()[:, None]
    a, b = x[..., :half], x[..., half:]
    return torch.cat([a * c - b * s, a * s + b * c], -1)


def _affine(x, bits):
    """rows of a quantised cache as they are read back: groups of 64, one bound of a group exact, scale and bias stored in 16 bits"""
    g = x.to(BF).float().reshape(*x.shape[:-1], 2, 64)
    hi, lo, n = g.amax(-1, keepdim=True), g.amin(-1, keepdim=True), 2.0 ** bits - 1
    low = lo.abs() > hi.abs()
    scale = ((hi - lo) / n).clamp_min(1e-7)
    scale, edge = torch.where(low, scale, -scale), torch.where(low, lo, hi)
    q0 = torch.round(edge / scale)
    scale, bias = torch.where(q0 != 0, edge / q0, scale), torch.where(q0 != 0, edge, torch.zeros_like(edge))
    code = ((g - bias) / scale).round().clamp(0, n)
    return (scale.to(BF).to(F64) * code.to(F64) + bias.to(BF).to(F64)).reshape(x.shape)


def _attend(q, k, v, scale, first, block=0, window=0, weigh=None):
    """q [T, H, d] at positions first .. on keys [n, G, d] from position 0; causal, within blocks or a window; -> [T, H d]"""
    T, H, d = q.shape
    G = k.shape[1]
    out = torch.empty(T, H, d, dtype=F64, device=DEV)
    j = torch.arange(k.shape[0], device=DEV)[None]
    for t0 in range(0, T, 256):
        i = torch.arange(first + t0, first + min(T, t0 + 256), device=DEV)[:, None]
        hide = j > i
        if block:
            hide |= (j // block) != (i // block)
        if window:
            hide |= i - j >= window
        for h in range(G):
            qs = q[t0:t0 + 256, h * (H // G):(h + 1) * (H // G)].transpose(0, 1)
            s = qs @ k[:, h].T * scale
            if weigh is None:
                p = torch.softmax(s.masked_fill(hide, float("-inf")), -1)
            else:
                p = weigh(s, (i - j).clamp_min(0).to(F64), slice(h * (H // G), (h + 1) * (H // G))).masked_fill(hide, 0.0)
            out[t0:t0 + 256, h * (H // G):(h + 1) * (H // G)] = (p @ v[:, h]).transpose(0, 1)
    return out.reshape(T, H * d)


def _exact_llama(case, seed):
    cfg, w, given = _llama_inputs(case, seed)
    ctx, eps, nh, nk = case.get("context", 0), cfg["rms_norm_eps"], cfg["num_attention_heads"], cfg["num_key_value_heads"]
    x = w["model.embed_tokens.weight"][given.long()].to(F64) if given.dim() == 1 else given.to(F64)
    n, L = x.shape[0], cfg["num_hidden_layers"]
    for i in range(L):
        p = f"model.layers.{i}."
        q0 = ctx if i == L - 1 else 0          # the last layer's output is wanted for the call's tokens alone

        def proj(name, z):
            y = z @ w[f"{p}self_attn.{name}_proj.weight"].to(F64).T
            b = w.get(f"{p}self_attn.{name}_proj.bias")
            return y if b is None else y + b.to(F64)

        h = _rms(x, eps) * w[p + "input_layernorm.weight"].to(F64)
        q = _rope(proj("q", h).view(n, nh, HD), cfg["rope_theta"])[q0:]
        k, v = _rope(proj("k", h).view(n, nk, HD), cfg["rope_theta"]), proj("v", h).view(n, nk, HD)
        if case["kv_bits"]:
            k, v = _affine(k, case["kv_bits"]), _affine(v, case["kv_bits"])
        x = x[q0:] + proj("o", _attend(q, k, v, HD ** -0.5, q0))
        h = _rms(x, eps) * w[p + "post_attention_layernorm.weight"].to(F64)

        def glu(z, gate, up, down):
            return (torch.nn.functional.silu(z @ gate.to(F64).T) * (z @ up.to(F64).T)) @ down.to(F64).T

        E = cfg.get("num_local_experts", 0)
        if E:
            m = p + "block_sparse_moe."
            top = (h @ w[m + "gate.weight"].to(F64).T).topk(cfg["num_experts_per_tok"], -1)
            share, y = torch.softmax(top.values, -1), torch.zeros_like(x)
            for e in range(E):
                t, j = (top.indices == e).nonzero(as_tuple=True)
                if t.numel():
                    y[t] += share[t, j, None] * glu(h[t], *(w[f"{m}experts.{e}.{c}.weight"] for c in ("w1", "w3", "w2")))
            x = x + y
        else:
            x = x + glu(h, *(w[f"{p}mlp.{c}_proj.weight"] for c in ("gate", "up", "down")))
    if case["kind"] == "layer":
        return x
    last = _rms(x[-1], eps) * w["model.norm.weight"].to(F64)
    logits = torch.cat([last @ r.to(F64).T for r in w["lm_head.weight"].split(16384)])
    return x, logits


def _conv(u, w):
    """causal, depthwise: y_t = sum_j w[:, j] u_(t - taps + 1 + j)"""
    J = w.shape[1]
    z = torch.cat([torch.zeros(J - 1, u.shape[1], dtype=F64, device=DEV), u])
    return sum(w[:, j].to(F64) * z[j:j + u.shape[0]] for j in range(J))


def _rotate_pairs(z, dims, base):
    ang = torch.arange(z.shape[0], device=DEV, dtype=F64)[:, None] * base ** (-2.0 * torch.arange(dims // 2, device=DEV, dtype=F64) / dims)
    c, s = ang.cos()[:, None], ang.sin()[:, None]
    a, b, out = z[..., 0:dims:2], z[..., 1:dims:2], z.clone()
    out[..., 0:dims:2], out[..., 1:dims:2] = a * c - b * s, b * c + a * s
    return out


def _delta(q, k, v, beta, decay):
    """q, k, v [T, H, d]; M <- decay M; M <- M + k (beta (v - M' k))'; o = M' q"""
    M = torch.zeros(q.shape[1], q.shape[2], v.shape[2], dtype=F64, device=DEV)
    out = torch.empty_like(v)
    for t in range(q.shape[0]):
        M *= decay[t][:, None, None]
        e = beta[t][:, None] * (v[t] - (k[t][:, None] @ M)[:, 0])
        M += k[t][:, :, None] * e[:, None]
        out[t] = (q[t][:, None] @ M)[:, 0]
    return out


def _exact_moputar(cfg, w, toks):
    silu, eps, S = torch.nn.functional.silu, cfg["norm"]["eps"], cfg["streams"]
    T = len(toks)
    x0 = w["embed"][torch.tensor(toks, device=DEV)].to(F64)
    xs, kv = torch.stack([x0] * S), {}

    def write(y, q):
        return torch.einsum("st,s...->t...", w[q + ".mix"].to(F64), xs) + w[q + ".out"].to(F64)[:, None, None] * y

    def read(q, norm):
        return _rms(torch.einsum("s,s...->...", w[q + ".in"].to(F64), xs), eps) * (1 + w[norm].to(F64))

    for i, L in enumerate(cfg["layers"]):
        p, mx = f"l{i}.", L["mixer"]
        H, G, d = mx["heads"], mx["kv_heads"], mx["dim"]
        h = read(p + "hc1", p + "norm1")

        def lin(name, z=h):
            return z @ w[p + name].to(F64).T

        def short(c):
            return _conv(lin("mix." + c), w[f"{p}mix.{c}.conv"])

        if L["type"] == "attention":
            def turned(c, heads):
                return _rotate_pairs((_rms(short(c), eps) * w[f"{p}mix.{c}.norm"].to(F64)).view(T, heads, d), mx["rot"]["dims"], mx["rot"]["base"])

            q = turned("q", H)
            kv[i] = kv[mx["kv_from"]] if mx.get("kv_from") is not None else (turned("k", G), short("v").view(T, G, d))
            y = _attend(q, *kv[i], mx["scale"], 0, block=mx["mask"]["size"])
        else:
            q, k, v = (silu(short(c)).view(T, -1, d) for c in "qkv")
            q, k = (z / torch.sqrt(z.pow(2).sum(-1, keepdim=True) + 1e-6) for z in (q, k))
            beta = torch.sigmoid(lin("mix.b"))
            decay = torch.exp(-torch.exp(w[p + "mix.A_log"].to(F64)) * torch.nn.functional.softplus(lin("mix.a") + w[p + "mix.dt_bias"].to(F64)))
            o = _delta((q * d ** -0.5).repeat_interleave(H // G, 1), k.repeat_interleave(H // G, 1), v, beta, decay)
            y = (_rms(o, eps) * w[p + "mix.norm"].to(F64) * silu(lin("mix.g")).view(T, H, d)).reshape(T, H * d)
        xs = write(lin("mix.o", y), p + "hc1")
        h = read(p + "hc2", p + "norm2")
        y = torch.nn.functional.gelu(lin("mlp.gate", h), approximate="tanh") * lin("mlp.up", h)
        xs = write(lin("mlp.down", y), p + "hc2")
    return _rms(xs.sum(0), eps) * (1 + w["final.norm"].to(F64))


def _exact_bokenex(cfg, w, toks):
    eps, T = cfg["norm"]["eps"], len(toks)
    x = w["embed"][torch.tensor(toks, device=DEV)].to(F64) + w["pos"][:T].to(F64)
    for i, L in enumerate(cfg["layers"]):
        p, mx, mlp = f"l{i}.", L["mixer"], L["mlp"]
        H, G, d = mx["heads"], mx["kv_heads"], mx["dim"]
        h = _rms(x, eps) * w[p + "norm1"].to(F64)

        def short(c, heads):
            return _conv(h @ w[f"{p}mix.{c}"].to(F64).T, w[f"{p}mix.{c}.conv"]).view(T, heads, d)

        q = _rms(short("q", H), eps) * w[p + "mix.q.norm"].to(F64)
        k = _rms(short("k", G), eps) * w[p + "mix.k.norm"].to(F64)
        r1, r2, pb = (w[f"{p}mix.{c}"].to(F64) for c in ("r1", "r2", "pb"))

        def weigh(s, dist, hs):
            return torch.sigmoid(s - r1[hs, None, None] * torch.log(1 + r2[hs, None, None] * dist) + pb[hs, None, None])

        y = _attend(q, k, short("v", G), mx["scale"], 0, window=mx["mask"]["size"], weigh=weigh) @ w[p + "mix.o"].to(F64).T

        def two(z, up, down):
            return torch.relu(z @ up.to(F64).T).pow(2) @ down.to(F64).T

        if mlp["kind"] == "moe":
            top = torch.sigmoid(h @ w[p + "mlp.router"].to(F64).T).topk(mlp["router"]["top"], -1)
            share, f = top.values / top.values.sum(-1, keepdim=True) * mlp["router"]["scale"], torch.zeros_like(x)
            for e in range(mlp["router"]["experts"]):
                t, j = (top.indices == e).nonzero(as_tuple=True)
                if t.numel():
                    f[t] += share[t, j, None] * two(h[t], w[f"{p}mlp.e{e}.up"], w[f"{p}mlp.e{e}.down"])
        else:
            f = two(h, w[p + "mlp.up"], w[p + "mlp.down"])
        x = x + cfg["residual_mult"] * (y + f)
    return _rms(x, eps) * w["final.norm"].to(F64)


def exact(case, seed):
    if "model" in case:
        return _exact_llama(case, seed)
    cfg, w, toks = _seq_inputs(case, seed)
    hidden = [(_exact_moputar if case["family"] == "moputar" else _exact_bokenex)(cfg, w, t) for t in toks]
    head = w["head"].to(F64).T
    if case["kind"] == "batch":
        return torch.stack([h[-1] for h in hidden]) @ head
    k = case["steps"]
    return [torch.stack([h[h.shape[0] - k - 1 + j] for h in hidden]) @ head for j in range(k + 1)]
